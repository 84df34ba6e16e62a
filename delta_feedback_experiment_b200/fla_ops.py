"""Operator boundary of the PKDA recurrence, mirroring the reference's
``delta_feedback_experiment/fla_ops.py`` for this path: the same custom-op
names, signatures, saved-intermediate contract and error behaviour, with the
B200 kernels behind them instead of the Triton fork.

* ``delta_feedback::pkda_recurrence`` (reference ``fla_ops.py:252-349``)
* ``delta_feedback::pkda_recurrence_backward`` (``fla_ops.py:381-499``)

Schema, CUDA kernel and autograd kernel of both are registered by the native host layer
(``csrc/pkda_torch.cpp``); the fake implementations (so that ``torch.compile(fullgraph=True)``
keeps them in one graph) stand here.  Launches go to the current stream,
never synchronise and allocate only through torch, so they can be captured in
CUDA graphs.  There is no fallback: without the CUDA library the operators
raise ``RuntimeError``.
"""

from __future__ import annotations

import torch
from torch import Tensor

from . import _lib, ops

CHUNK_SIZE = 64
"""Chunk length shared by forward and backward (reference ``fla_ops.py:32``)."""

PKDA_INTERMEDIATES = ("Aqk", "Akk", "k_precond", "ac_atk", "a_atk", "sa_atk")
"""Always handed to the backward, in this order (reference ``fla_ops.py:46-53``).
Contents here: ``Aqk`` the scaled causal query-key products, ``Akk`` the inverse
UT transform, ``k_precond`` the preconditioned write keys, ``a_atk`` the
preconditioner state at every chunk start, ``sa_atk`` its per-chunk log-decay
sums, and ``ac_atk`` the main gate's per-chunk decay totals."""

PKDA_RETAINED = ("w", "kg", "v_new", "h", "qg")
"""Kept as well unless ``lean`` (reference ``fla_ops.py:57``); a lean backward
rebuilds them with the forward's own kernels, so its gradients are bitwise those
of a retaining backward."""


def fla_ops_available() -> bool:
    """True when the CUDA library loads (name kept from the reference,
    ``fla_ops.py:69-70``)."""
    return _lib.available()


def _intermediate_meta(q: Tensor, v: Tensor, lean: bool):
    return ops.intermediate_meta(q, v, lean)


def _check_intermediates(tensors, q: Tensor, v: Tensor, lean: bool) -> None:
    """The check that the operator's CUDA kernel runs on the list it hands back: count, and per
    entry shape, dtype, device and contiguity as the fake implementation promises them (same
    contract as the reference's check, ``fla_ops.py:100-128``)."""
    _lib.native().check_intermediates(tensors, q, v, lean)


def _operator(name: str):
    """The registered operator ``delta_feedback::<name>``.  While the native layer does not load, a
    stand-in: each call tries to load it again and raises the reason if that fails."""
    if _lib.available():
        return getattr(torch.ops.delta_feedback, name).default

    def stand_in(*args, **kwargs):
        _lib.native()
        return getattr(torch.ops.delta_feedback, name).default(*args, **kwargs)

    stand_in.__name__ = name
    return stand_in


def _register_fake(name: str):
    """``torch.library.register_fake`` for an operator of the native layer, as soon as there is one."""
    def register(fn):
        _lib.when_loaded(lambda: torch.library.register_fake(f"delta_feedback::{name}", fn))
        return fn
    return register


pkda_recurrence = _operator("pkda_recurrence")
"""``(q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale, scale, squash_x,
squash_eps, lean) -> (o, saved)``: dense training / prefill forward without recurrent state;
returns the output and the intermediates its backward reuses (all eleven unless ``lean``).
``g`` is the raw decay projection; the gate and its chunk-local cumulative sum are computed
inside the kernels.  bf16 activations of 128-channel heads take the chunked kernels, everything
else the exact token-by-token ones (which leave the intermediates unwritten)."""


@_register_fake("pkda_recurrence")
def _pkda_recurrence_fake(q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale,
                          scale, squash_x, squash_eps, lean):
    output = torch.empty((*q.shape[:3], v.shape[-1]), device=q.device, dtype=q.dtype)
    saved = [torch.empty(shape, device=q.device, dtype=dt)
             for shape, dt in _intermediate_meta(q, v, lean)]
    return output, saved


@_register_fake("pkda_recurrence_backward")
def _pkda_recurrence_backward_fake(q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias,
                                   log_atk_scale, saved, do, scale, squash_x, squash_eps,
                                   autocast_dtype, lean):
    # the real operator returns fresh contiguous tensors whatever the inputs' strides
    return [t.new_empty(t.shape) for t in
            (q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale)]


__all__ = ["CHUNK_SIZE", "PKDA_INTERMEDIATES", "PKDA_RETAINED", "fla_ops_available",
           "pkda_recurrence"]
