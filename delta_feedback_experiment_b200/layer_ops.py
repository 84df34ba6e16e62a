"""The two fused operators next to the recurrence inside the PKDA layer, behind
the reference's operator names and signatures:

* ``pkda_qkv_conv(x, weight, head_dim, norm_channels, eps) -> (q, k, v)`` --
  ``delta_feedback::pkda_qkv_conv`` of the reference
  (``delta_feedback_experiment/fla_ops.py:134-249``): causal depthwise short
  convolution over the concatenated Q|K|V projection, SiLU, per-head L2
  normalisation of the first ``norm_channels`` channels, three output slabs.
* ``pkda_norm_gate(x, gate, weight, eps) -> (y, rstd)`` --
  ``delta_feedback::pkda_norm_gate`` (``fla_ops.py:572-657``): per-head RMS
  normalisation times a learned weight times ``sigmoid(gate)``.

Both are dispatcher operators with autograd (registered by ``csrc/pkda_torch.cpp``) and
fake implementations (here), as the reference registers them, and both call the C ABI of
``libpkda_b200.so``; there is no other implementation behind them.
"""

from __future__ import annotations

import ctypes as C

import torch
from torch import Tensor

from . import _lib, ops
from .fla_ops import _operator, _register_fake

_DTYPES = {torch.bfloat16: _lib.PKDA_BF16, torch.float32: _lib.PKDA_F32}


def _dtype_code(t: Tensor) -> int:
    if t.dtype not in _DTYPES:
        raise RuntimeError(f"PKDA layer operators take bf16 or fp32 activations, got {t.dtype}")
    return _DTYPES[t.dtype]


# ----------------------------------------------------------------- convolution
def qkv_conv_forward(x: Tensor, weight: Tensor, head_dim: int, norm_channels: int, eps: float):
    return _lib.native().conv(x, weight, head_dim, norm_channels, eps)


def qkv_conv_backward(x: Tensor, weight: Tensor, dq: Tensor, dk: Tensor, dv: Tensor, head_dim: int,
                      norm_channels: int, eps: float):
    return tuple(_lib.native().conv(x, weight, dq, dk, dv, head_dim, norm_channels, eps))


pkda_qkv_conv = _operator("pkda_qkv_conv")
"""Signature and meaning of the reference's operator (``fla_ops.py:137-170``)."""


@_register_fake("pkda_qkv_conv")
def _pkda_qkv_conv_fake(x, weight, head_dim, norm_channels, eps):
    batch, length, _ = x.shape
    width = weight.shape[0] // 3
    return tuple(x.new_empty(batch, length, width) for _ in range(3))


@_register_fake("pkda_qkv_conv_backward")
def _pkda_qkv_conv_backward_fake(x, weight, dq, dk, dv, head_dim, norm_channels, eps):
    # the real operators return contiguous tensors whatever the inputs' strides
    return x.new_empty(x.shape), weight.new_empty(weight.shape)


# ------------------------------------------------------------------- norm gate
def norm_gate_forward(x: Tensor, gate: Tensor, weight: Tensor, eps: float):
    return tuple(_lib.native().norm_gate(x, gate, weight, eps))


def norm_gate_backward(x: Tensor, gate: Tensor, weight: Tensor, rstd: Tensor, dy: Tensor, eps: float):
    return _lib.native().norm_gate(x, gate, weight, rstd, dy, eps)


pkda_norm_gate = _operator("pkda_norm_gate")
"""Signature and meaning of the reference's operator (``fla_ops.py:575-593``);
``rstd`` has one fp32 entry per row and feeds the backward."""


@_register_fake("pkda_norm_gate")
def _pkda_norm_gate_fake(x, gate, weight, eps):
    rows = x.numel() // x.shape[-1]
    return x.new_empty(x.shape), torch.empty((rows,), device=x.device, dtype=torch.float32)


@_register_fake("pkda_norm_gate_backward")
def _pkda_norm_gate_backward_fake(x, gate, weight, rstd, dy, eps):
    return x.new_empty(x.shape), gate.new_empty(gate.shape), weight.new_empty(weight.shape)


# ----------------------------------------------------------------- decode step
def pkda_decode_step(qkv: Tensor, conv_state, conv_weight: Tensor, g: Tensor, g_atk: Tensor,
                     beta_atk: Tensor, beta: Tensor, A_log: Tensor, dt_bias: Tensor,
                     log_atk_scale: Tensor, state: Tensor, a_state: Tensor, gate, norm_weight,
                     head_dim: int, scale=None, squash_x: float = 1.5, squash_eps: float = 1e-6,
                     qk_eps: float = 1e-6, norm_eps: float = 1e-6) -> Tensor:
    """One cached decoding step of the layer's token mixer in one launch: the
    history-prefixed Q|K|V convolution, one recurrence step and the RMS-norm gate
    (reference: ``pkda.py:239-288, 473-474, 539-541`` and the cache update of
    ``model.py:775-787``).  ``conv_state`` (three ``[B, W, taps-1]`` tensors), ``state``
    (``[B,H,D,D]`` fp32) and ``a_state`` (``[B,H,D]`` fp32) are the decode cache and are
    UPDATED IN PLACE.  ``qkv`` is the new projection row ``[B, 3W]``; ``g`` the raw decay
    ``[B,H,D]``; ``g_atk`` (fp32), ``beta_atk``, ``beta`` are ``[B,H]``; ``gate`` the
    output-gate logits ``[B,H,D]`` or None (the result is then the recurrence output).
    Returns ``[B,H,D]``."""
    conv_q, conv_k, conv_v = conv_state
    return _lib.native().decode_step(
        qkv, conv_q, conv_k, conv_v, conv_weight, g, g_atk, beta_atk, beta, A_log, dt_bias,
        log_atk_scale, state, a_state, gate, norm_weight, head_dim, scale, squash_x, squash_eps,
        qk_eps, norm_eps)


# ------------------------------------------------------------ control epilogue
def pack_control_gradients(gradients) -> Tensor:
    """The reference's ``pack_control_gradients`` (``cuda_kernels.py:1529-1535``): five
    contiguous slices with a common leading shape -> one row-major packed tensor."""
    if len(gradients) != 5:
        raise ValueError("PKDA has exactly five packed control gradients")
    g0 = gradients[0]
    ops._require_cuda(*gradients)
    prefix = g0.shape[:-1]
    if any(g.shape[:-1] != prefix or g.dtype != g0.dtype for g in gradients[1:]):
        raise ValueError("control gradients must share their leading shape and dtype")
    if any(not g.is_contiguous() for g in gradients):
        raise ValueError("control gradients must be contiguous")
    lib = _lib.load()
    return _pack_on_device(g0, lib, gradients, prefix)


@ops._on_tensor_device
def _pack_on_device(g0, lib, gradients, prefix) -> Tensor:
    a = _lib.PackControlArgs()
    a.rows = g0.numel() // max(g0.shape[-1], 1) if g0.shape[-1] else (gradients[1].numel() // max(gradients[1].shape[-1], 1))
    total = 0
    for i, g in enumerate(gradients):
        a.sizes[i] = g.shape[-1]
        a.grads[i] = g.data_ptr()
        total += g.shape[-1]
    a.dtype = _dtype_code(g0)
    out = torch.empty((*prefix, total), device=g0.device, dtype=g0.dtype)
    a.out = out.data_ptr()
    _lib.check(lib.pkda_pack_control_gradients(C.byref(a), _lib.current_stream()), "pkda_pack_control_gradients")
    ops._count(lib)
    return out


@torch.library.custom_op("delta_feedback::pack_control_gradients", mutates_args=(), device_types="cuda")
def _pack_control_gradients_op(grad0: Tensor, grad1: Tensor, grad2: Tensor, grad3: Tensor,
                               grad4: Tensor) -> Tensor:
    """Name and signature of the reference's operator (``cuda_kernels.py:1493-1506``)."""
    return pack_control_gradients((grad0, grad1, grad2, grad3, grad4))


@_pack_control_gradients_op.register_fake
def _pack_control_gradients_fake(grad0, grad1, grad2, grad3, grad4):
    total = sum(g.shape[-1] for g in (grad0, grad1, grad2, grad3, grad4))
    return torch.empty((*grad0.shape[:-1], total), device=grad0.device, dtype=grad0.dtype)


def pkda_controls(packed: Tensor, A_log_precond: Tensor, dt_bias_precond: Tensor, hidden: int):
    """``(decay_hidden, beta, precond_decay, precond_beta, output_gate_hidden)`` from the packed
    control projection ``[..., hidden + 3H + hidden]`` -- the middle of the reference's
    ``PreconditionedKDA._controls`` (``pkda.py:318-353``) with its backward packing
    (``pkda.py:56-74``).  The two hidden pieces are views of ``packed``."""
    return _lib.native().controls(packed, A_log_precond, dt_bias_precond, hidden)


__all__ = ["pkda_controls", "pack_control_gradients", "pkda_decode_step", "pkda_qkv_conv", "pkda_norm_gate", "qkv_conv_forward", "qkv_conv_backward",
           "norm_gate_forward", "norm_gate_backward"]
