"""Low-level launchers.  The chunked and the exact kernels are called through the native
host layer (``csrc/pkda_torch.cpp``), which allocates outputs and scratch, fills the C structs
and enqueues on the current CUDA stream; the no-allocation forward goes straight to the C ABI.
No arithmetic happens in Python.
"""

from __future__ import annotations

import ctypes as C
import functools
from typing import Optional, Sequence

import torch
from torch import Tensor

from . import _lib

CHUNK_SIZE = _lib.CHUNK

_STATIC_LAUNCHES = 0     # kernels enqueued by the ctypes calls of this module


def __getattr__(name: str):
    """``ops.LAUNCHES``: kernels enqueued by the operators since import (launch accounting)."""
    if name == "LAUNCHES":
        return _STATIC_LAUNCHES + (_lib.native().launches() if _lib.available() else 0)
    raise AttributeError(name)


_STATIC_STATUS = None    # (device address, device) of the no-allocation forward's status word


def track_device_status(enable: bool) -> None:
    """Debugging aid.  While enabled, every chunked forward / backward copies its
    device status word (4 bytes, one extra copy on the launch stream) into a tensor
    of its own that ``last_device_status`` / ``last_backward_status`` read.  Off by
    default: production callers learn of a device-side failure through the NaN the
    library writes over the head of the outputs, without any read-back."""
    global _STATIC_STATUS
    _STATIC_STATUS = None
    _lib.native().track_status(bool(enable))


def last_device_status() -> int:
    """Status word the most recent chunked forward's kernels left on the device
    (0 = ok, 1 = a bounded wait inside a kernel gave up and its CTA skipped its
    stores); 0 when tracking is off.  Synchronises; meant for tests and debugging."""
    word = _lib.native().last_status(False)
    if word is not None:
        return int(word.view(torch.int32).item())
    if _STATIC_STATUS is None:
        return 0
    address, device = _STATIC_STATUS     # (device address inside the library's static array, device)
    with torch.cuda.device(device):
        return int(torch.as_tensor(_DeviceWord(address), device=device).item())


def last_backward_status() -> int:
    """The same for the most recent chunked backward (its results are void if a
    bounded wait gave up)."""
    word = _lib.native().last_status(True)
    return 0 if word is None else int(word.view(torch.int32).item())


def _count(lib) -> None:
    global _STATIC_LAUNCHES
    _STATIC_LAUNCHES += int(lib.pkda_last_launch_count())


_DTYPES = {torch.bfloat16: _lib.PKDA_BF16, torch.float32: _lib.PKDA_F32}


def _require_cuda(*tensors: Optional[Tensor]) -> None:
    """Every given tensor must live on one and the same CUDA device (the kernels
    run on a single device and dereference every pointer there)."""
    device = None
    for t in tensors:
        if t is None:
            continue
        if not t.is_cuda:
            raise RuntimeError("PKDA CUDA operators need CUDA tensors; there is no CPU path")
        if device is None:
            device = t.device
        elif t.device != device:
            raise RuntimeError(
                f"PKDA operator arguments live on different devices ({device} and {t.device})")


def _on_tensor_device(fn):
    """Runs a launcher with its first tensor's device current, so that the library
    launches (and encodes its tensor maps) on the device that owns the data and
    torch's current stream of THAT device is the one used, whatever device the
    caller had current (the reference's kernels guard the same way)."""
    @functools.wraps(fn)
    def wrapper(first, *args, **kwargs):
        if not getattr(first, "is_cuda", False):
            raise RuntimeError("PKDA CUDA operators need CUDA tensors; there is no CPU path")
        with torch.cuda.device(first.device):
            return fn(first, *args, **kwargs)
    return wrapper


def _problem(q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale, scale, x, eps,
             initial_state, initial_A_state, keep) -> _lib.Problem:
    """Problem struct of the no-allocation forward (dense batches); ``keep`` collects every
    tensor whose storage must outlive the launch call (detached or cast parameters)."""
    B, T, H, D = q.shape
    if q.dtype not in _DTYPES:
        raise RuntimeError(f"PKDA supports bf16 and fp32 activations, not {q.dtype}")
    act = q.dtype
    _require_cuda(q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale,
                  initial_state, initial_A_state)

    def act_c(t, shape):
        if tuple(t.shape) != tuple(shape):
            raise RuntimeError(f"PKDA input has shape {tuple(t.shape)}, expected {tuple(shape)}")
        t = t.to(act).contiguous()
        keep.append(t)
        return t.data_ptr()

    def f32_c(t, numel):
        if t.numel() != numel:
            raise RuntimeError(f"PKDA parameter has {t.numel()} elements, expected {numel}")
        t = t.detach().to(torch.float32).contiguous()
        keep.append(t)
        return t.data_ptr()

    p = _lib.Problem()
    p.n_seqs, p.seq_len, p.total_tokens = B, T, B * T
    p.heads, p.head_dim = H, D
    p.dtype = _DTYPES[act]
    p.scale = float(D ** -0.5 if scale is None else scale)
    p.squash_x, p.squash_eps = float(x), float(eps)
    p.q, p.k, p.v, p.g = (act_c(t, (B, T, H, D)) for t in (q, k, v, g))
    p.g_atk = f32_c(g_atk, B * T * H)
    p.beta_atk, p.beta = act_c(beta_atk, (B, T, H)), act_c(beta, (B, T, H))
    p.A_log = f32_c(A_log, H)
    p.dt_bias = f32_c(dt_bias, H * D)
    p.log_atk_scale = f32_c(log_atk_scale, H)
    if initial_state is not None:
        p.initial_state = f32_c(initial_state, B * H * D * D)
    if initial_A_state is not None:
        p.initial_A_state = f32_c(initial_A_state, B * H * D)
    return p


def recurrent_forward(q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale, scale,
                      x, eps, initial_state=None, initial_A_state=None, cu_seqlens=None,
                      output_final_state=True, inplace_state=False):
    """Token-by-token kernel.  Returns ``(o, S, A)`` (states ``None`` unless
    requested).  ``inplace_state`` writes the new states over the given fp32
    contiguous initial states and returns those same tensors."""
    return _lib.native().recurrent_forward(
        q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale, initial_state,
        initial_A_state, cu_seqlens, scale, x, eps, output_final_state, inplace_state)


def intermediate_meta(q: Tensor, v: Tensor, lean: bool, chunks_flat: Optional[int] = None):
    """Shapes and dtypes of the saved intermediates, in the reference's order
    (``delta_feedback_experiment/fla_ops.py:73-97``)."""
    B, T, H, K = q.shape
    V = v.shape[-1]
    NT = -(-T // CHUNK_SIZE) if chunks_flat is None else chunks_flat
    act = q.dtype
    meta = [
        ((B, T, H, CHUNK_SIZE), act), ((B, T, H, CHUNK_SIZE), act), ((B, T, H, K), act),
        ((B, NT, H, K), torch.float32), ((B, NT, H, K), torch.float32),
        ((B, NT, H), torch.float32),
    ]
    if not lean:
        meta += [((B, T, H, K), act), ((B, T, H, K), act), ((B, T, H, V), act),
                 ((B, NT, H, K, V), act), ((B, T, H, K), act)]
    return tuple(meta)


def chunk_forward(q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale, scale, x,
                  eps, initial_state=None, initial_A_state=None, cu_seqlens=None,
                  output_final_state=False):
    """Chunked forward (bf16, D = 128).  Returns ``(o, S_T, A_T, saved)`` where
    ``saved`` is the full list of eleven intermediates."""
    return _lib.native().chunk_forward(
        q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale, initial_state,
        initial_A_state, cu_seqlens, scale, x, eps, output_final_state)


def chunk_backward(q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale, scale, x,
                   eps, saved: Sequence[Tensor], do, initial_state=None, initial_A_state=None,
                   cu_seqlens=None, d_final_state=None, lean=False, want_state_grads=False):
    """Chunked backward.  ``saved`` holds the six always-kept intermediates and,
    unless ``lean``, the five retained ones.  Returns the ten gradients (plus
    ``dS0, dA0`` when ``want_state_grads``)."""
    return _split_grads(_lib.native().backward(
        q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale, initial_state,
        initial_A_state, cu_seqlens, scale, x, eps, list(saved), do, d_final_state, lean,
        want_state_grads))


def recurrent_backward(q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale, scale, x,
                       eps, do, initial_state=None, initial_A_state=None, cu_seqlens=None,
                       d_final_state=None, want_state_grads=False):
    """Exact fp32 backward of the recurrence (any supported head width, bf16 or
    fp32 activations); needs no saved intermediates.  Returns the ten gradients
    (plus ``dS0, dA0`` when ``want_state_grads``)."""
    return _split_grads(_lib.native().backward(
        q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale, initial_state,
        initial_A_state, cu_seqlens, scale, x, eps, None, do, d_final_state, False,
        want_state_grads))


def _split_grads(grads):
    dS0, dA0 = grads[10:] if len(grads) == 12 else (None, None)
    return grads[:10], dS0, dA0


def static_scratch_bytes() -> int:
    return int(_lib.load().pkda_static_scratch_bytes())


@_on_tensor_device
def chunk_forward_static(q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale, scale,
                         x, eps, o, saved, initial_state=None, initial_A_state=None,
                         final_state=None, final_A_state=None):
    """Chunked forward through ``pkda_chunk_fwd_static``: for hosts that must not
    allocate device memory while the operator runs.  The caller supplies every
    buffer -- contiguous bf16 inputs, the output ``o`` and the eleven
    intermediates ``saved`` (shapes of ``intermediate_meta``), optionally the
    fp32 final-state buffers -- and the library takes its scratch from the fixed
    array built into it, so nothing is allocated here or below.  Raises
    ``RuntimeError`` when the problem needs more scratch than that array has
    (``static_scratch_bytes()``).  Calls share the array: do not let two of them
    overlap on the GPU, and make the first call on a device outside stream
    capture."""
    _require_cuda(q, k, v, g, g_atk, beta_atk, beta, o)
    lib = _lib.load()
    tensors = (q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale)
    if not all(t.is_contiguous() for t in tensors) or g_atk.dtype != torch.float32:
        raise RuntimeError("the no-allocation entry point needs contiguous inputs (fp32 g_atk)")
    keep: list = []
    p = _problem(q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale, scale, x, eps,
                 initial_state, initial_A_state, keep)
    if len(saved) != 11:
        raise RuntimeError("eleven intermediate buffers are required")
    args = _lib.ChunkFwdArgs()
    args.p = p
    args.o = o.data_ptr()
    if final_state is not None:
        args.final_state, args.final_A_state = final_state.data_ptr(), final_A_state.data_ptr()
    (args.Aqk, args.Akk, args.k_precond, args.ac_atk, args.a_atk, args.sa_atk, args.w, args.kg,
     args.v_new, args.h, args.qg) = [t.data_ptr() for t in saved]
    _lib.check(lib.pkda_chunk_fwd_static(C.byref(args), _lib.current_stream()),
               "pkda_chunk_fwd_static")
    _count(lib)
    native = _lib.native()
    if native.tracking():
        global _STATIC_STATUS
        native.drop_forward_status()
        _STATIC_STATUS = _static_status_view(lib, p)
    return o


class _DeviceWord:
    """Presents a raw device address as a one-element int32 array to
    ``torch.as_tensor``."""

    def __init__(self, address: int):
        self.__cuda_array_interface__ = {
            "shape": (1,), "typestr": "<i4", "data": (int(address), False), "version": 2}


def _static_status_view(lib, p):
    """Where the static-scratch forward keeps its status word: the device address
    inside the library's own array and the device (nothing is allocated or copied
    here; ``last_device_status`` reads the word, before the next such call
    overwrites it)."""
    addr = C.c_void_p()
    _lib.check(lib.pkda_static_status_ptr(C.byref(p), C.byref(addr)), "pkda_static_status_ptr")
    return int(addr.value), torch.device("cuda", torch.cuda.current_device())
