"""Workloads by which the operators of this package are timed.

A case is one call, or one chain of calls, that a host makes through the public entry
points: a cached decoding step, the prefill of a prompt, the forward + backward of a
training step (dense, packed, or the layer's whole token mixer), and the streaming
operators next to the recurrence.  ``listed()`` names representative sizes, ``draw()``
gives further sizes of the same ranges.

Gate distributions.  ``"unit"``: the effective log-decay of every channel is
-softplus(N(0,1)), as the benchmark configurations state it.  ``"production"``: what the
layer's initialisation produces, exp(A_log) ~ U(1, 16) with small gate logits, up to
about 11 nats of decay per token in the fastest heads.
"""

from __future__ import annotations

import math
import random

import torch
import torch.nn.functional as F

from delta_feedback_experiment_b200 import (chunk_precond_kda, pkda_cuda_recurrence,
                                            pkda_norm_gate, pkda_qkv_conv)
from delta_feedback_experiment_b200.layer_ops import pkda_controls, pkda_decode_step

TAPS = 4     # short-convolution length of the layer
EPS = 1e-6
NAMES = ("q", "k", "v", "g", "g_atk", "beta_atk", "beta", "A_log", "dt_bias", "log_atk_scale")


def listed():
    return [
        # One user, one token: the latency of a decoding step of the smallest layer (8 heads).
        {"name": "decode-b1", "kind": "decode", "B": 1, "H": 8},
        # The decoding configuration of the benchmark: 256 users, 32 heads, 512 MB of state.
        {"name": "decode-b256", "kind": "decode", "B": 256, "H": 32},
        # A few cached tokens appended at once (a short prompt, a speculative block): at most
        # 64 tokens, where the dispatcher takes the token-by-token kernel.
        {"name": "prefill-short", "kind": "prefill", "B": 4, "T": 48, "H": 16, "dist": "production",
         "state": True},
        # One long prompt of odd length, no earlier state: forward only, final state kept.
        {"name": "prefill-long", "kind": "prefill", "B": 1, "T": 8191, "H": 16, "dist": "production",
         "state": False},
        # The headline training configuration, with recurrent states in and out.
        {"name": "train-unit", "kind": "train", "B": 8, "T": 4096, "H": 16, "dist": "unit",
         "state": True, "lean": False},
        # What the layer runs in training: no states, lean saving, two 4,096-token rows.
        {"name": "train-production", "kind": "train", "B": 2, "T": 4096, "H": 12,
         "dist": "production", "state": False, "lean": True},
        # One short ragged row (a test, a probe, the tail of a data set).
        {"name": "train-small", "kind": "train", "B": 1, "T": 300, "H": 8, "dist": "production",
         "state": False, "lean": False},
        # The packed configuration: 65,536 tokens cut into sequences of 128 to 8,192 tokens.
        {"name": "packed", "kind": "packed", "total": 65536, "lo": 128, "hi": 8192, "H": 32,
         "dist": "unit", "cut": 7},
        # The fp32 configuration (exact token-by-token kernels), heads of 64 channels.
        {"name": "exact-fp32", "kind": "exact", "B": 2, "T": 512, "H": 4, "D": 64},
        # Q|K|V convolution of a training step at the headline shape.
        {"name": "conv", "kind": "conv", "B": 8, "T": 4096, "H": 16},
        # RMS-norm gate of a training step at the headline shape.
        {"name": "gate", "kind": "gate", "B": 8, "T": 4096, "H": 16},
        # The layer's token mixer in one training step: convolution, controls, recurrence, gate.
        {"name": "mixer", "kind": "mixer", "B": 2, "T": 1000, "H": 8},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, its logarithm spread evenly."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


MOST_UNITS = 8 * 4096 * 16       # (token, head) pairs of a drawn dense case, at most


def draw(rng: random.Random):
    kind = rng.choice(("decode", "prefill", "prefill", "train", "train", "packed", "exact", "conv", "gate",
                       "mixer"))
    if kind == "decode":
        return {"kind": kind, "B": _log(rng, 1, 256), "H": rng.choice((8, 12, 16, 32))}
    if kind == "packed":
        hi = rng.choice((1024, 2048, 4096, 8192))
        return {"kind": kind, "total": _log(rng, 4096, 65536), "lo": rng.choice((16, 128)), "hi": hi,
                "H": rng.choice((8, 12, 16, 32)), "dist": rng.choice(("unit", "production")),
                "cut": rng.randrange(1000)}
    if kind == "exact":
        return {"kind": kind, "B": rng.randint(1, 4), "T": _log(rng, 32, 1024), "H": rng.choice((2, 4, 8)),
                "D": rng.choice((32, 64, 128))}
    H = rng.choice((8, 12, 16))
    T = _log(rng, 16, 8192) if kind == "prefill" else _log(rng, 64, 8192)
    c = {"kind": kind, "B": _log(rng, 1, max(1, min(16, MOST_UNITS // (T * H)))), "T": T, "H": H}
    if kind == "prefill":
        c.update(dist=rng.choice(("unit", "production")), state=rng.random() < 0.5)
    elif kind == "train":
        state = rng.random() < 0.4
        c.update(dist=rng.choice(("unit", "production")), state=state,
                 lean=not state and rng.random() < 0.7)
    return c


# ------------------------------------------------------------------------- inputs
class _Draws:
    """Seeded random tensors on the GPU."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(int(seed))

    def n(self, *size, dtype=torch.float32):
        return torch.randn(size, generator=self.gen, device="cuda", dtype=dtype)

    def u(self, lo, hi, *size):
        return torch.rand(size, generator=self.gen, device="cuda") * (hi - lo) + lo


def _head_params(r, H, D, dist):
    """``A_log``, ``dt_bias``, ``log_atk_scale`` of the main gate."""
    a_log = torch.zeros(H, device="cuda") if dist == "unit" else r.u(1.0, 16.0, H).log()
    return a_log, torch.zeros(H * D, device="cuda"), torch.full((H,), -0.2, device="cuda")


def _precond_params(r, H):
    """``A_log_precond`` and ``dt_bias_precond`` as the layer initialises them."""
    dt = r.u(math.log(1e-3), math.log(1e-1), H).exp()
    return r.u(1.0, 16.0, H).log(), dt + torch.log(-torch.expm1(-dt))


def _recurrence_inputs(r, B, T, H, D, dist, dtype):
    """The ten operator inputs: activations in ``dtype``, ``g_atk`` and parameters fp32."""
    d = {}
    if dist == "unit":
        d["q"] = F.normalize(r.n(B, T, H, D), dim=-1).to(dtype)
        d["k"] = F.normalize(r.n(B, T, H, D), dim=-1).to(dtype)
        d["v"] = r.n(B, T, H, D, dtype=dtype)
        d["g"] = r.n(B, T, H, D, dtype=dtype)
        d["g_atk"] = -F.softplus(r.n(B, T, H))
        d["beta_atk"] = torch.sigmoid(r.n(B, T, H)).to(dtype)
        d["beta"] = torch.sigmoid(r.n(B, T, H)).to(dtype)
    else:
        a_log, bias = _precond_params(r, H)
        d["q"] = F.normalize(F.silu(r.n(B, T, H, D)), dim=-1).to(dtype)
        d["k"] = F.normalize(F.silu(r.n(B, T, H, D)), dim=-1).to(dtype)
        d["v"] = F.silu(r.n(B, T, H, D)).to(dtype)
        d["g"] = (r.n(B, T, H, D) * 0.2).to(dtype)
        d["g_atk"] = -a_log.exp() * F.softplus(r.n(B, T, H) * 0.2 + bias)
        d["beta_atk"] = torch.sigmoid(r.n(B, T, H) * 0.2).to(dtype)
        d["beta"] = torch.sigmoid(r.n(B, T, H) * 0.2).to(dtype)
    d["A_log"], d["dt_bias"], d["log_atk_scale"] = _head_params(r, H, D, dist)
    return d


def _states(r, N, H, D):
    return r.n(N, H, D, D) * 0.02, r.u(0.0, 0.02, N, H, D)


def _cut(case):
    """Offsets of the packed sequences: lengths uniform in [lo, hi], the last one truncated."""
    rng = random.Random(case["cut"])
    offs = [0]
    while offs[-1] < case["total"]:
        offs.append(min(case["total"], offs[-1] + rng.randint(case["lo"], case["hi"])))
    return offs


def _leaf(t):
    return t.detach().requires_grad_(True)


def prepare(case, seed):
    r = _Draws(seed)
    kind, H = case["kind"], case["H"]
    D = case.get("D", 128)
    W = H * D
    bf = torch.bfloat16
    s = {"kind": kind, "case": case}
    if kind == "decode":
        B = case["B"]
        a_log, bias = _precond_params(r, H)
        A_log, dt_bias, centre = _head_params(r, H, D, "production")
        state, a_state = _states(r, B, H, D)
        s["qkv"] = r.n(B, 3 * W, dtype=bf)
        s["args"] = dict(
            conv_state=tuple(r.n(B, W, TAPS - 1, dtype=bf) for _ in range(3)),
            conv_weight=r.n(3 * W, TAPS) * 0.5, g=r.n(B, H, D, dtype=bf) * 0.2,
            g_atk=-a_log.exp() * F.softplus(r.n(B, H) * 0.2 + bias),
            beta_atk=torch.sigmoid(r.n(B, H) * 0.2).to(bf), beta=torch.sigmoid(r.n(B, H) * 0.2).to(bf),
            A_log=A_log, dt_bias=dt_bias, log_atk_scale=centre, state=state, a_state=a_state,
            gate=r.n(B, H, D, dtype=bf), norm_weight=1 + 0.1 * r.n(D), head_dim=D)
    elif kind == "prefill":
        s["in"] = _recurrence_inputs(r, case["B"], case["T"], H, D, case["dist"], bf)
        s["state"], s["a_state"] = _states(r, case["B"], H, D) if case["state"] else (None, None)
    elif kind in ("train", "packed", "exact"):
        B, T = (1, case["total"]) if kind == "packed" else (case["B"], case["T"])
        dist = case.get("dist", "unit")
        d = _recurrence_inputs(r, B, T, H, D, dist, torch.float32 if kind == "exact" else bf)
        s["in"] = {n: _leaf(d[n]) for n in NAMES}
        s["wrt"] = [s["in"][n] for n in NAMES]
        s["do"] = r.n(B, T, H, D, dtype=d["q"].dtype)
        N = B
        if kind == "packed":
            offs = _cut(case)
            N = len(offs) - 1
            s["cu"] = torch.tensor(offs, dtype=torch.int32, device="cuda")
        if case.get("state", kind == "packed"):
            s["state"], s["a_state"] = (_leaf(t) for t in _states(r, N, H, D))
            s["wrt"] += [s["state"], s["a_state"]]
            s["dS"] = r.n(N, H, D, D) * 0.1
    elif kind == "conv":
        B, T = case["B"], case["T"]
        s["x"], s["w"] = _leaf(r.n(B, T, 3 * W, dtype=bf)), _leaf(r.n(3 * W, TAPS) * 0.5)
        s["d"] = [r.n(B, T, W, dtype=bf) for _ in range(3)]
    elif kind == "gate":
        B, T = case["B"], case["T"]
        s["x"], s["gate"] = _leaf(r.n(B, T, H, D, dtype=bf)), _leaf(r.n(B, T, H, D, dtype=bf))
        s["w"] = _leaf(1 + 0.1 * r.n(D))
        s["dy"] = r.n(B, T, H, D, dtype=bf)
    else:  # mixer
        B, T = case["B"], case["T"]
        a_log, bias = _precond_params(r, H)
        A_log, dt_bias, centre = _head_params(r, H, D, "production")
        s["x"], s["w"] = _leaf(r.n(B, T, 3 * W, dtype=bf)), _leaf(r.n(3 * W, TAPS) * 0.5)
        s["packed"] = _leaf(r.n(B, T, 2 * D + 3 * H, dtype=bf) * 0.2)
        s["g"], s["gate"] = _leaf(r.n(B, T, H, D, dtype=bf) * 0.2), _leaf(r.n(B, T, H, D, dtype=bf))
        s["p"] = {"A_log": _leaf(A_log), "dt_bias": _leaf(dt_bias), "log_precond_center": _leaf(centre)}
        s["a_pre"], s["b_pre"], s["norm"] = _leaf(a_log), _leaf(bias), _leaf(1 + 0.1 * r.n(D))
        s["wrt"] = [s["x"], s["w"], s["packed"], s["g"], s["gate"], *s["p"].values(), s["a_pre"], s["b_pre"],
                    s["norm"]]
        s["cot"] = [r.n(B, T, H, D, dtype=bf), r.n(B, T, D, dtype=bf), r.n(B, T, D, dtype=bf)]
    return s


# --------------------------------------------------------------------------- passes
def run(s):
    kind, c = s["kind"], s["case"]
    if kind == "decode":
        a = s["args"]
        out = pkda_decode_step(s["qkv"], **a)
        return {"out": out, "state": a["state"], "a_state": a["a_state"], "conv": a["conv_state"]}
    if kind == "prefill":
        d = s["in"]
        with torch.no_grad():
            o, S, A = pkda_cuda_recurrence(
                d["q"], d["k"], d["v"], d["g"], d["beta"], d["g_atk"], d["beta_atk"], s["state"], s["a_state"],
                True, A_log=d["A_log"], dt_bias=d["dt_bias"], log_precond_center=d["log_atk_scale"],
                head_dim=d["q"].shape[-1])
        return o, S, A
    if kind == "conv":
        q, k, v = pkda_qkv_conv(s["x"], s["w"], 128, s["x"].shape[-1] * 2 // 3, EPS)
        return (q, k, v, *torch.autograd.grad([q, k, v], [s["x"], s["w"]], s["d"]))
    if kind == "gate":
        y, rstd = pkda_norm_gate(s["x"], s["gate"], s["w"], EPS)
        return (y, rstd, *torch.autograd.grad(y, [s["x"], s["gate"], s["w"]], s["dy"]))
    if kind == "mixer":
        B, T, H, D = s["g"].shape
        q, k, v = pkda_qkv_conv(s["x"], s["w"], D, 2 * H * D, EPS)
        h0, beta, g_atk, beta_atk, h1 = pkda_controls(s["packed"], s["a_pre"], s["b_pre"], D)
        q, k, v = (t.view(B, T, H, D) for t in (q, k, v))
        o, _, _ = pkda_cuda_recurrence(q, k, v, s["g"], beta, g_atk, beta_atk, None, None, False, head_dim=D,
                                       lean_recurrence=True, training=True, **s["p"])
        y, _ = pkda_norm_gate(o, s["gate"], s["norm"], EPS)
        return (y, *torch.autograd.grad([y, h0, h1], s["wrt"], s["cot"]))
    d = s["in"]
    if kind == "train" and not c["state"]:
        o, _, _ = pkda_cuda_recurrence(
            d["q"], d["k"], d["v"], d["g"], d["beta"], d["g_atk"], d["beta_atk"], None, None, False,
            A_log=d["A_log"], dt_bias=d["dt_bias"], log_precond_center=d["log_atk_scale"],
            head_dim=d["q"].shape[-1], lean_recurrence=c["lean"], training=True)
        return (o, *torch.autograd.grad(o, s["wrt"], s["do"]))
    has_state = "state" in s
    o, S, A = chunk_precond_kda(
        **d, initial_state=s.get("state"), initial_A_state=s.get("a_state"), output_final_state=has_state,
        disable_recompute=True, cu_seqlens=s.get("cu"))
    if not has_state:
        return (o, *torch.autograd.grad(o, s["wrt"], s["do"]))
    return (o, S, A, *torch.autograd.grad([o, S], s["wrt"], [s["do"], s["dS"]]))


# ------------------------------------------------------------------ necessary work
def work(case):
    """Every input read once, every output written once; flops of the chunked form with
    64-token chunks (forward 182,955 per (token, head) at 128 channels, backward twice
    that), or of the token-by-token recurrence where that is the path."""
    kind, H = case["kind"], case["H"]
    D = case.get("D", 128)
    if kind == "decode":
        n = case["B"] * H
        # S and A read and written; the projection row, gates and history in; history and output row out
        return {"bytes": n * (8 * D * D + 8 * D + 2 * 3 * D * (1 + 2 * (TAPS - 1)) + 6 * D + 8),
                "flops": n * 7 * D * D}
    tokens = case["total"] if kind == "packed" else case["B"] * case["T"]
    units = tokens * H
    rows = len(_cut(case)) - 1 if kind == "packed" else case["B"]
    state = rows * H * 4 * (D * D + D)
    if kind == "prefill":
        per = 182955 if case["T"] > 64 else 7 * D * D
        return {"bytes": units * (10 * D + 8) + state * (2 if case["state"] else 1), "flops": units * per}
    if kind == "exact":
        return {"bytes": units * (4 * 14 * D + 4 * 9), "flops": units * 21 * D * D}
    if kind == "conv":
        return {"bytes": 2 * tokens * 15 * H * D, "flops": tokens * 3 * H * D * 50}
    if kind == "gate":
        return {"bytes": units * (2 * 8 * D + 8), "flops": units * D * 30}
    chunked = {"bytes": units * 3616, "flops": units * 548864}
    if kind == "mixer":
        # x, packed controls, g, gate and the cotangents in; their gradients and y out
        by = tokens * (2 * H * D * (2 * 3 + 2 + 2 + 2) + 2 * (2 * (2 * D + 3 * H) + 2 * D))
        return {"bytes": by, "flops": chunked["flops"] + tokens * 3 * H * D * 50 + units * D * 30}
    has_state = kind == "packed" or case["state"]
    return {"bytes": chunked["bytes"] + (4 * state if has_state else 0), "flops": chunked["flops"]}


def tolerance(case):
    """fp32: sums of up to a thousand products in 32 bits.  bf16: rounding of operands and
    results; the gradients of the gate parameters are sums whose terms partly cancel."""
    kind = case["kind"]
    if kind == "exact":
        return {"rel": 5e-5, "max": 2e-3}
    if kind in ("decode", "conv", "gate"):
        return {"rel": 5e-3, "max": 0.05}
    if kind == "prefill":
        return {"rel": 1e-2, "max": 0.2}
    return {"rel": 2e-2, "max": 0.4}
