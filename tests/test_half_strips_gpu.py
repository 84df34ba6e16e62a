"""Strips of a chunk that decay by more than one reference row can take are paired by halves of four rows, each relative
to its own first row.  That keeps one operand of the pairs at a half's edge as it is (no rounding of a gated
value), and has to hold for gates that jump: fast tokens next to slow ones, fast channels next to slow ones."""

import math

import pytest
import torch
import torch.nn.functional as F

from conftest import assert_close, rel_rms
from delta_feedback_experiment_b200 import chunk_precond_kda, pkda_recurrence
from delta_feedback_experiment_b200.synthetic import INPUT_NAMES, make_inputs
from oracle.pkda_oracle import pkda_oracle_with_grads

pytestmark = pytest.mark.gpu
D = 128


def test_pairs_at_the_edge_of_a_half_keep_an_operand():
    """One channel carries everything, so an entry of the saved pair matrix is a single product: an operand rounded to
    bf16 and the result, or both operands and the result.  With mantissas spread evenly over their logarithm one rounding
    has a relative rms of 2^-8 sqrt(E[1/m^2] / 3) = 0.849 x 2^-9: two of them 1.20, three 1.47.  (The decays, fp32 sums of up
    to a thousand, are good for 2^-13.)"""
    T, H = 2048, 4
    d = make_inputs(1, T, H, D, seed=31, dist="production", dtype=torch.bfloat16)
    for seed, n in enumerate(("q", "k")):
        one = torch.zeros(1, T, H, D)
        one[..., 77] = torch.rand(1, T, H, generator=torch.Generator().manual_seed(seed)) + 0.5
        d[n] = one.to(torch.bfloat16)
    d["A_log"] = torch.tensor([14.5, 14.75, 15.0, 15.5]).log()
    _, saved = pkda_recurrence(*[d[n].cuda() for n in INPUT_NAMES], 1.0, 1.5, 1e-6, False)
    P, kt = saved[0].double().cpu(), saved[2].double().cpu()[..., 77]
    q, decay = d["q"].double()[..., 77], d["A_log"].double().exp() * F.softplus(d["g"].double()[..., 77])
    i = torch.arange(1, T)
    i = i[i % 64 != 0]  # pairs (i, i - 1) of one chunk
    want = q[:, i] * kt[:, i - 1] * torch.exp(-decay[:, i])
    got = torch.stack([P[:, t, :, t % 64 - 1] for t in i.tolist()], dim=1)
    err = ((got - want) / want) * 2 ** 9
    for row in (0, 1, 4, 5):
        assert float(err[:, i % 8 == row].square().mean().sqrt()) < 0.849 * math.sqrt(2.5), row


# Decay in log2 units of the eight tokens of a strip.  By halves: any five up to 112, the outer two up to 45, the last three up to 90.
JUMPS = {"even": [16] * 8, "before the fifth row": [1, 30, 1, 1, 60, 1, 1, 40], "behind the fifth row": [1, 1, 1, 1, 1, 70, 19, 26],
         "line of the last three": [1, 30, 1, 1, 1, 66, 1, 24], "beyond it": [1, 30, 1, 1, 1, 66, 1, 40],
         "one token": [1, 1, 110, 1, 1, 1, 1, 1], "across strips": [90, 1, 1, 1, 30, 1, 1, 44]}


@pytest.mark.parametrize("T", [64, 128, 75])
@pytest.mark.parametrize("channels", ["all", "few"])
@pytest.mark.parametrize("which", list(JUMPS))
def test_gates_that_jump(which, channels, T):
    """All channels together, or a few of them beside channels that hardly decay (whose pairs reach across the chunk)."""
    H = 2
    d = make_inputs(1, T, H, D, seed=T, dist="production", dtype=torch.bfloat16, with_state=True)
    rate = torch.tensor([JUMPS[which][t % 8] for t in range(T)], dtype=torch.float64) * math.log(2)
    rate = rate[None, :, None, None].expand(1, T, H, D).clone()
    if channels == "few":
        rate[..., torch.arange(D) % 16 != 5] = 0.02
    d["g"] = torch.where(rate > 20, rate, torch.expm1(rate).log()).to(torch.bfloat16)  # softplus(g) = rate
    d["A_log"] = torch.zeros(H)
    ref = pkda_oracle_with_grads([d[n] for n in INPUT_NAMES], d["do"], initial_state=d["initial_state"],
                                 initial_A_state=d["initial_A_state"], dtype=torch.float64)
    leaves = {n: d[n].cuda().requires_grad_(True) for n in INPUT_NAMES}
    o, S, A = chunk_precond_kda(**leaves, initial_state=d["initial_state"].cuda(), initial_A_state=d["initial_A_state"].cuda(),
                                output_final_state=True)
    assert rel_rms(o, ref["o"]) < 0.005
    assert_close(S, ref["final_state"], 2e-2, "S")
    assert_close(A, ref["final_A_state"], 1e-4, "A")
    # The limits of tests/test_strip_pairs_gpu.py.  Not for the sums over all tokens of a head (A_log, log_atk_scale), which cancel, and
    # of 64 tokens and slow channels leave too little; the preconditioner's gates are such sums over channels: a third more.
    limit = dict(q=0.007, k=0.008, v=0.007, dt_bias=0.02, g_atk=0.02, beta_atk=0.02)
    for n, g in zip(INPUT_NAMES, torch.autograd.grad(o, list(leaves.values()), d["do"].cuda())):
        assert torch.isfinite(g).all(), n
        if n not in ("A_log", "log_atk_scale"):
            assert rel_rms(g, ref["d" + n]) < limit.get(n, 0.015), f"d{n} rel-rms {rel_rms(g, ref['d' + n]):.3e}"
