"""Chunks that decay too much for one reference row are paired strip by strip (8 rows), each strip relative to
reference rows of its own.  Which rows those are follows the decay: the strip's first and last row, the first of
either half and the fifth, or a reference of its own for every level of pairs.  Each of the three, the lines between
them, ragged tails and a chunk of mixed heads are compared with the float64 oracle here, and the
recompute pass of a lean backward with the forward it rebuilds."""

import math

import pytest
import torch

from conftest import assert_close, rel_rms
from delta_feedback_experiment_b200 import chunk_precond_kda
from delta_feedback_experiment_b200.synthetic import INPUT_NAMES, make_inputs
from oracle.pkda_oracle import pkda_oracle_with_grads, pkda_recurrent_oracle

pytestmark = pytest.mark.gpu
D = 128

# Decay per token in log2 units (about; the raw gate spreads it by a seventh).  64 tokens: one reference row up to 112;
# 7 tokens: first and last row up to 112; 5 tokens up to 112 and two up to 45: by halves.
RATES = {"two strips meet": 2.0, "first and last row": 9.0, "line of the first": 13.5, "by halves": 15.5,
         "line of the second": 18.0, "own rows": 40.0, "everything vanishes": 300.0}


def _problem(T, rates, seed):
    H = len(rates)
    d = make_inputs(2, T, H, D, seed=seed, dist="production", dtype=torch.bfloat16, with_state=True)
    d["A_log"] = torch.tensor(rates).log().float()  # softplus(0) log2(e) = 1
    d["dt_bias"] = torch.zeros(H * D)
    return d


def _forward(d, **kw):
    t = {n: d[n].cuda() for n in INPUT_NAMES}
    return chunk_precond_kda(**t, initial_state=d["initial_state"].cuda(), initial_A_state=d["initial_A_state"].cuda(),
                             output_final_state=True, **kw)


@pytest.mark.parametrize("T", [64, 71, 193])
@pytest.mark.parametrize("which", [*RATES, "mixed"])
def test_reference_rows(which, T):
    rates = list(RATES.values()) if which == "mixed" else [RATES[which]] * 2
    d = _problem(T, rates, seed=700 + T)
    ref = pkda_recurrent_oracle(*[d[n] for n in INPUT_NAMES], initial_state=d["initial_state"],
                                initial_A_state=d["initial_A_state"], dtype=torch.float64)
    o, S, A = _forward(d)
    # bf16 operands and results: the limits every chunked forward test uses
    assert rel_rms(o, ref[0]) < 0.005, which
    assert_close(o, ref[0], 2e-2, f"{which} o")
    assert_close(S, ref[1], 2e-2, f"{which} S")
    assert_close(A, ref[2], 1e-4, f"{which} A")


@pytest.mark.parametrize("T", [64, 71, 193])
@pytest.mark.parametrize("which", [*RATES, "mixed"])
def test_gradients(which, T):
    """The chunk-parallel backward pairs the same strips; every gradient within the limits of the reference's own
    operator benchmark (relative rms)."""
    rates = list(RATES.values()) if which == "mixed" else [RATES[which]] * 2
    d = _problem(T, rates, seed=900 + T)
    ref = pkda_oracle_with_grads([d[n] for n in INPUT_NAMES], d["do"], initial_state=d["initial_state"],
                                 initial_A_state=d["initial_A_state"], dtype=torch.float64)
    leaves = {n: d[n].cuda().requires_grad_(True) for n in INPUT_NAMES}
    o, _, _ = chunk_precond_kda(**leaves, initial_state=d["initial_state"].cuda(), initial_A_state=d["initial_A_state"].cuda(),
                                output_final_state=True)
    limit = dict(q=0.007, k=0.008, v=0.007, A_log=0.025, dt_bias=0.02, log_atk_scale=0.02)
    for n, g in zip(INPUT_NAMES, torch.autograd.grad(o, list(leaves.values()), d["do"].cuda())):
        assert rel_rms(g, ref["d" + n]) < limit.get(n, 0.015), f"{which}: d{n} rel-rms {rel_rms(g, ref['d' + n]):.3e}"


@pytest.mark.parametrize("which", list(RATES))
def test_recompute_rebuilds_the_same_bits(which):
    d = _problem(135, [RATES[which], RATES["two strips meet"]], seed=801)
    do = torch.randn(2, 135, 2, D, generator=torch.Generator().manual_seed(5)).to(torch.bfloat16).cuda()

    def grads(disable_recompute):
        leaves = {n: d[n].cuda().requires_grad_(True) for n in INPUT_NAMES}
        o, _, _ = chunk_precond_kda(**leaves, initial_state=d["initial_state"].cuda(), initial_A_state=d["initial_A_state"].cuda(),
                                    output_final_state=True, disable_recompute=disable_recompute)
        return torch.autograd.grad(o, list(leaves.values()), do)

    for n, a, b in zip(INPUT_NAMES, grads(True), grads(False)):
        assert torch.equal(a, b), f"{which}: d{n}"
        assert math.isfinite(float(a.float().abs().max()))
