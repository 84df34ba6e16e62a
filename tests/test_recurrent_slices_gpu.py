"""Edges of the column-sliced token-by-token kernels: blocks of 8 staged tokens, checkpoints every
32 tokens, both slice widths, every head width, several CTAs per (sequence, head)."""

import pytest
import torch

from conftest import assert_close, rel_rms
from delta_feedback_experiment_b200 import chunk_precond_kda, fused_recurrent_precond_kda
from delta_feedback_experiment_b200.synthetic import INPUT_NAMES, make_inputs
from oracle.pkda_oracle import pkda_oracle_with_grads

pytestmark = pytest.mark.gpu


def _kw(d):
    return {n: d[n] for n in INPUT_NAMES}


def _grads(d, S0, A0, do, dS, lean, cu=None):
    leaves = {n: d[n].cuda().requires_grad_(True) for n in INPUT_NAMES}
    S0, A0 = (t.cuda().requires_grad_(True) for t in (S0, A0))
    o, S, A = chunk_precond_kda(**leaves, initial_state=S0, initial_A_state=A0, output_final_state=True,
                                disable_recompute=not lean, cu_seqlens=cu)
    g = torch.autograd.grad([o, S], [*leaves.values(), S0, A0], [do.cuda(), dS.cuda()])
    return [o, S, A, *g]


@pytest.mark.parametrize("D,T,B,H", [(8, 9, 2, 3), (16, 33, 1, 2), (32, 65, 2, 1), (64, 7, 1, 4), (64, 96, 3, 5),
                                     (64, 33, 20, 4), (128, 40, 1, 2), (128, 31, 5, 32)])
def test_exact_forward_and_backward(D, T, B, H):
    d = make_inputs(B, T, H, D, seed=D + T, dist="production", dtype=torch.float32, with_state=True)
    dS = torch.randn(B, H, D, D, generator=torch.Generator().manual_seed(1)) * 0.1
    ref = pkda_oracle_with_grads([d[n] for n in INPUT_NAMES], d["do"], initial_state=d["initial_state"],
                                 initial_A_state=d["initial_A_state"], d_final_state=dS, dtype=torch.float64)
    names = ["o", "final_state", "final_A_state", *("d" + n for n in INPUT_NAMES), "dinitial_state",
             "dinitial_A_state"]
    runs = [_grads(d, d["initial_state"], d["initial_A_state"], d["do"], dS, lean) for lean in (False, True)]
    for n, a, b in zip(names, *runs):
        assert rel_rms(a, b) < 1e-5, n       # kept and repeated forward by-products
        if n in ("dA_log", "ddt_bias", "dlog_atk_scale"):   # sums whose terms cancel
            assert rel_rms(a, ref[n]) < 1e-3, n
        else:
            gate = n in ("dg", "dg_atk", "dbeta_atk", "dinitial_A_state")
            assert_close(a, ref[n], 1e-3 if gate else 1e-4, n)


@pytest.mark.parametrize("B,H,D,T", [(2, 2, 128, 20), (4, 16, 128, 48), (40, 8, 128, 3), (40, 8, 128, 8), (3, 4, 64, 17)])
def test_in_place_states_equal_separate_ones(B, H, D, T):
    """Several CTAs of a unit read the preconditioner state that one of them overwrites."""
    d = make_inputs(B, T, H, D, seed=B + T, dist="production", dtype=torch.bfloat16, with_state=True)
    c = {n: v.cuda() for n, v in d.items()}
    want = fused_recurrent_precond_kda(**_kw(c), initial_state=c["initial_state"],
                                       initial_A_state=c["initial_A_state"], output_final_state=True)
    S, A = c["initial_state"].clone(), c["initial_A_state"].clone()
    got = fused_recurrent_precond_kda(**_kw(c), initial_state=S, initial_A_state=A, output_final_state=True,
                                      inplace_state=True)
    assert got[1] is S and got[2] is A
    for x, y in zip(got, want):
        assert torch.equal(x, y)


def test_packed_sequences_shorter_than_a_block():
    offs = [0, 1, 9, 41, 41, 73, 200]
    D, H, N = 64, 2, 6
    d = make_inputs(1, offs[-1], H, D, seed=5, dist="unit", dtype=torch.float32, n_states=N, with_state=True)
    dS = torch.randn(N, H, D, D, generator=torch.Generator().manual_seed(2)) * 0.1
    ref = pkda_oracle_with_grads([d[n] for n in INPUT_NAMES], d["do"], initial_state=d["initial_state"],
                                 initial_A_state=d["initial_A_state"], d_final_state=dS, cu_seqlens=offs,
                                 dtype=torch.float64)
    cu = torch.tensor(offs, dtype=torch.int32, device="cuda")
    got = _grads(d, d["initial_state"], d["initial_A_state"], d["do"], dS, False, cu)
    for n, a in zip(["o", "final_state", "final_A_state", *("d" + n for n in INPUT_NAMES), "dinitial_state",
                     "dinitial_A_state"], got):
        assert rel_rms(a, ref[n]) < 1e-4, n
