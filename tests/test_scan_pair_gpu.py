"""The two state scans of a lean backward run side by side while both fit the chip, on fewer CTAs a unit than either takes
alone.  Every split multiplies the same operands in the same order, so a lean backward keeps the bits of a retaining
one, which runs its one scan alone."""

import pytest
import torch

from delta_feedback_experiment_b200 import chunk_precond_kda, ops
from delta_feedback_experiment_b200.synthetic import INPUT_NAMES, make_inputs

pytestmark = pytest.mark.gpu
D = 128


def _grads(d, dS, lean, cu):
    x = {n: d[n].cuda().detach().requires_grad_(True) for n in INPUT_NAMES}
    S0, A0 = (d[n].cuda().detach().requires_grad_(True) for n in ("initial_state", "initial_A_state"))
    o, S, _ = chunk_precond_kda(**x, initial_state=S0, initial_A_state=A0, output_final_state=True, cu_seqlens=cu,
                                disable_recompute=not lean)
    grads = torch.autograd.grad([o, S], [*x.values(), S0, A0], [d["do"].cuda(), dS])
    assert ops.last_backward_status() == 0
    return o, S, *grads


# CTAs a unit on 148 SMs: 8 + 8 up to 9 units, 4 + 8 up to 12, 4 + 4 up to 18, 2 + 4 up to 24, 2 + 2 up to 37, the
# tensor-memory scans up to 74; one after the other from there.
@pytest.mark.parametrize("B,H", [(1, 1), (3, 3), (5, 2), (6, 2), (13, 1), (6, 3), (19, 1), (8, 3), (5, 5), (37, 1), (19, 2),
                                 (37, 2), (25, 3)])
@pytest.mark.parametrize("T", [64, 330])
def test_lean_equals_retaining(B, H, T):
    d = make_inputs(B, T, H, D, seed=T + B, dist="production", dtype=torch.bfloat16, with_state=True)
    dS = torch.randn(B, H, D, D, generator=torch.Generator().manual_seed(B)).cuda() * 0.1
    for a, b in zip(_grads(d, dS, True, None), _grads(d, dS, False, None)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("lens", [[1, 700, 64, 3], [130, 64, 1, 77, 200, 65, 63, 190]])
def test_packed(lens):
    offs = torch.tensor([0, *lens]).cumsum(0)
    d = make_inputs(1, int(offs[-1]), 3, D, seed=11, dist="unit", dtype=torch.bfloat16, with_state=True, n_states=len(lens))
    dS = torch.randn(len(lens), 3, D, D, generator=torch.Generator().manual_seed(3)).cuda() * 0.1
    cu = offs.int().cuda()
    for a, b in zip(_grads(d, dS, True, cu), _grads(d, dS, False, cu)):
        assert torch.equal(a, b)


def test_captured():
    """Replays of a captured lean step: what follows the scans waits for both."""
    d = make_inputs(3, 500, 4, D, seed=9, dist="production", dtype=torch.bfloat16, with_state=True)
    d = {n: t.cuda() for n, t in d.items()}
    dS = torch.randn(3, 4, D, D, device="cuda") * 0.1
    want = _grads(d, dS, False, None)
    _grads(d, dS, True, None)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        x = {n: d[n].detach().requires_grad_(True) for n in INPUT_NAMES}
        S0, A0 = (d[n].detach().requires_grad_(True) for n in ("initial_state", "initial_A_state"))
        o, S, _ = chunk_precond_kda(**x, initial_state=S0, initial_A_state=A0, output_final_state=True, disable_recompute=False)
        got = (o, S, *torch.autograd.grad([o, S], [*x.values(), S0, A0], [d["do"], dS]))
    for _ in range(3):
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            assert torch.equal(a, b)
