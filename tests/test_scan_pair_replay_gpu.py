"""Replays of a captured lean step, each of which has to produce its own results: the outputs are overwritten and the inputs
changed in front of every one."""

import pytest
import torch

from delta_feedback_experiment_b200 import chunk_precond_kda, ops
from delta_feedback_experiment_b200.synthetic import INPUT_NAMES, make_inputs

pytestmark = pytest.mark.gpu
D = 128


def _step(d, lean):
    x = {n: d[n].detach().requires_grad_(True) for n in INPUT_NAMES}
    S0, A0 = (d[n].detach().requires_grad_(True) for n in ("initial_state", "initial_A_state"))
    o, S, _ = chunk_precond_kda(**x, initial_state=S0, initial_A_state=A0, output_final_state=True, disable_recompute=not lean)
    return (o, S, *torch.autograd.grad([o, S], [*x.values(), S0, A0], [d["do"], d["dS"]]))


# 12 and 24 units by columns side by side, 50 on the tensor-memory scans
@pytest.mark.parametrize("B,H", [(3, 4), (6, 4), (10, 5)])
def test_every_replay_makes_its_own_results(B, H):
    inputs = []
    for seed in (9, 10):
        d = make_inputs(B, 500, H, D, seed=seed, dist="production", dtype=torch.bfloat16, with_state=True)
        d = {n: t.cuda() for n, t in d.items() if torch.is_tensor(t)}
        d["dS"] = torch.randn(B, H, D, D, device="cuda") * 0.1
        inputs.append(d)
    want = [_step(d, False) for d in inputs]
    live = {n: t.clone() for n, t in inputs[0].items()}
    _step(live, True)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = _step(live, True)
    for turn in range(4):
        for t in got:
            t.fill_(float("nan"))
        for n, t in inputs[turn % 2].items():
            live[n].copy_(t)
        graph.replay()
        torch.cuda.synchronize()
        assert ops.last_device_status() == 0 and ops.last_backward_status() == 0
        for a, b in zip(got, want[turn % 2]):
            assert torch.equal(a, b)
