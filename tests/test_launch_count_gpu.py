"""The launch count that the library reports against the kernel nodes of a captured graph, on every route that
puts its own set of kernels in front of the intra stage."""

import pytest
import torch
from cuda.bindings import runtime

from delta_feedback_experiment_b200 import chunk_precond_kda, ops, pkda_recurrence
from delta_feedback_experiment_b200.synthetic import INPUT_NAMES, make_inputs

pytestmark = pytest.mark.gpu
D = 128


def _kernels(call):
    """(kernel nodes of the captured call, kernels the library counted for it)"""
    call()  # (what the first call of a process sets up)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    before = ops.LAUNCHES
    with torch.cuda.graph(graph):
        keep = call()
    counted = ops.LAUNCHES - before
    handle = runtime.cudaGraph_t(graph.raw_cuda_graph())
    n = runtime.cudaGraphGetNodes(handle)[-1]
    nodes = runtime.cudaGraphGetNodes(handle, n)[1][:n]
    kinds = [runtime.cudaGraphNodeGetType(node)[1] for node in nodes]
    del keep
    return sum(k == runtime.cudaGraphNodeType.cudaGraphNodeTypeKernel for k in kinds), counted


@pytest.mark.parametrize("B,T,H", [(1, 65, 1), (2, 200, 16), (1, 1601, 2)])
@pytest.mark.parametrize("lean", [False, True])
def test_dense(B, T, H, lean):
    d = {n: t.cuda() for n, t in make_inputs(B, T, H, D, seed=T).items()}
    x, const = [d[n] for n in INPUT_NAMES], (D ** -0.5, 1.5, 1e-6)
    nodes, counted = _kernels(lambda: pkda_recurrence(*x, *const, lean))
    assert nodes == counted
    _, saved = pkda_recurrence(*x, *const, lean)
    nodes, counted = _kernels(lambda: torch.ops.delta_feedback.pkda_recurrence_backward(
        *x, saved, d["do"], *const, None, lean))
    assert nodes == counted


def test_packed():
    d = {n: t.cuda() for n, t in make_inputs(1, 300, 2, D, seed=9).items()}
    cu = torch.tensor([0, 100, 300], dtype=torch.int32, device="cuda")
    nodes, counted = _kernels(lambda: chunk_precond_kda(**{n: d[n] for n in INPUT_NAMES}, cu_seqlens=cu))
    assert nodes == counted
