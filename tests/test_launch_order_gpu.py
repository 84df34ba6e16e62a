"""A kernel that runs beside the one in front of it reads what earlier kernels left before it has waited for anything.
Only an ordinary (not programmatic) launch between the two makes that complete and visible, so every such reader has one
behind its last writer.  Shown on the captured launches: a programmatic launch is a programmatic edge of the graph."""

from typing import NamedTuple

import pytest
import torch

from delta_feedback_experiment_b200 import _lib, chunk_precond_kda
from delta_feedback_experiment_b200.synthetic import INPUT_NAMES, make_inputs

pytestmark = pytest.mark.gpu


class Launch(NamedTuple):
    name: str     # of the kernel, mangled; copies and fills have none
    early: bool   # a programmatic launch
    grid: int     # CTAs along x
    threads: int  # of a CTA


def captured_launches(fn):
    """Everything that ``fn`` launches, in stream order."""
    from cuda.bindings import driver

    def ok(result):
        assert result[0] == driver.CUresult.CUDA_SUCCESS, result[0]
        return result[1:]

    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        fn()
    raw = driver.CUgraph(graph.raw_cuda_graph())
    nodes = ok(driver.cuGraphGetNodes(raw, ok(driver.cuGraphGetNodes(raw, 0))[1]))[0]
    n_edges = ok(driver.cuGraphGetEdges_v2(raw, 0))[3]
    src, dst, data = ok(driver.cuGraphGetEdges_v2(raw, n_edges))[:3]
    follows, early = {int(a): int(b) for a, b in zip(src, dst)}, {}
    for b, e in zip(dst, data):
        early[int(b)] = e.type == int(driver.CUgraphDependencyType.CU_GRAPH_DEPENDENCY_TYPE_PROGRAMMATIC)
    by_id = {int(x): x for x in nodes}
    at = next(i for i in by_id if i not in early)
    launches = []
    while at is not None:
        name, grid, threads = "", 0, 0
        if ok(driver.cuGraphNodeGetType(by_id[at]))[0] == driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            params = ok(driver.cuGraphKernelNodeGetParams(by_id[at]))[0]
            raw_name = driver.cuFuncGetName(params.func) if int(params.func) else driver.cuKernelGetName(params.kern)
            name, grid, threads = ok(raw_name)[0].decode(), params.gridDimX, params.blockDimX
        launches.append(Launch(name, early.get(at, False), grid, threads))
        at = follows.get(at)
    assert len(launches) == len(by_id)  # one stream, one chain
    return launches


def _exact(d):
    x = {n: d[n].detach().requires_grad_(True) for n in INPUT_NAMES}
    o, _, _ = chunk_precond_kda(**x)
    return torch.autograd.grad(o, list(x.values()), d["do"])


def _lean(d):
    x = {n: d[n].detach().requires_grad_(True) for n in INPUT_NAMES}
    o, _, _ = chunk_precond_kda(**x, disable_recompute=False)
    return torch.autograd.grad(o, list(x.values()), d["do"])


def _inputs(step, seed=1, H=4):
    if step is _exact:
        d = make_inputs(2, 200, H, 64, seed=seed, dist="unit", dtype=torch.float32)
    else:
        d = make_inputs(2, 200, H, 128, seed=seed, dist="production", dtype=torch.bfloat16)
    return {n: t.cuda() for n, t in d.items() if torch.is_tensor(t)}


@pytest.mark.parametrize("step,writer,reader", [(_exact, "pkda_recurrent_grad_kernel", "pkda_recurrent_bwd_reduce_kernel"),
                                                (_lean, "pkda_intra_fwd_tc_kernel", "pkda_scan_bwd"),
                                                (_lean, "pkda_scan_bwd", "pkda_intra_bwd_kernel"),
                                                (_lean, "pkda_intra_bwd_kernel", "pkda_param_reduce_kernel")])
def test_an_ordinary_launch_stands_between_writer_and_reader(step, writer, reader):
    d = _inputs(step)
    step(d)
    torch.cuda.synchronize()
    launches = captured_launches(lambda: step(d))
    names = [x.name for x in launches]
    r = next(i for i, name in enumerate(names) if reader in name)
    w = max(i for i, name in enumerate(names[:r]) if writer in name)
    assert launches[r].early
    assert any(not x.early for x in launches[w + 1:r]), names[w:r + 1]


def test_exact_backwards_of_changing_inputs_in_a_row():
    """The partial sums lie where those of the call before lay: no gradient of a parameter may take any of them."""
    inputs = [_inputs(_exact, seed) for seed in (1, 2)]
    want = []
    for d in inputs:
        want.append(_exact(d))
        torch.cuda.synchronize()
    for _ in range(20):
        got = [_exact(d) for d in inputs]
        for g, w in zip(got, want):
            for name, a, b in zip(INPUT_NAMES, g, w):
                assert torch.equal(a, b), name


@pytest.mark.parametrize("pinned", [(), ("scan_fwd",), ("scan_bwd",)])
def test_a_scan_with_nothing_beside_it_takes_all_its_columns(pinned):
    """16 units: four CTAs each for the recompute pass's scan where the reverse scan runs beside it, else eight (the pinned
    mma.sync scan: four of 32 value columns)."""
    d = _inputs(_lean, H=8)
    for stage in pinned:
        _lib.set_variant(stage, True)
    try:
        _lean(d)
        torch.cuda.synchronize()
        launches = captured_launches(lambda: _lean(d))
    finally:
        for stage in pinned:
            _lib.set_variant(stage, False)
    assert [x.grid for x in launches if "scan_fwd" in x.name] == {(): [128, 64], ("scan_fwd",): [64, 64], ("scan_bwd",): [128, 128]}[pinned]


@pytest.mark.parametrize("H,D,early", [(20, 32, False), (4, 64, True), (20, 64, False)])
def test_the_exact_reverse_scan_is_placed_when_the_forward_has_ended(H, D, early):
    """Its CTAs are a long chain each: where two fit an SM they must not be laid beside one another while others stay idle."""
    d = {n: t.cuda() for n, t in make_inputs(2, 200, H, D, seed=1, dist="unit", dtype=torch.float32).items() if torch.is_tensor(t)}
    _exact(d)
    torch.cuda.synchronize()
    assert [x.early for x in captured_launches(lambda: _exact(d)) if "dscan" in x.name] == [early]
