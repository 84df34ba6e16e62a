"""Edges of the control epilogue's backward: odd head counts (no paired moves), head counts past the limits of
the rows taken per turn, rows that do not fill a turn."""

import pytest
import torch

from conftest import assert_close, rel_rms
from oracle.pkda_layer_oracle import controls_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,H,D", [(1, 1, 8), (9, 3, 16), (5, 7, 33), (17, 256, 8), (6, 520, 4), (21000, 4, 2)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_controls_backward_edges(rows, H, D, dtype):
    from delta_feedback_experiment_b200.layer_ops import pkda_controls
    gen = torch.Generator().manual_seed(rows + H)
    packed = torch.randn(rows, 2 * D + 3 * H, generator=gen).to(dtype)
    A = torch.log(torch.empty(H).uniform_(1, 8, generator=gen))
    b = 0.3 * torch.randn(H, generator=gen)
    cot = [torch.randn(rows, n, generator=gen).to(t) for n, t in
           ((D, dtype), (H, dtype), (H, torch.float32), (H, dtype), (D, dtype))]
    leaves = [t.float().requires_grad_(True) for t in (packed, A, b)]
    ref = torch.autograd.grad(sum((o * c.float()).sum() for o, c in zip(controls_oracle(*leaves, D), cot)), leaves)
    dev = [t.cuda().requires_grad_(True) for t in (packed, A, b)]
    got = torch.autograd.grad(pkda_controls(*dev, D), dev, [c.cuda() for c in cot])
    rtol = 2e-2 if dtype == torch.bfloat16 else 1e-4
    assert_close(got[0], ref[0], rtol, "d_packed")
    for x, y in zip(got[1:], ref[1:]):
        assert rel_rms(x, y) < (1e-2 if dtype == torch.bfloat16 else 1e-4)
