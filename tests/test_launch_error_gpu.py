"""A launch that the driver refuses is an error of the call, also when a later launch of the same call succeeds."""

import pytest
import torch

from delta_feedback_experiment_b200 import layer_ops

pytestmark = pytest.mark.gpu


def _conv_backward(rows):
    x = torch.randn(rows, 1, 24, device="cuda", dtype=torch.bfloat16)
    d = [torch.randn(rows, 1, 8, device="cuda", dtype=torch.bfloat16) for _ in range(3)]
    w = torch.randn(24, 4, device="cuda")
    return layer_ops.qkv_conv_backward(x, w, *d, 8, 16, 1e-6)


def test_refused_first_launch_is_reported():
    """65,536 rows are one block of grid.y too many for the convolution's walk; the sum of the weight gradient behind it is
    a valid launch."""
    with pytest.raises(RuntimeError):
        _conv_backward(65536)
    torch.cuda.synchronize()
    dx, dw = _conv_backward(65535)  # the largest that is taken; the error above is not reported a second time
    assert torch.isfinite(dx.float()).all() and torch.isfinite(dw).all()
