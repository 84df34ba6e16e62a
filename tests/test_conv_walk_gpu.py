"""The convolution's token walks at the sizes where they can go wrong: rows shorter than a step, spans that
end inside, at and right after a step or a span, the longest span, channel counts that leave lanes, warps
and whole 16-byte pieces of the last block idle, and every width of the head sums."""

import pytest
import torch

from conftest import assert_close, rel_rms
from oracle import pkda_layer_oracle

pytestmark = pytest.mark.gpu

SHAPES = [
    # B, T, H, D, taps
    (2, 1, 1, 8, 4), (1, 4, 3, 8, 3), (2, 5, 1, 16, 4), (1, 15, 1, 128, 4), (1, 16, 2, 32, 2), (1, 17, 3, 64, 4),
    (3, 61, 2, 16, 4), (2, 65, 1, 128, 4), (1, 127, 7, 8, 4), (1, 513, 1, 64, 4),
    (300, 130, 1, 128, 4),  # enough CTAs for the longest span
]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_walk_matches_oracle(shape, dtype):
    from delta_feedback_experiment_b200 import layer_ops
    B, T, H, D, taps = shape
    W = H * D
    gen = torch.Generator().manual_seed(B + T + W)
    x = torch.randn(B, T, 3 * W, generator=gen).to(dtype)
    w = torch.randn(3 * W, taps, generator=gen) * 0.5
    grads = [torch.randn(B, T, W, generator=gen).to(dtype) for _ in range(3)]
    xo, wo = x.float().requires_grad_(True), w.clone().requires_grad_(True)
    ref = pkda_layer_oracle.qkv_conv_oracle(xo, wo, D, 2 * W, 1e-6)
    rdx, rdw = torch.autograd.grad(sum((r * d.float()).sum() for r, d in zip(ref, grads)), [xo, wo])
    got = layer_ops.qkv_conv_forward(x.cuda(), w.cuda(), D, 2 * W, 1e-6)
    dx, dw = layer_ops.qkv_conv_backward(x.cuda(), w.cuda(), *[d.cuda() for d in grads], D, 2 * W, 1e-6)
    rtol = 2e-2 if dtype == torch.bfloat16 else 1e-4
    for key, a, e in zip("qkv", got, ref):
        assert_close(a, e, rtol, f"{shape}:{key}")
    assert_close(dx, rdx, rtol, f"{shape}:dx")
    assert rel_rms(dw, rdw) < (1e-2 if dtype == torch.bfloat16 else 1e-5), rel_rms(dw, rdw)
