"""The operators are differentiable once.  A second derivative must be refused, not left out: shapes only, on the
meta device, where the operators' autograd kernels run and no CUDA kernel does."""

import pytest
import torch

from delta_feedback_experiment_b200 import pkda_norm_gate, pkda_qkv_conv, pkda_recurrence

B, T, H, D = 2, 70, 3, 128


def _meta(*shape, dtype=torch.bfloat16):
    return torch.empty(shape, device="meta", dtype=dtype, requires_grad=True)


def _conv():
    leaves = [_meta(B, T, 3 * H * D), _meta(3 * H * D, 4, dtype=torch.float32)]
    return leaves, pkda_qkv_conv(*leaves, D, 2 * H * D, 1e-6)[0]


def _gate():
    leaves = [_meta(B, T, H, D), _meta(B, T, H, D), _meta(D, dtype=torch.float32)]
    return leaves, pkda_norm_gate(*leaves, 1e-6)[0]


def _recurrence(lean):
    f32 = torch.float32
    leaves = [*(_meta(B, T, H, D) for _ in range(4)), _meta(B, T, H, dtype=f32), _meta(B, T, H), _meta(B, T, H),
              _meta(H, dtype=f32), _meta(H * D, dtype=f32), _meta(H, dtype=f32)]
    return leaves, pkda_recurrence(*leaves, D ** -0.5, 1.5, 1e-6, lean)[0]


CASES = {"conv": _conv, "gate": _gate, "recurrence": lambda: _recurrence(False),
         "lean recurrence": lambda: _recurrence(True)}


@pytest.mark.parametrize("name", CASES)
def test_second_derivative_is_refused(name):
    leaves, out = CASES[name]()
    first = torch.autograd.grad(out, leaves, torch.empty_like(out), create_graph=True)
    assert all(g.shape == t.shape and g.dtype == t.dtype and g.requires_grad for g, t in zip(first, leaves))
    with pytest.raises(RuntimeError, match="_backward"):
        torch.autograd.grad(first[0].sum(), leaves[0])


@pytest.mark.parametrize("name", CASES)
def test_first_derivative_records_nothing(name):
    leaves, out = CASES[name]()
    first = torch.autograd.grad(out, leaves, torch.empty_like(out))
    assert not any(g.requires_grad for g in first)
