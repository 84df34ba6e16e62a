"""NaN and infinities are not hidden: a row and head whose exact result is not finite at a token is not finite there.
Every way a chunk can take (one direct block, strips, strips by halves, by level), full chunks and a ragged tail."""

import math

import pytest
import torch

from delta_feedback_experiment_b200 import chunk_precond_kda, ops
from delta_feedback_experiment_b200.synthetic import INPUT_NAMES, make_inputs
from oracle.pkda_oracle import pkda_oracle_with_grads

pytestmark = pytest.mark.gpu
RATES = [0.5, 4.0, 15.0, 40.0]
T, WHERE = 200, 75


def _bad(x):
    """[T, H]: anything not finite at that token and head of row 0."""
    return ~torch.isfinite(x[0].detach().cpu().double().reshape(T, len(RATES), -1)).all(-1)


@pytest.mark.parametrize("token", [WHERE, 195])
@pytest.mark.parametrize("which,value", [("q", math.nan), ("k", math.nan), ("k", math.inf), ("v", math.nan), ("v", -math.inf),
                                         ("g", math.nan), ("beta", math.nan), ("beta_atk", math.nan), ("g_atk", math.nan)])
def test_what_is_not_finite_shows(which, value, token):
    H = len(RATES)
    d = make_inputs(2, T, H, 128, seed=11, dist="production", dtype=torch.bfloat16, with_state=True)
    d["A_log"] = torch.tensor(RATES).log()
    d[which].view(2, T, H, -1)[0, token, :, -1] = value
    ref = pkda_oracle_with_grads([d[n] for n in INPUT_NAMES], d["do"], initial_state=d["initial_state"],
                                 initial_A_state=d["initial_A_state"])
    leaves = {n: d[n].cuda().requires_grad_(True) for n in INPUT_NAMES}
    o, S, A = chunk_precond_kda(**leaves, initial_state=d["initial_state"].cuda(), initial_A_state=d["initial_A_state"].cuda(),
                                output_final_state=True)
    got = dict(zip(["d" + n for n in INPUT_NAMES[:7]], torch.autograd.grad(o, [leaves[n] for n in INPUT_NAMES[:7]], d["do"].cuda())))
    assert ops.last_device_status() == 0 and ops.last_backward_status() == 0
    for n, x in {"o": o, **got}.items():
        hidden = (_bad(ref[n]) & ~_bad(x)).nonzero()
        assert not len(hidden), f"{n}: finite at (token, head) {hidden[:4].tolist()}"
        assert torch.isfinite(x[1].float()).all(), f"{n}: the other row"
    for n, x in (("final_state", S), ("final_A_state", A)):
        e = ref[n][0].flatten(1)
        assert not (~torch.isfinite(e).all(1) & torch.isfinite(x[0].cpu().flatten(1)).all(1)).any(), n
        assert torch.isfinite(x[1]).all(), n
    assert not _bad(o)[:token // 64 * 64].any()  # (what comes before the chunk does not see it)
