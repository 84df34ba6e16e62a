"""A token's decay and write-key factor must not depend on the kernel that a call's size takes: the column-sliced
scan (few units) and the whole-state kernel (more units than SMs, few tokens) form them from the same functions, bit
for bit.  The inputs make the factors stand bare in the state: with a zero state and v = 1, S = beta * kw after one
token; with k = 0 and an all-one state, S = the product of the decays."""

import pytest
import torch

from delta_feedback_experiment_b200 import fused_recurrent_precond_kda
from delta_feedback_experiment_b200.synthetic import INPUT_NAMES, make_inputs

pytestmark = pytest.mark.gpu
ROWS, H = 64, 8        # 512 units; one row alone has 8


def _states(d, rows):
    args = {n: (d[n][rows] if d[n].dim() > 1 else d[n]).cuda() for n in INPUT_NAMES}
    S0 = None if "S0" not in d else d["S0"][rows].cuda()
    return fused_recurrent_precond_kda(**args, initial_state=S0, output_final_state=True)[1].cpu()


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("dist", ["unit", "production"])
@pytest.mark.parametrize("factor", ["write key", "decay"])
def test_factors_do_not_depend_on_the_kernel(D, dist, factor):
    tokens = 1 if factor == "write key" else 2   # one token on a given state is the decoding kernel's
    d = make_inputs(ROWS, tokens, H, D, seed=D, dist=dist, dtype=torch.float32)
    if factor == "write key":
        d["v"] = torch.ones_like(d["v"])
    else:
        d["k"], d["S0"] = torch.zeros_like(d["k"]), torch.ones(ROWS, H, D, D)
    many = _states(d, slice(0, ROWS))
    for row in (0, 1, ROWS - 1):
        assert torch.equal(_states(d, slice(row, row + 1)), many[row:row + 1]), row
