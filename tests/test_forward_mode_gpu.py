"""Forward-mode differentiation is not implemented and has to say so: a tangent must not be dropped on the way."""

import pytest
import torch
import torch.autograd.forward_ad as fwad

from delta_feedback_experiment_b200 import chunk_precond_kda
from delta_feedback_experiment_b200.synthetic import INPUT_NAMES, make_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,dtype", [(128, torch.bfloat16), (32, torch.float32)])
@pytest.mark.parametrize("name", ["q", "dt_bias", "initial_state"])
def test_tangent_is_refused(D, dtype, name):
    d = {n: t.cuda() for n, t in make_inputs(1, 70, 2, D, seed=1, dist="unit", dtype=dtype, with_state=True).items()}
    names = (*INPUT_NAMES, "initial_state", "initial_A_state")
    with fwad.dual_level():
        args = {n: fwad.make_dual(d[n], torch.ones_like(d[n])) if n == name else d[n] for n in names}
        with pytest.raises(RuntimeError, match="jvp"):
            chunk_precond_kda(**args, output_final_state=True)
