"""The token-by-token scans ask for a token's row vectors one or two tokens ahead, by the number of chain warps in a CTA (which
follows the number of units): at both sides of every line the form that is meant runs, and a unit has the same bits in both."""

import re

import pytest
import torch

from delta_feedback_experiment_b200 import chunk_precond_kda
from delta_feedback_experiment_b200.synthetic import INPUT_NAMES, make_inputs
from test_launch_order_gpu import captured_launches

pytestmark = pytest.mark.gpu


def _step(d, rows=None):
    x = {n: (d[n] if rows is None or n in ("A_log", "dt_bias", "log_atk_scale") else d[n][:rows]) for n in INPUT_NAMES}
    x = {n: t.detach().requires_grad_(True) for n, t in x.items()}
    o, S, _ = chunk_precond_kda(**x, output_final_state=True, disable_recompute=True)
    grads = torch.autograd.grad([o, S], [x[n] for n in INPUT_NAMES[:7]], [d["do"][:rows], d["dS"][:rows]])
    return o, S, *grads


# 148 SMs.  Chain warps in a CTA: one up to 9 units of 64 rows and 18 of 32, at 64 rows four up to 37 units
@pytest.mark.parametrize("D,units,forward,reverse", [(64, 9, True, True), (64, 10, False, True), (64, 37, False, True),
                                                     (64, 38, False, False), (64, 150, False, False), (32, 18, True, False),
                                                     (32, 19, False, False), (32, 150, False, False), (16, 3, False, False),
                                                     (128, 2, False, False)])
def test_form_and_bits(D, units, forward, reverse):
    d = make_inputs(units, 67, 1, D, seed=units, dist="unit", dtype=torch.float32)
    d = {n: t.cuda() for n, t in d.items() if torch.is_tensor(t)}
    d["dS"] = torch.randn(units, 1, D, D, device="cuda") * 0.1
    all_units = _step(d)
    for a, b in zip(all_units, _step(d, 1)):
        assert torch.equal(a[:1], b)
    torch.cuda.synchronize()
    launches = captured_launches(lambda: _step(d))
    one = lambda pattern: [m.group(1) == "1" for m in (re.search(pattern, x.name) for x in launches) if m]
    assert one(r"recurrent_kernelI.*Lb1ELb([01])EEE") == [forward]
    assert one(r"dscan_kernelI.*Lb([01])EEE") == [reverse]


@pytest.mark.parametrize("units,threads", [(148, 192), (149, 160)])
def test_producers_are_spread_only_on_an_sm_of_their_own(units, threads):
    """8 rows: one chain warp and four producers' warps a CTA, and an empty one where the producers keep off the chain's scheduler."""
    d = make_inputs(units, 67, 1, 8, seed=units, dist="unit", dtype=torch.float32)
    d = {n: t.cuda() for n, t in d.items() if torch.is_tensor(t)}
    d["dS"] = torch.randn(units, 1, 8, 8, device="cuda") * 0.1
    for a, b in zip(_step(d), _step(d, 1)):
        assert torch.equal(a[:1], b)
    torch.cuda.synchronize()
    launches = captured_launches(lambda: _step(d))
    assert [x.threads for x in launches if "recurrent_kernel" in x.name or "dscan_kernel" in x.name] == [threads, threads]
