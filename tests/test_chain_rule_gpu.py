"""Where the forward chains the preconditioner state inside the intra kernel: one launch in front of it, two where
it does not.  Either side of every line of the rule, rows of up to 65,600 tokens of one or two heads a row."""

import pytest
import torch

from delta_feedback_experiment_b200 import _lib, chunk_precond_kda

pytestmark = pytest.mark.gpu
D = 128


def _stages(B, T, H):
    g = torch.Generator(device="cuda").manual_seed(1)

    def rn(*size):
        return torch.randn(*size, generator=g, device="cuda", dtype=torch.bfloat16)

    x = rn(B, T, H, D)
    s = torch.rand(B, T, H, generator=g, device="cuda")
    _lib.stage_timing(True)
    try:
        chunk_precond_kda(x, x, x, x, -s, s.bfloat16(), s.bfloat16(), A_log=torch.zeros(H, device="cuda"),
                          dt_bias=torch.zeros(H * D, device="cuda"), log_atk_scale=torch.zeros(H, device="cuda"))
        torch.cuda.synchronize()
        return set(_lib.stage_timing_read())
    finally:
        _lib.stage_timing(False)


@pytest.mark.parametrize("units,longest", [(1, 1536), (7, 1536), (8, 16384), (23, 16384), (24, 65536), (31, 65536)])
def test_lines(units, longest):
    for T, chained in ((longest, True), (longest + 1, False)):
        stages = _stages(units, T, 1)
        assert ("chain_init" in stages) == chained and ("atk_carry" in stages) != chained, (units, T)


def test_many_units_chain_at_any_length():
    assert "chain_init" in _stages(16, 65600, 2)
