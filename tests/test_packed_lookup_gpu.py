"""Chunk lookup of packed batches at the counts where its steps change (one sequence, a full warp of
candidates, one more, several narrowing steps): every sequence must come out as it does alone, bit for bit."""

import pytest
import torch

from delta_feedback_experiment_b200.synthetic import make_inputs

pytestmark = pytest.mark.gpu

TOKEN_INPUTS = ("q", "k", "v", "g", "g_atk", "beta_atk", "beta")
PARAMS = ("A_log", "dt_bias", "log_atk_scale")


def _run(d, do, cu=None):
    from delta_feedback_experiment_b200 import chunk_precond_kda
    leaves = {n: d[n].cuda().requires_grad_(True) for n in TOKEN_INPUTS}
    o, _, _ = chunk_precond_kda(**leaves, **{n: d[n].cuda() for n in PARAMS},
                                cu_seqlens=None if cu is None else torch.tensor(cu, dtype=torch.int32, device="cuda"))
    return [o, *torch.autograd.grad(o, list(leaves.values()), do.cuda())]


@pytest.mark.parametrize("n_seqs", [1, 31, 32, 33, 97, 300])
def test_packed_sequences_match_their_own(n_seqs):
    gen = torch.Generator().manual_seed(n_seqs)
    lens = torch.randint(1, 140, (n_seqs,), generator=gen).tolist()
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    d = make_inputs(1, cu[-1], 2, 128, seed=n_seqs, dist="unit", dtype=torch.bfloat16)
    packed = _run(d, d["do"], cu)
    for i in range(n_seqs):
        rows = slice(cu[i], cu[i + 1])
        one = {n: (d[n][:, rows].contiguous() if n in TOKEN_INPUTS else d[n]) for n in TOKEN_INPUTS + PARAMS}
        alone = _run(one, d["do"][:, rows].contiguous())
        for name, a, b in zip(("o",) + TOKEN_INPUTS, packed, alone):
            assert torch.equal(a[:, rows], b), (i, name)
