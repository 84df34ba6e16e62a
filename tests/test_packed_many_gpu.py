"""Packed batches at the counts where the local preconditioner scan starts to halve its candidates: every sequence,
empty ones among them, must come out as it does alone, bit for bit."""

import pytest
import torch

from delta_feedback_experiment_b200 import chunk_precond_kda
from delta_feedback_experiment_b200.synthetic import INPUT_NAMES, make_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_seqs", [256, 257, 511, 1030])
def test_each_sequence_matches_its_own(n_seqs):
    lens = torch.randint(0, 20, (n_seqs,), generator=torch.Generator().manual_seed(n_seqs))
    lens[[3, n_seqs // 2]], lens[[0, -1]] = 130, 9
    cu = [0, *lens.cumsum(0).tolist()]
    d = {n: t.cuda() for n, t in make_inputs(1, cu[-1], 2, 128, seed=n_seqs, dist="unit").items()}
    o, S, A = chunk_precond_kda(**{n: d[n] for n in INPUT_NAMES}, output_final_state=True,
                                cu_seqlens=torch.tensor(cu, dtype=torch.int32, device="cuda"))
    assert A[lens == 0].abs().sum() == 0 and S[lens == 0].abs().sum() == 0
    for i in range(n_seqs):
        rows = slice(cu[i], cu[i + 1])
        if cu[i] == cu[i + 1]:
            continue
        one = {n: (d[n][:, rows].contiguous() if d[n].dim() > 1 else d[n]) for n in INPUT_NAMES}
        alone = chunk_precond_kda(**one, output_final_state=True)
        for a, b in zip((o[:, rows], S[i:i + 1], A[i:i + 1]), alone):
            assert torch.equal(a, b), i
