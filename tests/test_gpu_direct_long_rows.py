"""Direct joins of few rows with many: rows of the result of up to 70,001 columns, in all forms of output."""
import numpy as np
import pytest
import torch

import oracle
import tensorjoin_variants_b200 as tj

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 3, 8])
@pytest.mark.parametrize("nr,ns", [(1, 40000), (16, 32768), (63, 32767), (129, 70001), (1185, 33000)])
def test_few_rows_with_many(nr, ns, d):
    rng = np.random.default_rng(nr + d)
    R, S = rng.random((nr, d), dtype=np.float32) - 0.5, rng.random((ns, d), dtype=np.float32) - 0.5
    S[7] = R[0]
    for T in (0.0, 0.001 * d, 0.3 * d, 2.0 * d):   # (all about the origin, where rows past R's last one would lie)
        res = tj.join_result(torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda(), eps2=T)
        assert res.stats["ms_index"] == 0.0   # direct
        want = oracle.join_f32(R, S, T, "rs")
        assert np.array_equal(res.keys().cpu().numpy().view(np.uint64), want)
        i, j = (t.cpu().numpy().astype(np.uint64) for t in res.pairs())   # rows of up to ns columns
        assert np.array_equal(i * np.uint64(ns) + j, want)
        counts, flat = (t.cpu().numpy() for t in res.neighbor_table())
        assert np.array_equal(counts, np.bincount(i.astype(np.int64), minlength=nr))
        assert np.array_equal(flat, j.astype(np.int64))
