"""Direct upper joins at the borders of their units (128 rows x 64 columns, those with a pair above the
diagonal)."""
import numpy as np
import pytest
import torch

import oracle
import tensorjoin_variants_b200 as tj

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 64, 65, 127, 128, 129, 191, 192, 193, 256, 257, 1000, 1409, 2944, 2945])
def test_upper_units(n):
    rng = np.random.default_rng(n)
    X = rng.random((n, 6), dtype=np.float32)
    for T in (0.3, 12.0):   # some pairs; all of them
        res = tj.join_result(torch.from_numpy(X).cuda(), None, eps2=T, mode="upper")
        assert res.stats["ms_index"] == 0.0   # direct
        assert np.array_equal(res.keys().cpu().numpy().view(np.uint64), oracle.join_f32(X, None, T, "upper"))
