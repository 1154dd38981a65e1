"""R-S joins of sides that share memory (R the first rows of S, or the same rows): every row of both sides is
looked at, and the join is an R-S join in its pairs and in its counters."""
import numpy as np
import pytest
import torch

import oracle
import tensorjoin_variants_b200 as tj
from tensorjoin_variants_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("screen", ["plain", "bf16", "fp16", "bf16x3", "fp16x3"])
@pytest.mark.parametrize("k", [1, 100, 256])
def test_refusals_in_rows_past_the_shared_ones(screen, k):
    rng = np.random.default_rng(k)
    X = torch.from_numpy(rng.random((700, 12), dtype=np.float32)).cuda()
    half = "fp16" in screen
    bad = [(np.nan, (-3,)), (np.inf, (-3,)), (-np.inf, (-3,)), (3e38, (-3, -4) if half else (-3,))]
    if half:
        bad.append((3e5, (-4,)))
    for value, codes in bad:
        for row in (k, 699):
            Y = X.clone()
            Y[row, 5] = value
            for options in ({}, {"chunk_items": 64}):   # direct, indexed
                with pytest.raises(_lib.TJError) as e:
                    tj.join(Y[:k], Y, 0.3, screen=screen, **options)
                assert e.value.code in codes


@pytest.mark.parametrize("k,n", [(1, 300), (256, 700), (700, 256), (500, 500)])
def test_pairs_and_counters(k, n):
    rng = np.random.default_rng(k + n)
    X = rng.random((max(k, n), 7), dtype=np.float32)
    Xd = torch.from_numpy(X).cuda()
    for T in (0.0, 0.2):   # 0: every row's own pair is left to FP64
        res = tj.join_result(Xd[:k], Xd[:n], eps2=T)
        want = oracle.join_f32(X[:k], X[:n], T, "rs")
        assert np.array_equal(res.keys().cpu().numpy().view(np.uint64), want)
        st = res.stats
        assert st["screen_accept"] + st["refine_accept"] == len(want)
        apart = tj.join_result(Xd[:k], Xd[:n].clone(), eps2=T).stats
        for f in ("screen_accept", "refine_accept", "band", "band_fp64", "rare_checks"):
            assert st[f] == apart[f], f
