"""int14 rows of small values, which the high limbs leave undecided: the join goes over to four products and
keeps no band; rows of the full range do not."""
import numpy as np
import pytest
import torch

import oracle
import tensorjoin_variants_b200 as tj

pytestmark = pytest.mark.gpu


def _rows(n, d, V, seed):
    return np.random.default_rng(seed).integers(-V, V + 1, (n, d)).astype(np.int16)


def _threshold(R, S, q):
    a, b = R[::37].astype(np.int64), S[::41].astype(np.int64)
    return int(np.quantile(((a[:, None] - b[None]) ** 2).sum(-1), q))


@pytest.mark.parametrize("V,d", [(3, 5), (20, 33), (100, 128), (300, 64), (60, 129), (200, 256)])
@pytest.mark.parametrize("mode,n,ns", [("upper", 6001, 0), ("directed", 6001, 0), ("rs", 6001, 4099)])
def test_small_values(mode, n, ns, V, d):
    R = _rows(n, d, V, V + d)
    S = _rows(ns, d, V, V) if ns else None
    T = _threshold(R, R if S is None else S, 1e-3)
    want = (oracle.join_i16)(R, S, T, mode)
    Rd, Sd = torch.from_numpy(R).cuda(), None if S is None else torch.from_numpy(S).cuda()
    for options in ({}, {"capacity": 3000}, {"chunk_items": 5, "guards": True}, {"stage_keys": True}):
        res = tj.join_result(Rd, Sd, eps2=T, mode=mode, screen="int8limb", **options)
        st = res.stats
        assert st["band"] == 0 and st["retries"] >= 1, (options, st)   # four products
        assert np.array_equal(res.keys().cpu().numpy().view(np.uint64), want), options
        assert st["pairs_screened"] <= (n * ns if ns else n * (n + 256))
        four = tj.join_result(Rd, Sd, eps2=T, mode=mode, screen="int8limb", i8_four_products=True, **options).stats
        for f in ("pairs_screened", "screen_ops", "tile_pairs"):
            assert st[f] == four[f], f
        if "stage_keys" in options:
            assert len(res.stage_keys(1)) == 0 and len(res.stage_keys(0)) == st["screen_accept"]


@pytest.mark.parametrize("d", [40, 200])
def test_full_range_keeps_the_high_limbs(d):
    R = _rows(6001, d, 8191, d)
    T = _threshold(R, R, 1e-3)
    res = tj.join_result(torch.from_numpy(R).cuda(), None, eps2=T, mode="upper", screen="int8limb", capacity=3000)
    assert res.stats["band"] > 0 and res.stats["retries"] >= 1   # (a retry for room alone)
    assert np.array_equal(res.keys().cpu().numpy().view(np.uint64), oracle.join_i16(R, None, T, "upper"))
