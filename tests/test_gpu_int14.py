"""int8 high-limb screen at the edges of its groups of R tiles, pairs of S tiles and folded norms: sides
of one row to a few tiles, rows of 1 to 256 elements, lists whose entries are for some R tiles of a
group only (clustered rows, with odd list lengths), norms beyond what the fold holds, and thresholds
that make most pairs candidates.  Pair sets equal the exact integer oracle's."""
import numpy as np
import pytest
import torch

import oracle
import tensorjoin_variants_b200 as tj

pytestmark = pytest.mark.gpu


def _check(R, S, T, mode="rs", **kw):
    Rt = torch.from_numpy(R).cuda()
    St = None if S is None else torch.from_numpy(S).cuda()
    res = tj.join_result(Rt, St, eps2=int(T), mode=mode, screen="int8limb", guards=True, **kw)
    assert np.array_equal(res.keys().cpu().numpy().view(np.uint64), oracle.join_i16(R, S, int(T), mode))
    return res.stats


def _quantile(R, S, q):
    return int(np.quantile(((R[:80, None, :].astype(np.int64) - S[None, :400]) ** 2).sum(-1), q))


@pytest.mark.parametrize("d", [1, 31, 64, 127, 128, 129, 192, 255, 256])
@pytest.mark.parametrize("nr,ns", [(1, 1), (127, 129), (130, 511), (520, 260)])
def test_edges(nr, ns, d):
    rng = np.random.default_rng(1000 * d + nr)
    R = rng.integers(-8192, 8192, (nr, d), dtype=np.int16)
    S = rng.integers(-8192, 8192, (ns, d), dtype=np.int16)
    S[: min(nr, ns) // 3] = np.clip(R[: min(nr, ns) // 3].astype(int) + 1, -8192, 8191)
    _check(R, S, _quantile(R, S, 0.02))


@pytest.mark.parametrize("chunk", [0, 3, 64])
@pytest.mark.parametrize("d", [24, 128, 200])
def test_partial_groups(d, chunk):
    """Clustered rows: most tiles meet few others, so list entries name one to all R tiles of their group and
    lists are of any length; `chunk` cuts them at odd places."""
    rng = np.random.default_rng(d + chunk)
    centres = rng.integers(-7000, 7000, (40, d))
    X = (centres[rng.integers(0, 40, 9000)] + rng.integers(-300, 301, (9000, d))).astype(np.int16)
    Y = (centres[rng.integers(0, 40, 5000)] + rng.integers(-300, 301, (5000, d))).astype(np.int16)
    T = int(2 * d * 300 ** 2 / 3 * 0.9)
    st = _check(X, Y, T, chunk_items=chunk)
    assert 0 < st["tile_pairs"] < 71 * 40
    for mode in ("upper", "directed"):
        _check(X, None, T, mode, chunk_items=chunk)


@pytest.mark.parametrize("d", [128, 256])
def test_large_norms_and_dense_candidates(d):
    """Rows at the corners of the range (at 256 elements their norm term is beyond the fold's largest) among
    ordinary ones, at thresholds from none to all of the pairs."""
    rng = np.random.default_rng(d)
    R = rng.integers(-8192, 8192, (700, d), dtype=np.int16)
    S = rng.integers(-8192, 8192, (900, d), dtype=np.int16)
    R[::9] = rng.choice(np.array([-8192, 8191], np.int16), (78, d))
    S[::7] = R[rng.integers(0, 78, 129) * 9]
    for q in (0.0, 0.1, 0.5, 0.9, 1.0):
        _check(R, S, _quantile(R, S, q))
    _check(R, S, d * 16383 ** 2)
