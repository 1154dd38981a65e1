"""Plain FP32 screen at the edges of its tiling: column quarters of 64, k chunks of 16 with one to
three elements left over, rows that are not multiples of 16 bytes, the diagonal of a self-join and
CTAs whose share of the candidates starts inside a tile pair.  Pair sets equal the oracle's exactly."""
import numpy as np
import pytest
import torch

import oracle
import tensorjoin_variants_b200 as tj

pytestmark = pytest.mark.gpu


def _keys(res):
    return res.keys().cpu().numpy().view(np.uint64)


@pytest.mark.parametrize("d", [1, 2, 3, 4, 5, 6, 7, 15, 16, 18, 19, 20, 36])
@pytest.mark.parametrize("nr,ns", [(1, 63), (127, 64), (129, 65), (128, 257), (300, 191)])
def test_plain_edges(nr, ns, d):
    rng = np.random.default_rng(1000 * d + ns)
    R, S = rng.random((nr, d), dtype=np.float32), rng.random((ns, d), dtype=np.float32)
    T = float(np.quantile(((R[:, None, :].astype(np.float64) - S[None]) ** 2).sum(-1), 0.3))
    res = tj.join_result(torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda(), eps2=T, screen="plain", guards=True)
    assert np.array_equal(_keys(res), oracle.join_f32(R, S, T, "rs"))


@pytest.mark.parametrize("n,d", [(65, 3), (256, 2), (1023, 16), (3001, 9)])
def test_plain_self_join_diagonal(n, d):
    rng = np.random.default_rng(n + d)
    X = rng.random((n, d), dtype=np.float32)
    T = float(np.quantile(((X[:60, None, :].astype(np.float64) - X[None]) ** 2).sum(-1), 0.2))
    for mode in ("upper", "directed"):
        res = tj.join_result(torch.from_numpy(X).cuda(), None, eps2=T, mode=mode, screen="plain", guards=True)
        assert np.array_equal(_keys(res), oracle.join_f32(X, None, T, mode))


def test_plain_batched_ragged_tiles():
    """Tiles of packed joins start and end anywhere in the packed rows, the last one at its end."""
    rng = np.random.default_rng(5)
    joins = []
    for k, (nr, ns) in enumerate([(130, 61), (1, 300), (513, 1), (77, 450), (128, 256), (255, 129)]):
        d = (2, 16, 7)[k % 3]
        R, S = rng.random((nr, d), dtype=np.float32), rng.random((ns, d), dtype=np.float32)
        joins.append((R, S, 0.3 * np.sqrt(d)))
    out = tj.join_batched([(torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda(), e) for R, S, e in joins],
                          screen="plain", guards=True)
    for (R, S, e), (i, j) in zip(joins, out):
        got = i.cpu().numpy().astype(np.uint64) * np.uint64(S.shape[0]) + j.cpu().numpy().astype(np.uint64)
        assert np.array_equal(got, oracle.join_f32(R, S, e * e, "rs"))
