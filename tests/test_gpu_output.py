"""Canonical output by rows: every way a row is put in order (ranked in a shared stage, sorted in a
warp's registers, sorted by a block) at the row lengths where one takes over from the next, empty rows
between full ones, the fallback to whole keys, and every form the result is read in."""
import numpy as np
import pytest
import torch

import oracle
import tensorjoin_variants_b200 as tj

pytestmark = pytest.mark.gpu


def _check(res, want, n_rows, n_cols):
    k = res.keys().cpu().numpy().view(np.uint64)
    assert np.array_equal(k, want)
    i, j = (t.cpu().numpy() for t in res.pairs())
    assert np.array_equal(i.astype(np.uint64) * np.uint64(n_cols) + j.astype(np.uint64), want)
    counts, flat = (t.cpu().numpy() for t in res.neighbor_table())
    assert np.array_equal(counts, np.bincount(i, minlength=n_rows))
    assert np.array_equal(flat, j)


@pytest.mark.parametrize("length", [1, 2, 31, 32, 33, 63, 64, 65, 128, 129, 256, 257, 511, 512, 513, 1024, 1025, 2500])
def test_row_lengths(length):
    """Rows with exactly `length` columns, rows with one and rows with none, in shuffled order."""
    rng = np.random.default_rng(length)
    S = np.zeros((length + 1, 4), np.float32)
    S[-1] = 50.0
    S = S[rng.permutation(length + 1)]
    R = np.full((200, 4), 100.0, np.float32)   # no column
    R[::3] = 0.0                               # `length` columns
    R[1::7] = 50.0                             # one column
    res = tj.join_result(torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda(), eps2=1.0, screen="plain", guards=True)
    _check(res, oracle.join_f32(R, S, 1.0, "rs"), 200, length + 1)


@pytest.mark.parametrize("ns", [16384, 16385])
def test_longest_row_and_fallback(ns):
    """A row as long as a block sorts, and one more (whole keys are sorted instead)."""
    rng = np.random.default_rng(ns)
    R, S = rng.random((3, 2), dtype=np.float32), rng.random((ns, 2), dtype=np.float32)
    res = tj.join_result(torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda(), eps2=9.0, screen="plain", guards=True)
    _check(res, np.arange(3 * ns, dtype=np.uint64), 3, ns)


def test_many_more_rows_than_pairs():
    rng = np.random.default_rng(3)
    R, S = rng.random((1_100_000, 2), dtype=np.float32), rng.random((3, 2), dtype=np.float32)
    res = tj.join_result(torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda(), eps2=1e-4, screen="plain", guards=True)
    _check(res, oracle.join_f32(R, S, 1e-4, "rs"), 1_100_000, 3)


@pytest.mark.parametrize("n,eps2", [(1, 0.1), (2, 4.0), (33, 4.0), (700, 0.02), (700, 4.0), (5000, 0.003)])
def test_directed_rows(n, eps2):
    rng = np.random.default_rng(n)
    X = rng.random((n, 2), dtype=np.float32)
    res = tj.join_result(torch.from_numpy(X).cuda(), None, eps2=eps2, mode="directed", screen="plain", guards=True)
    _check(res, oracle.join_f32(X, None, eps2, "directed"), n, n)


def test_capacity_retry_counts_once():
    rng = np.random.default_rng(8)
    X = rng.random((3000, 3), dtype=np.float32)
    for mode in ("upper", "directed"):
        res = tj.join_result(torch.from_numpy(X).cuda(), None, eps2=0.02, mode=mode, screen="plain", capacity=512)
        assert res.stats["retries"] >= 1
        _check(res, oracle.join_f32(X, None, 0.02, mode), 3000, 3000)


def test_batch_rows_with_empty_joins():
    """Joins with no rows, no columns, no pairs and one pair, whose row and key ranges touch."""
    rng = np.random.default_rng(9)
    joins = []
    for k, (nr, ns, eps) in enumerate([(0, 5, 1.0), (40, 0, 1.0), (300, 200, 0.3), (10, 10, 0.0), (0, 0, 1.0),
                                       (1, 1, 9.0), (129, 700, 9.0), (50, 60, 0.2), (7, 0, 1.0)]):
        d = (2, 5)[k % 2]
        joins.append((rng.random((nr, d), dtype=np.float32), rng.random((ns, d), dtype=np.float32), eps))
    dev = [(torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda(), e) for R, S, e in joins]
    res = tj.api.join_batched_result(dev, screen="plain", guards=True)
    keys, base, kk = [], 0, res.keys().cpu().numpy().view(np.uint64)
    for (R, S, e), (i, j) in zip(joins, res.split()):
        want = oracle.join_f32(R, S, e * e, "rs") if len(R) and len(S) else np.zeros(0, np.uint64)
        got = i.cpu().numpy().astype(np.uint64) * np.uint64(len(S)) + j.cpu().numpy().astype(np.uint64)
        assert np.array_equal(got, want)
        keys.append(want + np.uint64(base))
        base += len(R) * len(S)
    assert np.array_equal(kk, np.concatenate(keys))
