"""Row order and chunk order of the index at the lengths where one way of sorting takes over from another
(a block per segment up to 8,192 rows, radix passes beyond; their status words cleared at once up to 2^21)
and where chunks fill blocks of lists."""
import numpy as np
import pytest
import torch

import oracle
import tensorjoin_variants_b200 as tj

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 63, 64, 65, 127, 1000, 4096, 4097, 8191, 8192, 8193, 12289, 70000, 2_200_000])
def test_row_order_is_sorted_and_stable(n):
    rng = np.random.default_rng(n)
    X = rng.integers(0, 9, (n, 3)).astype(np.float32)   # many rows per cell
    idx = tj.build_index(torch.from_numpy(X).cuda(), 0.5 if n < 100000 else 0.0)
    perm, keys = idx.perm.cpu().numpy().view(np.uint32).astype(np.int64), idx.keys.cpu().numpy().view(np.uint64)
    assert np.array_equal(np.sort(perm), np.arange(n))
    assert np.all(keys[1:] >= keys[:-1])
    assert np.all(perm[1:][keys[1:] == keys[:-1]] > perm[:-1][keys[1:] == keys[:-1]])
    cell = np.concatenate([[True], keys[1:] != keys[:-1]])
    assert np.array_equal(idx.cell_start.cpu().numpy(), np.concatenate([np.flatnonzero(cell), [n]]))
    # one cell holds equal rows
    rows = X[perm]
    assert np.all((rows[1:] == rows[:-1]).all(1) == ~cell[1:])


@pytest.mark.parametrize("chunk", [1, 2, 7, 64, 1000])
def test_chunks_cover_every_candidate_once(chunk):
    """Clustered rows (lists of very different lengths): no pair is lost or doubled however lists are cut."""
    rng = np.random.default_rng(chunk)
    c = rng.random((30, 5))
    w = rng.dirichlet(np.full(30, 0.4))
    R = (c[rng.choice(30, 20000, p=w)] + rng.standard_normal((20000, 5)) * 0.02).astype(np.float32)
    S = (c[rng.choice(30, 9000, p=w)] + rng.standard_normal((9000, 5)) * 0.02).astype(np.float32)
    T = 0.0004
    want = oracle.join_f32(R, S, T, "rs")
    for screen in ("plain", "bf16x3"):
        res = tj.join_result(torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda(), eps2=T, screen=screen,
                             chunk_items=chunk, guards=True)
        assert np.array_equal(res.keys().cpu().numpy().view(np.uint64), want)


@pytest.mark.parametrize("largest", [8192, 8193])
def test_packed_joins_by_their_largest(largest):
    """Packed joins whose largest side is the longest a block sorts, and one row more."""
    rng = np.random.default_rng(largest)
    joins = [(rng.random((n, 4), dtype=np.float32), rng.random((m, 4), dtype=np.float32), 0.08)
             for n, m in ((largest, 40), (1, 300), (500, largest), (0, 10), (77, 1))]
    out = tj.join_batched([(torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda(), e) for R, S, e in joins],
                          screen="bf16x3", guards=True)
    for (R, S, e), (i, j) in zip(joins, out):
        want = oracle.join_f32(R, S, e * e, "rs") if len(R) else np.zeros(0, np.uint64)
        assert np.array_equal(i.cpu().numpy().astype(np.uint64) * np.uint64(len(S)) + j.cpu().numpy().astype(np.uint64),
                              want)
