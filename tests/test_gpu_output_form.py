"""Which results are kept by rows and which as whole keys (most pairs in long rows): the rule at its borders,
and the same pairs in every form of output on both sides of it."""
import numpy as np
import pytest
import torch

import oracle
import tensorjoin_variants_b200 as tj
from tensorjoin_variants_b200 import _lib

pytestmark = pytest.mark.gpu


def _by_rows(res):
    """Keys of a result by rows are written by a kernel, whole keys are copied."""
    before = _lib.lib().tj_kernel_launches()
    keys = res.keys()
    return keys, _lib.lib().tj_kernel_launches() > before


def _check(res, want, n_rows, n_cols, by_rows):
    keys, form = _by_rows(res)
    assert form == by_rows
    assert np.array_equal(keys.cpu().numpy().view(np.uint64), want)
    i, j = (t.cpu().numpy() for t in res.pairs())
    assert np.array_equal(i.astype(np.uint64) * np.uint64(n_cols) + j.astype(np.uint64), want)
    counts, flat = (t.cpu().numpy() for t in res.neighbor_table())
    assert np.array_equal(counts, np.bincount(i, minlength=n_rows))
    assert np.array_equal(flat, j)


def _clusters(sizes, rng):
    """Points of one place per size, 10 apart, in shuffled order."""
    X = np.zeros((sum(sizes), 2), np.float32)
    X[:, 0] = 10.0 * np.repeat(np.arange(len(sizes)), sizes)
    return X[rng.permutation(len(X))]


# rows x columns of each place; more than 2^20 pairs unless said otherwise
CASES = [
    ([(300, 2000), (1300, 500)], False),           # 781 a row on average
    ([(300, 2000), (1500, 450)], True),            # 708, and 47 % of the pairs in long rows
    ([(350, 2000), (1500, 450)], False),           # 51 %
    ([(300, 513), (2000, 512)], True),             # rows of 513 are long, of 512 are not
    ([(2100, 513)], False),
    ([(1, 4096), (3000, 400)], True),              # the longest row a block sorts
    ([(1, 4097), (3000, 400)], False),
    ([(200, 4096)], True),                         # 819,200 pairs: no share asked for
    ([(1370, 766), (9000, 0)], False),
    ([(1049, 1000)], False),                       # too long on average to be counted
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_form(case):
    places, by_rows = CASES[case]
    rng = np.random.default_rng(case)
    R, S = (_clusters([p[k] for p in places], rng) for k in (0, 1))
    res = tj.join_result(torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda(), eps2=1.0, screen="bf16", guards=True)
    _check(res, oracle.join_f32(R, S, 1.0, "rs"), len(R), len(S), by_rows)


@pytest.mark.parametrize("sizes,by_rows", [([700] + [300] * 40, True), ([1500] + [100] * 30, False), ([1500, 400], False)])
def test_form_directed(sizes, by_rows):
    X = _clusters(sizes, np.random.default_rng(len(sizes)))
    res = tj.join_result(torch.from_numpy(X).cuda(), None, eps2=1.0, mode="directed", screen="plain", chunk_items=64)
    _check(res, oracle.join_f32(X, None, 1.0, "directed"), len(X), len(X), by_rows)
    small = tj.join_result(torch.from_numpy(X).cuda(), None, eps2=1.0, mode="directed", screen="plain", capacity=4096)
    assert small.stats["retries"] >= 1
    _check(small, oracle.join_f32(X, None, 1.0, "directed"), len(X), len(X), by_rows)
