"""Small joins through the index and the tensor-core screen (an option keeps them off the direct pass), beside
the direct pass where both share a thread, a workspace or a result buffer."""
import threading

import numpy as np
import pytest
import torch

import oracle
import tensorjoin_variants_b200 as tj
from tensorjoin_variants_b200 import workloads as W

pytestmark = pytest.mark.gpu

INDEXED = {"chunk_items": 64}


def _dev(*xs):
    return tuple(torch.from_numpy(x).cuda() for x in xs)


def _keys(res):
    return res.keys().cpu().numpy().view(np.uint64)


def _indexed(res):
    return res.stats["ms_index"] > 0.0


@pytest.mark.parametrize("per_call", [(INDEXED,), (INDEXED, {})])   # the index alone; in turn with the direct pass
def test_host_threads(per_call):
    ws = [W.mixture64(n=6000, d=32, seed=s, samples=1 << 14) for s in (11, 12)]
    want = [oracle.join_f32(w.R, w.S, w.T, "rs") for w in ws]
    errs = []

    def run(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                R, S = _dev(ws[k].R, ws[k].S)
                for opts in per_call * 4:
                    res = tj.join_result(R, S, eps2=ws[k].T, screen="bf16x3", **opts)
                    assert _indexed(res) == bool(opts)
                    assert np.array_equal(_keys(res), want[k]), (k, opts)
        except Exception as e:   # surfaced below
            errs.append(e)

    th = [threading.Thread(target=run, args=(k,)) for k in (0, 1)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not errs, errs


def test_results_alive_across_joins():
    """Held results keep their pairs while joins of other sizes and of the other form reuse freed buffers."""
    ws = [W.mixture64(n=n, d=d, samples=1 << 14) for n, d in ((3000, 16), (12000, 64), (1500, 32))]
    want = [oracle.join_f32(w.R, w.S, w.T, "rs") for w in ws]
    held = []
    for opts in (INDEXED, {}, INDEXED):
        for k, w in enumerate(ws):
            held.append((k, tj.join_result(*_dev(w.R, w.S), eps2=w.T, screen="bf16x3", **opts)))
            if len(held) % 2 == 0:
                held[-2] = None   # release one while the others stay alive
    for k, res in (h for h in held if h is not None):
        assert np.array_equal(_keys(res), want[k]), k


@pytest.mark.parametrize("opts", [INDEXED, {}])
def test_neighbor_table_and_host_rows(opts):
    w = W.uniform16(n=3000)
    res = tj.join_result(_dev(w.R)[0], None, eps2=w.T, mode="directed", **opts)
    assert _indexed(res) == bool(opts)
    want = oracle.join_f32(w.R, None, w.T, "directed")
    counts, flat = res.neighbor_table()
    assert np.array_equal(counts.cpu().numpy(), np.bincount((want // 3000).astype(np.int64), minlength=3000))
    assert np.array_equal(flat.cpu().numpy(), (want % 3000).astype(np.int64))
    i, j = tj.self_join(w.R, eps2=w.T, **opts)   # host rows in, host ids out
    assert not i.is_cuda and not j.is_cuda
    assert np.array_equal(i.numpy().astype(np.uint64) * np.uint64(3000) + j.numpy().astype(np.uint64),
                          oracle.join_f32(w.R, None, w.T, "upper"))


@pytest.mark.parametrize("opts", [INDEXED, {}])
def test_batch_equals_single_joins(opts):
    g = np.random.default_rng(42)
    joins = []
    for k in range(8):
        R, S = (g.random((int(g.integers(200, 3000)), 32), dtype=np.float32) for _ in range(2))
        joins.append((*_dev(R, S), 1.2 + 0.05 * k))
    for (R, S, eps), (i, j) in zip(joins, tj.join_batched(joins, screen="bf16x3")):
        res = tj.join_result(R, S, eps, screen="bf16x3", **opts)
        assert _indexed(res) == bool(opts)
        i1, j1 = res.pairs()
        assert torch.equal(i, i1) and torch.equal(j, j1)
