"""Plain screen over a batch of several row lengths: candidates taken in short runs, in turn."""
import numpy as np
import pytest
import torch

import oracle
import tensorjoin_variants_b200 as tj

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[(1, 1, 3), (700, 900, 16)], [(300, 5000, 2), (4000, 2500, 8), (2500, 3100, 33), (1, 700, 64)],
                                   [(20000, 9000, 4), (9000, 12000, 9), (257, 256, 130)]])
def test_plain_batch_of_several_lengths(sizes):
    rng = np.random.default_rng(len(sizes))
    joins, want = [], []
    for nr, ns, d in sizes:
        R, S = rng.random((nr, d), dtype=np.float32), rng.random((ns, d), dtype=np.float32)
        eps = float(np.sqrt(np.quantile(((R[:60, None, :].astype(np.float64) - S[None, :300]) ** 2).sum(-1), 0.002)))
        joins.append((torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda(), eps))
        want.append(oracle.join_f32(R, S, eps * eps, "rs"))
    for (i, j), w, (_, ns, _) in zip(tj.join_batched_result(joins, screen="plain").split(), want, sizes):
        got = i.cpu().numpy().astype(np.uint64) * np.uint64(ns) + j.cpu().numpy().astype(np.uint64)
        assert np.array_equal(got, w)
