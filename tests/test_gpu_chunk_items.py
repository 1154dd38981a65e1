"""Chunk sizes up to the option's largest value ("do not cut the lists"): the oracle's pairs in every mode."""
import numpy as np
import pytest
import torch

import oracle
import tensorjoin_variants_b200 as tj

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunk", [1, 7, 2**16, 2**31 - 5, 2**31 - 1])
@pytest.mark.parametrize("screen", ["plain", "bf16x3", "int8limb"])
def test_chunk_items(screen, chunk):
    rng = np.random.default_rng(chunk % 1000)
    if screen == "int8limb":
        X = rng.integers(-900, 900, (1500, 20)).astype(np.int16)
        T, join = float(20 * 3 * 10**5), oracle.join_i16
    else:
        X = rng.random((1500, 20), dtype=np.float32)
        T, join = 1.5, oracle.join_f32
    Xd = torch.from_numpy(X).cuda()
    for mode in ("upper", "directed", "rs"):
        res = tj.join_result(Xd, Xd[:900] if mode == "rs" else None, eps2=T, mode=mode, screen=screen, chunk_items=chunk)
        want = join(X, X[:900] if mode == "rs" else None, T, mode)
        assert len(want) > 0 and np.array_equal(res.keys().cpu().numpy().view(np.uint64), want), mode
    if screen != "int8limb":
        e = float(np.sqrt(T))
        for (i, j), n in zip(tj.join_batched([(Xd, Xd[:900], e), (Xd[:900], Xd[:300], e)], screen=screen,
                                             chunk_items=chunk), (900, 300)):
            R = X if n == 900 else X[:900]
            got = i.cpu().numpy().astype(np.uint64) * np.uint64(n) + j.cpu().numpy().astype(np.uint64)
            assert np.array_equal(got, join(R, X[:n], e * e, "rs"))
