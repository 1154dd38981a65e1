"""Small joins done directly (no index): equal to the indexed path and to the oracle over every form they
take -- R-S, upper and directed, rows that are and are not multiples of 16 bytes, inputs that start at any
4-byte address, sides of one row, ties and duplicates -- and refused exactly where the screen that was
asked for refuses.  Options make a join take the indexed path."""
import numpy as np
import pytest
import torch

import oracle
import tensorjoin_variants_b200 as tj
from tensorjoin_variants_b200 import _lib

pytestmark = pytest.mark.gpu


def _dev(A, shift=0):
    """A on the device, starting `shift` floats into an allocation."""
    buf = torch.empty(A.size + shift, device="cuda")
    t = buf[shift:].view(A.shape)
    t.copy_(torch.from_numpy(A))
    return t


def _both(R, S, T, mode, screen="bf16", shift=0):
    Rt, St = _dev(R, shift), None if S is None else _dev(S, shift)
    direct = tj.join_result(Rt, St, eps2=T, mode=mode, screen=screen)
    indexed = tj.join_result(Rt, St, eps2=T, mode=mode, screen=screen, chunk_items=64)
    want = oracle.join_f32(R, S, T, mode)
    for res in (direct, indexed):
        assert np.array_equal(res.keys().cpu().numpy().view(np.uint64), want)
        i, j = (t.cpu().numpy().astype(np.uint64) for t in res.pairs())
        assert np.array_equal(i * np.uint64((R if S is None else S).shape[0]) + j, want)
        counts, flat = (t.cpu().numpy() for t in res.neighbor_table())
        assert np.array_equal(counts, np.bincount(i.astype(np.int64), minlength=len(R)))
        assert np.array_equal(flat, j.astype(np.int64))
    st = direct.stats
    assert st["result_pairs"] == len(want) and st["pairs_screened"] == st["pairs_all"]
    own = len(R) if mode == "directed" else 0
    sym = 2 if mode == "directed" else 1
    assert st["screen_accept"] + st["refine_accept"] == (len(want) - own) // sym
    return direct


@pytest.mark.parametrize("d", [1, 2, 3, 4, 15, 16, 17, 20, 64, 65, 128, 191, 192])
@pytest.mark.parametrize("nr,ns", [(1, 1), (1, 300), (129, 64), (128, 65), (300, 1), (513, 700)])
def test_rs(nr, ns, d):
    rng = np.random.default_rng(100 * d + nr)
    R, S = rng.random((nr, d), dtype=np.float32), rng.random((ns, d), dtype=np.float32)
    T = float(np.quantile(((R[:60, None].astype(np.float64) - S[None, :200]) ** 2).sum(-1), 0.1))
    _both(R, S, T, "rs", shift=nr % 4)


@pytest.mark.parametrize("mode", ["upper", "directed"])
@pytest.mark.parametrize("n,d", [(1, 4), (2, 3), (64, 8), (65, 5), (127, 16), (1000, 2), (2111, 33)])
def test_self(n, d, mode):
    rng = np.random.default_rng(n + d)
    X = rng.random((n, d), dtype=np.float32)
    X[n // 2:n // 2 + n // 8] = X[: n // 8]
    for T in (0.0, float(d) / 12, 4.0 * d):
        _both(X, None, T, mode, shift=n % 3)


def test_ties_are_decided_in_fp64():
    """Thresholds equal to sampled FP64 distances, which an FP32 sum cannot decide."""
    rng = np.random.default_rng(7)
    R, S = rng.random((200, 24), dtype=np.float32), rng.random((300, 24), dtype=np.float32)
    d2 = np.zeros((200, 300))
    for k in range(24):
        t = R[:, None, k].astype(np.float64) - S[None, :, k]
        d2 += t * t
    for T in np.quantile(d2, [0.001, 0.03, 0.4], method="lower"):
        for q in (T, np.nextafter(T, 0)):
            assert _both(R, S, float(q), "rs", "plain").stats["band"] >= 1


@pytest.mark.parametrize("screen", ["plain", "bf16", "fp16", "bf16x3", "fp16x3"])
def test_refusals_and_large_values(screen):
    rng = np.random.default_rng(9)
    X = rng.random((150, 12)).astype(np.float32)
    for bad in (np.nan, np.inf, -np.inf, 3e38):
        Y = X.copy()
        Y[77, 5] = bad
        with pytest.raises(_lib.TJError) as e:
            tj.self_join(_dev(Y), 0.3, screen=screen)
        assert e.value.code in ((-3, -4) if np.isfinite(bad) and "fp16" in screen else (-3,))
    big = X.copy()
    big[:75] += np.float32(50000.0)     # centred: +-25000, inside the FP16 range
    i, j = tj.self_join(_dev(big), 0.5, screen=screen)
    want = oracle.join_f32(big, None, 0.25, "upper")
    assert np.array_equal(i.cpu().numpy().astype(np.uint64) * np.uint64(150) + j.cpu().numpy().astype(np.uint64), want)
    big[:75] += np.float32(200000.0)    # beyond it
    if "fp16" in screen:
        with pytest.raises(_lib.TJError) as e:
            tj.self_join(_dev(big), 0.5, screen=screen)
        assert e.value.code == -4
    else:
        tj.self_join(_dev(big), 0.5, screen=screen)


def test_concurrent_streams():
    import threading
    rng = np.random.default_rng(11)
    sets = [rng.random((400 + 100 * k, 6), dtype=np.float32) for k in range(4)]
    want = [oracle.join_f32(X, None, 0.1, "directed") for X in sets]
    got = [None] * 4

    def run(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            X = torch.from_numpy(sets[k]).cuda()
            for _ in range(20):
                got[k] = tj.join_result(X, None, eps2=0.1, mode="directed").keys().cpu().numpy().view(np.uint64)

    th = [threading.Thread(target=run, args=(k,)) for k in range(4)]
    [t.start() for t in th]
    [t.join() for t in th]
    for k in range(4):
        assert np.array_equal(got[k], want[k])
