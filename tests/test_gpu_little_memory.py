"""Joins on a device with little memory left: the accept buffer's usual size (256 MB from 2^25 pairs on) does
not fit, the join does."""
import numpy as np
import pytest
import torch

import oracle
import tensorjoin_variants_b200 as tj
from tensorjoin_variants_b200 import _lib

pytestmark = pytest.mark.gpu
LEFT = 200 << 20


def _fill():
    """Takes the device's free memory down to about LEFT bytes (allocated, never written)."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    assert _lib.lib().tj_pool_trim(0) == 0
    held = []
    for step in (1 << 30, 64 << 20, 8 << 20):
        while torch.cuda.mem_get_info()[0] > LEFT + step:
            n = (torch.cuda.mem_get_info()[0] - LEFT) // step * step
            held.append(torch.empty(n, dtype=torch.uint8, device="cuda"))
    return held


@pytest.mark.parametrize("mode", ["rs", "upper", "directed"])
def test_join_beside_a_nearly_full_device(mode):
    rng = np.random.default_rng(3)
    R, S = (rng.random((n, 8), dtype=np.float32) for n in (9000, 6000))
    S = S if mode == "rs" else None
    T = 0.05
    want = oracle.join_f32(R, S, T, mode)
    Rd, Sd = torch.from_numpy(R).cuda(), None if S is None else torch.from_numpy(S).cuda()

    def keys(capacity=0):
        return tj.join_result(Rd, Sd, eps2=T, mode=mode, screen="bf16x3", capacity=capacity,
                              chunk_items=64).keys().cpu().numpy().view(np.uint64)

    assert np.array_equal(keys(capacity=1 << 20), want)   # the kernels are loaded
    held = _fill()
    try:
        got = keys()
    finally:
        del held
        torch.cuda.empty_cache()
    assert np.array_equal(got, want)
    assert np.array_equal(keys(), want)
