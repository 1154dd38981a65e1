"""Exact integer refinement of int14 rows at every width of its loads: rows on 16-, 8-, 4- and 2-byte
boundaries (by the row length and by where the first row lies), with remainders."""
import numpy as np
import pytest
import torch

import tensorjoin_variants_b200 as tj

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1, 2, 4])
@pytest.mark.parametrize("d", [1, 6, 17, 20, 24, 34, 100, 130])
def test_int_refinement(d, offset):
    g = torch.Generator(device="cuda").manual_seed(d * 8 + offset)
    nr, ns = 700, 900
    flat = torch.randint(-8192, 8192, ((nr + ns) * d + offset,), generator=g, device="cuda", dtype=torch.int16)
    R = flat[offset:offset + nr * d].view(nr, d)
    S = flat[offset + nr * d:].view(ns, d)
    d2 = torch.zeros((nr, ns), dtype=torch.int64, device="cuda")
    for k in range(d):
        d2 += (R[:, k, None].long() - S[None, :, k].long()) ** 2
    T = int(d2.flatten().sort().values[nr * ns // 5])
    want = torch.nonzero(d2 <= T)
    want = (want[:, 0] * ns + want[:, 1]).cpu().numpy().view(np.uint64)
    res = tj.join_result(R, S, eps2=T, screen="int8limb")
    assert np.array_equal(np.sort(res.keys().cpu().numpy().view(np.uint64)), np.sort(want))
    assert res.stats["band"] > 0
