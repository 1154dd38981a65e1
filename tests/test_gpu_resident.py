"""The CTA-pair screen with its R tile held in shared memory: two buffers, one, and none (rows too wide),
with chunks of one tile pair so that the buffers turn over several times per pair of CTAs."""
import numpy as np
import pytest
import torch

import tensorjoin_variants_b200 as tj

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,kw", [(256, {}), (256, {"stages": 2}), (272, {}), (512, {}), (512, {"k_block": 16}),
                                  (528, {}), (640, {}), (640, {"stages": 2})])
def test_resident_rows(d, kw):
    g = torch.Generator(device="cuda").manual_seed(d)
    R = torch.randn((5000, d), generator=g, device="cuda") / d ** 0.5
    S = torch.randn((3001, d), generator=g, device="cuda") / d ** 0.5
    d2 = torch.cdist(R.double(), S.double()) ** 2
    T = float(torch.quantile(d2[:500].flatten(), 0.002))
    # pairs within FP64 rounding of the threshold would make the comparison unsound
    assert float((d2 - T).abs().min()) > 1e-12 * T
    want = torch.nonzero(d2 <= T)
    want = (want[:, 0] * 3001 + want[:, 1]).cpu().numpy().view(np.uint64)
    res = tj.join_result(R, S, eps2=T, screen="fp16", chunk_items=1, **kw)
    assert res.stats["screen_pair"] == 1, res.stats
    assert np.array_equal(np.sort(res.keys().cpu().numpy().view(np.uint64)), np.sort(want))
