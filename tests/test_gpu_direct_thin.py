"""The line between the direct pass and the index for joins of few rows with many: whole tiles of R rows
count, since the pass computes whole tiles."""
import pytest
import torch

import tensorjoin_variants_b200 as tj

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,ns,d,direct", [(1, 1 << 18, 192, False), (32, 1 << 19, 64, False), (16, 1 << 20, 32, False),
                                            (1, 1 << 17, 192, True), (128, 1 << 20, 8, True)])
def test_line_by_whole_tiles(nr, ns, d, direct):
    g = torch.Generator("cuda").manual_seed(5)
    R, S = torch.rand((nr, d), generator=g, device="cuda"), torch.rand((ns, d), generator=g, device="cuda")
    S[ns // 2] = R[0]
    T = 0.02 * d
    res = tj.join_result(R, S, eps2=T, screen="bf16x3")
    assert (res.stats["ms_index"] == 0.0) == direct
    d2 = torch.cdist(R.double(), S.double(), compute_mode="donot_use_mm_for_euclid_dist") ** 2
    assert not bool(((d2 - T).abs() < 1e-9).any())   # no tie that the order of the sum could decide
    i, j = res.pairs()
    assert torch.equal(i * ns + j, (d2.flatten() <= T).nonzero().flatten())
