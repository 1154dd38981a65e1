"""The candidate test with 16 R tiles per block and its early exit (large joins) against the same rows
joined as a batch, whose candidate test has neither."""
import pytest
import torch

import tensorjoin_variants_b200 as tj

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,spread", [(15, 8.0), (16, 1.0), (40, 4.0)])
def test_large_join_candidates(d, spread):
    g = torch.Generator(device="cuda").manual_seed(d)
    centres = torch.randn((64, d), generator=g, device="cuda") * spread

    def rows(n):
        at = torch.randint(0, 64, (n,), generator=g, device="cuda")
        return (centres[at] + torch.randn((n, d), generator=g, device="cuda")).contiguous()

    R, S = rows(153_700), rows(131_100)
    i = torch.randint(0, R.shape[0], (1 << 20,), generator=g, device="cuda")
    j = torch.randint(0, S.shape[0], (1 << 20,), generator=g, device="cuda")
    d2 = (R[i].double() - S[j].double()).square().sum(1)
    eps = float(torch.kthvalue(d2, 16).values.sqrt())
    one = tj.join_result(R, S, eps, screen="bf16x3", index_frame="axes")
    assert one.count > 0
    i, j = one.pairs()
    # two joins, so that the batch runs its own candidate test
    many = tj.join_batched_result([(R, S, eps), (R[:300], S[:300], eps)], screen="bf16x3").split()
    assert torch.equal(i, many[0][0]) and torch.equal(j, many[0][1])
