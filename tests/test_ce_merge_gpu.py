"""Merge of the loss statistics at the edges of its row and column groups."""
import pytest
import torch

from create_llm_by_cupy_b200.ops import functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 31, 33, 8192])
@pytest.mark.parametrize("nt", [1, 7, 8, 9, 125])
def test_ce_merge_groups(M, nt):
    g = torch.Generator().manual_seed(0)
    pmax, psum = torch.randn(nt, M, generator=g) * 3, torch.rand(nt, M, generator=g) + 0.5
    rmax, rsum = F.ce_merge(pmax.cuda(), psum.cuda())
    want = (psum.double() * (pmax.double() - pmax.double().max(0).values).exp()).sum(0)
    assert torch.equal(rmax.cpu(), pmax.max(0).values)
    # positive terms: fp32 products and sums 125 * 2^-24, the fast exponential of an argument below 24 about 24 * 2^-22
    assert ((rsum.cpu().double() - want).abs() <= 2e-5 * want).all()
