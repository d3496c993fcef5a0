"""Gradient statistics at the edges of their CTAs, against fp64."""
import pytest
import torch

from create_llm_by_cupy_b200.ops import functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,shift", [(1, 0), (7, 1), (2048, 0), (2049, 0), (8 * 2048 + 1, 3), (8192, 0), (8193, 1), (5_000_011, 0)])
def test_grad_stats_clusters(n, shift, dtype):
    g = (torch.randn(n + shift, generator=torch.Generator().manual_seed(0)) * 1e-2).to(dtype).cuda()[shift:]
    stats = torch.tensor([2.0, 0.0], device="cuda")
    F.grad_stats(g, stats)
    want = 2.0 + g.double().square().sum()
    # positive terms: at most 39 additions in a thread's chain, 7 + 5 + 31 above it and 148 at the end; bf16 products are
    # exact, and the chains of fp32 are shorter
    assert abs(float(stats[0]) - float(want)) <= 230 * 2.0 ** -24 * float(want) and float(stats[1]) == 0.0
    for bad in (float("nan"), float("inf")):
        b = g.clone()
        b[n // 2] = bad
        F.grad_stats(b, stats := torch.zeros(2, device="cuda"))
        assert float(stats[1]) == 1.0 and torch.isfinite(stats[0])
