"""AdamW at the edges of its CTAs, on both grids and with an unaligned shard, against fp64."""
import pytest
import torch

from create_llm_by_cupy_b200.ops import functional as F
from create_llm_by_cupy_b200.ops import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit", [0, 3])                           # whole grid / a limited, streaming one
@pytest.mark.parametrize("gdtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,shift", [(1, 0), (3, 0), (1023, 0), (1024, 0), (1025, 0), (5000, 0), (5000, 1)])
def test_adamw_grids(n, shift, gdtype, limit):
    gen = torch.Generator().manual_seed(0)
    rnd = lambda scale: (torch.randn(n + shift, generator=gen) * scale).cuda()
    grad = rnd(1e-2).to(gdtype)[shift:]
    m, v, w = rnd(1e-3)[shift:], rnd(1e-3).square()[shift:], rnd(0.02)[shift:]
    p = torch.zeros(n + shift, dtype=torch.bfloat16, device="cuda")[shift:]
    lr, b1, b2, eps, wd, step = 1e-3, 0.9, 0.95, 1e-6, 0.1, 7
    g64, m64, v64, w64 = (t.double() for t in (grad, m, v, w))
    m64, v64 = b1 * m64 + (1 - b1) * g64, b2 * v64 + (1 - b2) * g64 * g64
    upd = lr * (m64 / (1 - b1 ** step)) / ((v64 / (1 - b2 ** step)).sqrt() + eps)
    w64 = w64 * (1 - lr * wd) - upd
    old = native.lib().b200_adamw_max_blocks(limit)
    try:
        F.adamw_step(grad, m, v, w, p, lr=lr, beta1=b1, beta2=b2, eps=eps, weight_decay=wd, step=step)
    finally:
        native.lib().b200_adamw_max_blocks(old)
    # a few fp32 roundings per element, relative to the terms that are added
    assert ((m.double() - m64).abs() <= 2e-6 * (m64.abs() + g64.abs())).all()
    assert ((v.double() - v64).abs() <= 2e-6 * v64.abs() + 1e-12).all()
    assert ((w.double() - w64).abs() <= 2e-6 * (w64.abs() + upd.abs()) + 1e-9).all()
    assert torch.equal(p, w.to(torch.bfloat16))
