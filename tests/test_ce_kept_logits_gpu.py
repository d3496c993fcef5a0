"""Loss whose backward reads the logits that the forward stored: the same as with recomputed ones, whole and in part."""
import pytest
import torch

from create_llm_by_cupy_b200.models.layers import ChunkedCrossEntropy_Share
from create_llm_by_cupy_b200.ops import functional as F

pytestmark = pytest.mark.gpu


def run(x, t, W, chunk, keep, monkeypatch):
    monkeypatch.setattr(ChunkedCrossEntropy_Share, "KEEP_LOGITS_BYTES", keep)
    monkeypatch.setattr(ChunkedCrossEntropy_Share, "KEEP_LOGITS_WIDTH", 0)
    layer = ChunkedCrossEntropy_Share(0, chunk_size=chunk)
    loss = layer.forward(x, t, W)
    stored = layer.cache[-1]
    dx = layer.backward(W, GradScale=0.5)
    return loss, dx, layer.dW, 0 if stored is None else stored.shape[1]


@pytest.mark.parametrize("M,H,V,chunk", [(256, 64, 256, 8192), (300, 72, 1000, 256), (257, 128, 1003, 512), (777, 768, 8192, 2048),
                                         (513, 64, 33000, 8192), (300, 64, 1001, 8192)])
def test_kept_logits(M, H, V, chunk, monkeypatch):
    g = torch.Generator().manual_seed(M + V)
    x, W = torch.randn(M, H, generator=g).bfloat16().cuda(), (torch.randn(V, H, generator=g) * 0.3).bfloat16().cuda()
    t = torch.randint(1, V, (M,), generator=g, dtype=torch.int32).cuda()
    t[::7] = 0
    base = run(x, t, W, chunk, 0, monkeypatch)
    assert base[3] == 0
    leaf = [x.double().requires_grad_(), W.double().requires_grad_()]
    loss = torch.nn.functional.cross_entropy(leaf[0] @ leaf[1].t(), t.long(), ignore_index=0)
    want = [loss.detach(), *(0.5 * q for q in torch.autograd.grad(loss, leaf))]
    for keep in (M * V * 4, M * chunk * 4, 2 * M * chunk * 4 - 1):
        got = run(x, t, W, chunk, keep, monkeypatch)
        assert got[3] == max([e for e in [*range(chunk, V, chunk), V] if M * e * 4 <= keep], default=0)
        assert abs(float(got[0] - base[0])) <= M * 2.0 ** -23 * float(base[0])        # the sum over rows is atomic
        for a, b, w in zip(got[1:3], base[1:3], want[1:]):
            # the same logits and the same formula: only what lies below the normal range may differ; a last chunk of fewer
            # than 256 columns, or of no multiple of 8, is formed from other row statistics when it is recomputed
            if V % 8 == 0 and (V % chunk == 0 or V % chunk >= 256):
                assert ((a - b).abs() <= 1e-30).all()
            err = [(q.double() - w).norm() / w.norm() for q in (a, b)]
            assert err[0] <= 1.05 * err[1] + 1e-4


def test_chunk_of_kept_logits():
    for M, C, pitch, s in ((5, 8, 8, 0), (3, 4097, 4104, 0), (64, 2050, 6000, 2048), (1, 1, 4, 0), (2, 4095, 8192, 4096)):
        L = torch.randn(M, pitch, device="cuda")[:, s:s + C] if s else torch.randn(M, pitch, device="cuda")[:, :C]
        t = torch.randint(s, s + C, (M,), device="cuda", dtype=torch.int32)
        lse, coef = torch.randn(M, device="cuda") + 3, torch.rand(M, device="cuda")
        p = torch.exp(L.double() - lse.double()[:, None])
        p[torch.arange(M), (t - s).long()] -= 1
        want = p * coef.double()[:, None]
        got = F.ce_dlogits_kept(L, t, lse, coef, s).double()
        # fp32 subtraction and exponential: 2^-22 of an argument of at most 12, then bf16
        assert ((got - want).abs() <= want.abs() * 2.0 ** -8 + (p.abs() + 2) * coef.double()[:, None] * 12 * 2.0 ** -22).all()
