"""Split-K form of the CTA-pair GEMM against the fp64 product."""
import pytest
import torch

from create_llm_by_cupy_b200.ops import gemm as G
from create_llm_by_cupy_b200.ops import native

pytestmark = pytest.mark.gpu


def bf(*shape, seed):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(torch.bfloat16).cuda()


def launches(call):
    before = native.launch_count()
    call()
    return native.launch_count() - before


@pytest.mark.parametrize("trans_a,trans_b", [(True, False), (False, False), (False, True), (True, True)])
@pytest.mark.parametrize("M,N,K", [(256, 256, 4096), (257, 300, 2056), (512, 264, 8192), (768, 1280, 8192), (777, 768, 4104),
                                   (300, 2000, 5504)])
def test_split_k(M, N, K, trans_a, trans_b):
    p8 = lambda n: (n + 7) // 8 * 8
    assert G._splits(M, N, K, 0, None, False) == G.split_count(M, N, K, 74) > 1
    # a bf16 result of a row-major A comes from the cluster kernel, as far as it takes it and has clusters for it
    ranges = G._splits(M, N, K, 0, None, not trans_a and G._cluster_result(N, torch.bfloat16, None))
    assert (ranges == 1) == (not trans_a and N % 8 == 0 and G.cluster_splits(M, N, K, 0) > 1)
    a = bf(K, p8(M), seed=1)[:, :M] if trans_a else bf(M, p8(K), seed=1)[:, :K]
    b = bf(N, p8(K), seed=2)[:, :K] if trans_b else bf(K, p8(N), seed=2)[:, :N]
    # (and a copy where the result's rows do not start on 16-byte boundaries)
    assert launches(lambda: G.gemm(a, b, trans_a=trans_a, trans_b=trans_b)) == (1 if ranges == 1 else 2) + (N % 8 != 0)
    ad, bd = (a.double().t() if trans_a else a.double()), (b.double().t() if trans_b else b.double())
    ref, bound = ad @ bd, ad.abs() @ bd.abs() * (K * 2.0 ** -23)
    y = G.gemm(a, b, trans_a=trans_a, trans_b=trans_b, out_dtype=torch.float32, alpha=0.5)
    assert ((y.double() - 0.5 * ref).abs() <= bound).all()
    assert torch.equal(y, G.gemm(a, b, trans_a=trans_a, trans_b=trans_b, out_dtype=torch.float32, alpha=0.5))
    for dt, ulp in ((torch.bfloat16, 2.0 ** -8), (torch.float32, 2.0 ** -23)):
        c = bf(M, N, seed=3).to(dt)
        want = ref + c.double()
        z = G.gemm(a, b, trans_a=trans_a, trans_b=trans_b, add=c, out=c)
        assert ((z.double() - want).abs() <= bound + ulp * want.abs()).all()


@pytest.mark.parametrize("dt,ulp", [(torch.bfloat16, 2.0 ** -8), (torch.float32, 2.0 ** -23)])
@pytest.mark.parametrize("M,N,K,cpitch", [(257, 301, 4104, 301), (300, 303, 4104, 304), (256, 256, 4096, 259)])
def test_split_k_element_by_element(M, N, K, cpitch, dt, ulp):
    """Columns beyond the last group of four, and an addend whose rows do not start on 16-byte boundaries."""
    a, b = bf(M, K, seed=1), bf(K, (N + 7) // 8 * 8, seed=2)[:, :N]
    c = bf(M, cpitch, seed=3).to(dt)[:, :N]
    assert not G._cluster_result(N, dt, c) and G._splits(M, N, K, 0, None, False) > 1
    assert N % 8 != 0 or launches(lambda: G.gemm(a, b, add=c)) == 2
    want = a.double() @ b.double() + c.double()
    out = torch.full((M, (N + 7) // 8 * 8), 7.0, dtype=dt, device="cuda")
    G.gemm(a, b, add=c, out=out[:, :N])
    bound = a.double().abs() @ b.double().abs() * (K * 2.0 ** -23) + ulp * want.abs()
    assert ((out[:, :N].double() - want).abs() <= bound).all() and (out[:, N:] == 7.0).all()


def test_split_rule():
    assert G.split_count(8192, 2048, 2048, 74) == 1          # enough tiles
    assert G.split_count(768, 768, 768, 74) == 1             # K too short to pay for the second kernel
    for M, N, K in [(256, 256, 1 << 20), (2048, 2048, 8192), (768, 1280, 8192), (1, 1, 64), (100000, 1, 4096)]:
        s = G.split_count(M, N, K, 74)
        tiles = -(-M // 256) * -(-N // 256)
        assert 1 <= s <= 16 and (s == 1 or (tiles * s <= 74 and s <= -(-K // 64)))


@pytest.mark.parametrize("M,N,K", [(777, 768, 768), (300, 264, 2056), (512, 1024, 2048), (256, 256, 16384)])
def test_switched_off(M, N, K, monkeypatch):
    """GEMM_SPLIT_K = 0 (and a weight gradient that has to stay whole): one range of K whatever kernel runs, so the sums are those
    of the single-CTA kernel bit for bit; with the switch on the same shapes are split."""
    a, b, c = bf(M, K, seed=1), bf(K, N, seed=2), bf(M, N, seed=3)
    want, plus = G.gemm(a, b, impl="1cta"), G.gemm(a, b, add=c, impl="1cta")
    assert not torch.equal(G.gemm(a, b), want)
    monkeypatch.setattr(G, "GEMM_SPLIT_K", 0)
    assert torch.equal(G.gemm(a, b), want) and torch.equal(G.gemm(a, b, add=c), plus)
    monkeypatch.setattr(G.native, "host", None)
    assert torch.equal(G.gemm(a, b), want) and torch.equal(G.gemm(a, b, add=c), plus)
    monkeypatch.setattr(G, "GEMM_SPLIT_K", 1)
    assert torch.equal(G.gemm(a, b, side=False), want) and not torch.equal(G.gemm(a, b), want)
