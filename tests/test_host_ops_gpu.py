"""The native host path (``chost/host_ops.cpp``) against the general Python path: the same bits for every form that it
takes, the same result or error for every form that it hands back."""
import pytest
import torch

from create_llm_by_cupy_b200.ops import functional as F
from create_llm_by_cupy_b200.ops import gemm as G
from create_llm_by_cupy_b200.ops import native

pytestmark = pytest.mark.gpu
BF, DEV = torch.bfloat16, "cuda"


def rnd(*shape, seed=0, dtype=BF):
    return torch.randn(*shape, device=DEV, generator=torch.Generator(device=DEV).manual_seed(seed)).to(dtype)


def outcome(call):
    try:
        r = call()
    except Exception as e:                                          # noqa: BLE001 - the type is what is compared
        return type(e)
    return [t for t in (r if isinstance(r, (tuple, list)) else [r]) if t is not None]


def same(call, monkeypatch, taken=None):
    """``call`` with and without the host path; ``taken``: whether the host path is the one that ran."""
    native.status_tensor()
    host, count = native.host, [0]

    class Spy:
        def __getattr__(self, name):
            f = getattr(host, name)

            def run(*a):
                r = f(*a)
                if r is not None and name not in ("tma_ok", "split_heads"):
                    count[0] += 1
                return r
            return run

    with monkeypatch.context() as mp:
        mp.setattr(native, "host", Spy())
        got = outcome(call)
    with monkeypatch.context() as mp:
        mp.setattr(native, "host", None)
        want = outcome(call)
    assert isinstance(got, type) == isinstance(want, type), (got, want)
    if isinstance(want, type):
        assert got is want
    else:
        assert len(got) == len(want)
        for a, b in zip(got, want):
            assert a.shape == b.shape and a.dtype == b.dtype and a.stride() == b.stride() and torch.equal(a, b)
    if taken is not None:
        assert (count[0] > 0) == taken
    return got


class Sub(torch.Tensor):
    pass


@pytest.mark.parametrize("make,taken", [
    (lambda: rnd(5, 768), True), (lambda: rnd(2, 3, 768), True), (lambda: rnd(1, 768), True), (lambda: rnd(300, 2048), True),
    (lambda: rnd(7, 771), True), (lambda: rnd(5, 1536)[:, :768], False), (lambda: rnd(768, 5).t(), False),
    (lambda: rnd(5, 768, dtype=torch.float32), False), (lambda: rnd(5, 768).as_subclass(Sub), False),
    (lambda: rnd(5, 768).requires_grad_(), True)])
@pytest.mark.parametrize("keep", [True, False, 1])
def test_rmsnorm(make, taken, keep, monkeypatch):
    x = make()
    g = rnd(x.shape[-1], seed=1)
    same(lambda: F.rmsnorm_fwd(x, g, 1e-5, keep), monkeypatch, taken)
    if x.dtype == BF and x.shape[-1] % 8 == 0:         # the any-width kernel adds its column sums with atomics
        rstd = F.rmsnorm_fwd(x.detach(), g)[1]
        dy, add = rnd(*x.shape, seed=2), rnd(*x.shape, seed=3)
        same(lambda: F.rmsnorm_bwd(dy, x, g, rstd, add=add), monkeypatch, taken)
        same(lambda: F.rmsnorm_bwd(dy, x, g, rstd), monkeypatch, taken)
        same(lambda: F.rmsnorm_bwd(dy, x, g, rstd, add=rnd(2 * x.numel(), seed=4)[::2].view(x.shape)), monkeypatch)


SIZES = [(1, 64, 64), (1, 768, 2048), (8, 40, 72), (9, 504, 264), (9, 512, 264), (64, 512, 3072), (64, 2048, 8200), (65, 768, 768),
         (255, 256, 512), (256, 64, 256), (257, 72, 264), (300, 8192, 264), (777, 2048, 768), (1, 8, 1), (5, 40, 1), (300, 33, 257)]


@pytest.mark.parametrize("M,K,N", SIZES)
@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
def test_gemm(M, K, N, ta, tb, monkeypatch):
    a = rnd(K, M, seed=1) if ta else rnd(M, K, seed=1)
    b = rnd(N, K, seed=2) if tb else rnd(K, N, seed=2)
    for dt in (BF, torch.float32):
        c = rnd(M, N, seed=3).to(dt)
        same(lambda: G.gemm(a, b, trans_a=ta, trans_b=tb, out_dtype=dt), monkeypatch)
        same(lambda: G.gemm(a, b, trans_a=ta, trans_b=tb, add=c, alpha=0.5), monkeypatch)
        for first in (0, 8, 1):
            same(lambda: G.gemm(a, b, trans_a=ta, trans_b=tb, out=rnd(M, N + 9, seed=4).to(dt)[:, first:first + N], add=c), monkeypatch)
    cat = rnd(a.shape[0], 2 * a.shape[1] + 1, seed=5)
    for view in (cat[:, :a.shape[1]], rnd(2 * a.shape[0], a.shape[1], seed=6)[::2], rnd(a.shape[1], a.shape[0], seed=7).t(), a.as_subclass(Sub)):
        same(lambda: G.gemm(view, b, trans_a=ta, trans_b=tb), monkeypatch)


def test_gemm_refusals(monkeypatch):
    a, b = rnd(256, 64), rnd(64, 256)
    for call in (lambda: G.gemm(a, rnd(72, 256)), lambda: G.gemm(a.float(), b), lambda: G.gemm(a, b, out_dtype=torch.float16),
                 lambda: G.gemm(a, b, out=rnd(256, 256, dtype=torch.float32), add=rnd(256, 256)), lambda: G.gemm(a, b, out=rnd(256, 255)),
                 lambda: G.gemm(a, b, out=rnd(256, 256).t()), lambda: G.gemm(a, b, add=rnd(255, 256))):
        assert isinstance(same(call, monkeypatch, False), type)
    for kw, taken in (({}, True), (dict(bn=128), False), (dict(impl="1cta"), False), (dict(force_fallback=True), False),
                      (dict(max_ctas=8), False)):
        same(lambda: G.gemm(a, b, **kw), monkeypatch, taken)


@pytest.mark.parametrize("B,T,QH,KVH,D", [(1, 300, 4, 2, 64), (2, 257, 6, 2, 128), (3, 100, 4, 4, 64)])
def test_attention_and_projection(B, T, QH, KVH, D, monkeypatch):
    H, N = QH * D, (QH + 2 * KVH) * D
    x, w = rnd(B * T, H), rnd(H, N, seed=1)
    cos, sin = F.rope_table(T + 3, D, 10000.0, x.device)
    same(lambda: G.gemm_rope(x, w, cos, sin, T, D, (QH + KVH) * D), monkeypatch, True)
    same(lambda: G.gemm_rope(rnd(B * T, H + 8, seed=2)[:, :H], w, cos, sin, T, D, (QH + KVH) * D), monkeypatch, True)
    for keep in (True, False):
        same(lambda: G.gemm_swiglu(x, rnd(H, 2 * 264, seed=3), keep), monkeypatch, True)
    vl = torch.full((B,), T - 7, dtype=torch.int32, device=DEV)
    for kqv in (rnd(B * T, N, seed=4), rnd(B * T, N + 16, seed=4)[:, :N]):
        q, k, v = same(lambda: F.split_heads(kqv, B, T, QH, KVH, D), monkeypatch)
        same(lambda: F.flash_attn_fwd(q, k, v, valid_len=vl, scale=0.1), monkeypatch, True)
        same(lambda: F.flash_attn_fwd(q, k, v), monkeypatch, True)
        same(lambda: F.flash_attn_fwd(q, k, v, rope=(cos, sin)), monkeypatch, False)


def test_embedding(monkeypatch):
    w, idx = rnd(100, 64), torch.tensor([0, 5, 99, 7], dtype=torch.int32, device=DEV)
    same(lambda: F.embedding_fwd(w, idx, 0), monkeypatch, True)
    same(lambda: F.embedding_fwd(w, idx, -1), monkeypatch, True)
    assert same(lambda: F.embedding_fwd(w, idx.long(), -1), monkeypatch, False) is AssertionError
    assert same(lambda: F.embedding_fwd(rnd(64, 100).t(), idx, -1), monkeypatch, False) is AssertionError
    assert native.read_status() == (0, 0)


@pytest.mark.parametrize("B,D,QH,KVH", [(1, 64, 12, 4), (3, 128, 8, 2), (2, 32, 4, 4)])
@pytest.mark.parametrize("pos", [0, 37, 63, 64])
def test_decode_block(B, D, QH, KVH, pos, monkeypatch):
    H, N, Tmax = QH * D, (QH + 2 * KVH) * D, 64
    x, w0, w1, res = rnd(B, H), rnd(H, N, seed=1), rnd(H, H, seed=2), rnd(B, H, seed=3)
    cos, sin = F.rope_table(128, D, 10000.0, x.device)
    lens = torch.full((B,), min(pos, Tmax - 1) + 1, dtype=torch.int32, device=DEV)
    keep = rnd(2, B, KVH, Tmax, D, seed=4)

    def call(x=x, w0=w0, res=res, dtype=torch.int32):
        kc, vc = keep[0].clone(), keep[1].clone()
        out = F.decode_attn_block(x, w0, w1, kc, vc, lens.to(dtype), pos, QH, KVH, cos, sin, 0.1, res)
        return [out, kc, vc]

    inside = pos < Tmax
    same(call, monkeypatch, inside)
    same(lambda: call(res=None), monkeypatch, inside)
    same(lambda: call(x=rnd(B, H + 8, seed=5)[:, :H], res=rnd(B, H + 1, seed=6)[:, :H]), monkeypatch, inside)
    same(lambda: call(w0=rnd(H, N + 8, seed=7)[:, :N]), monkeypatch, False)
    same(lambda: call(dtype=torch.int64), monkeypatch, False)
    for I in (256, 520, 36):
        wg, wo = rnd(H, 2 * I, seed=8), rnd(I, H, seed=9)
        same(lambda: F.mlp_few_rows(x, wg, wo, res), monkeypatch, I % 8 == 0)
        same(lambda: F.mlp_few_rows(x, wg, wo), monkeypatch, I % 8 == 0)
        same(lambda: F.mlp_few_rows(x, rnd(H + 8, 2 * I, seed=8), wo), monkeypatch, False)
