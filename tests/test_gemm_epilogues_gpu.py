"""Epilogues of the CTA-pair GEMM with two warpgroups (addend fetched ahead, delta, rotation, SwiGLU backward) against fp64: part-filled
tiles, several rounds, last rounds of half tiles, inner dimensions on both sides of the dispatch."""
import pytest
import torch

from create_llm_by_cupy_b200.ops import functional as F
from create_llm_by_cupy_b200.ops import gemm as G

pytestmark = pytest.mark.gpu
BF_ULP = 2.0 ** -8


def bf(*shape, seed, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(torch.bfloat16).cuda()


def product(a, b):
    """(fp64 product, bound on the fp32 sums' error)."""
    a, b = a.double(), b.double()
    return a @ b, (a.abs() @ b.abs()) * (a.shape[1] * 2.0 ** -23)


# 256 x 256 tiles: 1, 4 with remainders (over K > 512 the cluster kernel's), 32 (one round, too many for that one), 80 and 100 (a
# round of 74 pairs and half tiles), 152 (two rounds and half tiles)
@pytest.mark.parametrize("M,N", [(256, 256), (300, 264), (513, 1000), (2048, 1024), (2304, 2304), (2048, 3200), (2050, 4104)])
@pytest.mark.parametrize("K", [64, 72, 768, 1280, 1344, 4096])
@pytest.mark.parametrize("trans_b", [False, True])
def test_addend(M, N, K, trans_b):
    assert (G.cluster_splits(M, N, K, 0) > 1) == (M < 2048 and K > 512) and G._splits(M, N, K, 0, None, True) == 1
    a, b, c = bf(M, K, seed=1), bf(K, N, seed=2), bf(M, N, seed=3)
    w = b.t().contiguous() if trans_b else b
    want, bound = product(a, b)
    for alpha in (1.0, 0.5):
        ref = alpha * want + c.double()
        lim = bound + BF_ULP * ref.abs() + 1e-30
        assert ((G.gemm(a, w, trans_b=trans_b, add=c, alpha=alpha).double() - ref).abs() <= lim).all()
        acc = c.clone()                                        # accumulation in place
        G.gemm(a, w, trans_b=trans_b, add=acc, out=acc, alpha=alpha)
        assert ((acc.double() - ref).abs() <= lim).all()
    pitched, addend = bf(M, N + 24, seed=4), bf(M, N + 8, seed=5)
    keep = pitched.clone()
    G.gemm(a, w, trans_b=trans_b, add=addend[:, :N], out=pitched[:, 8:8 + N])
    ref = want + addend[:, :N].double()
    assert ((pitched[:, 8:8 + N].double() - ref).abs() <= bound + BF_ULP * ref.abs() + 1e-30).all()
    assert torch.equal(pitched[:, :8], keep[:, :8]) and torch.equal(pitched[:, 8 + N:], keep[:, 8 + N:])


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,T,heads,K", [(1, 256, 4, 64), (2, 150, 6, 200), (1, 2304, 18, 256), (3, 700, 20, 768), (4, 513, 34, 72)])
def test_delta(D, B, T, heads, K):
    M, N = B * T, heads * D
    dy, w, o = bf(M, K, seed=1, scale=0.1), bf(N, K, seed=2, scale=0.1), bf(M, N, seed=3)
    do, delta = G.gemm_delta(dy, w, o, T, D)
    want, bound = product(dy, w.t())
    assert ((do.double() - want).abs() <= bound + BF_ULP * want.abs() + 1e-30).all()
    prod = (do.double() * o.double()).view(B, T, heads, D)
    lim = prod.abs().sum(-1) * (D * 2.0 ** -23)
    assert ((delta.double().permute(0, 2, 1) - prod.sum(-1)).abs() <= lim + 1e-30).all()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,T,QH,KVH,K", [(1, 256, 2, 2, 64), (2, 150, 6, 2, 200), (1, 2304, 12, 3, 256), (3, 700, 16, 4, 72)])
def test_rotation(D, B, T, QH, KVH, K):
    M, N, cols = B * T, (QH + 2 * KVH) * D, (QH + KVH) * D
    x, w = bf(M, K, seed=1), bf(K, N, seed=2)
    cos, sin = F.rope_table(T, D, 10000.0, x.device)
    y = G.gemm_rope(x, w, cos, sin, T, D, cols).double()
    want, bound = product(x, w)
    pos = torch.arange(M, device=x.device) % T
    c, s = cos.double()[pos][:, None, :], sin.double()[pos][:, None, :]
    h, e = want[:, :cols].reshape(M, -1, D), bound[:, :cols].reshape(M, -1, D)
    x1, x2, e1, e2 = h[..., :D // 2], h[..., D // 2:], e[..., :D // 2], e[..., D // 2:]
    ref = torch.cat([x1 * c - x2 * s, x2 * c + x1 * s], -1).reshape(M, cols)
    # the sums' error through the rotation, and two roundings of fp32 in it
    lim = torch.cat([e1 + e2, e1 + e2], -1).reshape(M, cols) + (x1.abs() + x2.abs()).repeat(1, 1, 2).reshape(M, cols) * 2.0 ** -22
    assert ((y[:, :cols] - ref).abs() <= lim + BF_ULP * ref.abs() + 1e-30).all()
    assert ((y[:, cols:] - want[:, cols:]).abs() <= bound[:, cols:] + BF_ULP * want[:, cols:].abs() + 1e-30).all()


# part-filled groups of 64 columns and groups wholly past the edge (264, 336), one item and several per pair, K of one block
@pytest.mark.parametrize("M,I", [(256, 256), (300, 264), (513, 336), (2304, 2304), (4100, 2736)])
@pytest.mark.parametrize("K", [64, 72, 768, 2048])
def test_swiglu_backward(M, I, K):
    dout, w, gv = bf(M, K, seed=1, scale=0.1), bf(I, K, seed=2, scale=0.1), bf(M, 2 * I, seed=3, scale=2.0)
    got = G.gemm_swiglu_bwd(dout, w, gv).double()
    d, bound = product(dout, w.t())
    gate, value = gv[:, :I].double(), gv[:, I:].double()
    s = torch.sigmoid(gate)
    for out, f in ((got[:, :I], value * s * (1 + gate * (1 - s))), (got[:, I:], gate * s)):
        # the sums' error times the factor, the factor's own (exp, reciprocal and four products in fp32), the rounding; the
        # terms of the gate's factor cancel, hence the bound on their size
        size = (value if out.data_ptr() == got.data_ptr() else torch.ones_like(gate)).abs() * s * (1 + gate.abs())
        lim = bound * f.abs() + d.abs() * size * 2.0 ** -19 + BF_ULP * (d * f).abs() + 1e-30
        assert ((out - d * f).abs() <= lim).all()


# K split over a cluster: 2, 3 (uneven shares of a tile's columns) and 4 pairs to a tile (24 and 26, 18 and 20, 2 and 6 tiles of
# 256 x 128), ranges of unequal length, three k-blocks each at least, tiles cut by M and N, one range up to K = 512; 35 tiles, for
# which a B200 holds too few clusters. Second: what the pairs alone would allow, on a GPU whose SMs make more clusters
CLUSTER_PAIRS = {(1100, 896): (1, 2), (777, 768): (2, 3), (300, 1544): (2, 2), (768, 768): (3, 4), (400, 1200): (3, 3),
                 (256, 256): (4, 4), (300, 264): (4, 4)}


@pytest.mark.parametrize("M,N", list(CLUSTER_PAIRS))
@pytest.mark.parametrize("K", [512, 520, 840, 2056])
@pytest.mark.parametrize("trans_b", [False, True])
def test_cluster_split(M, N, K, trans_b):
    assert G.cluster_splits(M, N, K, 0) in ([1] if K <= 512 else [min(n, -(-K // 64) // 3) for n in CLUSTER_PAIRS[M, N]])
    a, b, c = bf(M, K, seed=1), bf(K, N, seed=2), bf(M, N, seed=3)
    w = b.t().contiguous() if trans_b else b
    want, bound = product(a, b)
    for add, alpha in ((None, 1.0), (c, 1.0), (c, -0.5)):
        ref = alpha * want + (c.double() if add is not None else 0)
        y = G.gemm(a, w, trans_b=trans_b, add=add, alpha=alpha)
        assert ((y.double() - ref).abs() <= bound + BF_ULP * ref.abs() + 1e-30).all()
        assert torch.equal(y, G.gemm(a, w, trans_b=trans_b, add=add, alpha=alpha))
    acc = torch.full((M, N + 16), 7.0, dtype=torch.bfloat16, device="cuda")     # in place, between columns that stay
    acc[:, 8:8 + N] = c
    G.gemm(a, w, trans_b=trans_b, add=acc[:, 8:8 + N], out=acc[:, 8:8 + N])
    assert torch.equal(acc[:, 8:8 + N], G.gemm(a, w, trans_b=trans_b, add=c)) and (acc[:, :8] == 7).all() and (acc[:, 8 + N:] == 7).all()
