"""Kernels of the decoding path against plain fp32 restatements, at the edges of their tiles."""
import pytest
import torch

from create_llm_by_cupy_b200.ops import functional as F
from create_llm_by_cupy_b200.ops.gemm import gemm

pytestmark = pytest.mark.gpu


def bf(*shape, seed):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(torch.bfloat16)


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("QH,KVH,Tmax,lens", [
    (2, 2, 1, [1]),                                 # one key, R = 1
    (6, 2, 33, [31, 32, 33]),                       # edges of a 32-key tile, 3 of 4 head slots used
    (4, 2, 300, [1, 255, 256, 257, 300]),           # edges of 8 tiles, one per CTA of a cluster; R = 2
    (16, 2, 2100, [2048, 2100, 5]),                 # 8 query heads per KV head: two CTA groups; 9 warps, a tile each
    (32, 8, 130, [129] * 20),                       # many (sequence, head) pairs: clusters of 4 CTAs of two warps
])
def test_decode_attention_edges(D, QH, KVH, Tmax, lens):
    B = len(lens)
    q, kc, vc = bf(B, QH, D, seed=1), bf(B, KVH, Tmax, D, seed=2), bf(B, KVH, Tmax, D, seed=3)
    ln = torch.tensor(lens, dtype=torch.int32)
    for b, n in enumerate(lens):                    # what lies beyond a prefix is never read
        kc[b, :, n:], vc[b, :, n:] = float("nan"), float("nan")
    out = F.decode_attn(q.cuda(), kc.cuda(), vc.cuda(), ln.cuda()).float().cpu()
    ref = F.decode_attn(q.float(), kc.nan_to_num().float(), vc.nan_to_num().float(), ln)
    # half a bf16 ulp of the result, and fp32 sums over at most 2100 weighted values (|v| < 6)
    assert ((out - ref).abs() <= 2.0 ** -8 * ref.abs() + 6 * 2100 * 2.0 ** -23).all()


def test_decode_attention_empty_long_and_unaligned():
    q, kc, vc = (bf(*s, seed=i).cuda() for i, s in enumerate([(3, 4, 64), (3, 2, 40, 64), (3, 2, 40, 64)]))
    out = F.decode_attn(q, kc, vc, torch.tensor([0, -3, 99], dtype=torch.int32, device="cuda"))
    assert (out[:2] == 0).all()                     # no key; a length past the cache means the whole cache
    full = F.decode_attn(q, kc, vc, torch.full((3,), 40, dtype=torch.int32, device="cuda"))
    assert torch.equal(out[2], full[2])
    shifted = [torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")[1:].view(t.shape).copy_(t) for t in (q, kc, vc)]
    assert torch.equal(F.decode_attn(*shifted, torch.full((3,), 40, dtype=torch.int32, device="cuda")), full)


# More 32-key tiles than a cluster has warps, so that warps walk several and rescale what they have summed: 8 CTAs of 4
# warps (more than one CTA per SM) take 32 tiles per round, 8 CTAs of 16 take 128.
ROUNDS = [(8, 32, 8, 128, [2100, 2099, 1025, 1024, 33, 1500, 2048, 700]), (1, 4, 1, 64, [9001]), (2, 2, 2, 32, [4097, 8200])]


@pytest.mark.parametrize("trend", [2.0, -2.0])      # the largest scores come last / first
@pytest.mark.parametrize("B,QH,KVH,D,lens", ROUNDS)
def test_decode_attention_several_tiles_per_warp(B, QH, KVH, D, lens, trend):
    Tmax = max(lens)
    q, kc, vc = bf(B, QH, D, seed=1), bf(B, KVH, Tmax, D, seed=2), bf(B, KVH, Tmax, D, seed=3)
    kc = (kc.float() * torch.exp(torch.linspace(-trend / 2, trend / 2, Tmax))[:, None]).bfloat16()
    ln = torch.tensor(lens, dtype=torch.int32)
    out = F.decode_attn(q.cuda(), kc.cuda(), vc.cuda(), ln.cuda()).double().cpu()
    assert ((out - attention64(q, kc, vc, lens)).abs() <= attention_bound(out, Tmax)).all()


def attention64(q, kc, vc, lens):
    B, QH, D = q.shape
    out = torch.zeros(B, QH, D, dtype=torch.float64)
    for b, n in enumerate(lens):
        k, v = (c[b, :, :n].double().repeat_interleave(QH // kc.shape[1], 0) for c in (kc, vc))
        out[b] = torch.einsum("ht,htd->hd", torch.einsum("hd,htd->ht", q[b].double(), k).mul(D ** -0.5).softmax(-1), v)
    return out


def attention_bound(out, n):
    """Half a bf16 ulp of the result, fp32 sums over n weighted values (|v| < 6), and weights whose exponents (fp32 sums
    below 64 in size) are good to 64 * 2^-22."""
    return 2.0 ** -8 * out.abs() + 6 * (n * 2.0 ** -23 + 64 * 2.0 ** -22)


@pytest.mark.parametrize("B,QH,KVH,D,lens", ROUNDS + [(3, 6, 2, 64, [33, 32, 40]), (2, 8, 2, 128, [1, 300]),
                                                      (2, 4, 2, 64, [33, 33]), (1, 4, 1, 128, [1]), (2, 2, 2, 32, [97, 65])])
def test_decode_append_against_fp64(B, QH, KVH, D, lens):
    """Tables of 0, 1 / 2 and 1 make the rotation exact, so that the rotated rows are known to the last bit."""
    Tmax = max(lens)
    cos, sin = (torch.randint(-2, 3, (Tmax, D // 2), generator=torch.Generator().manual_seed(s)).float() / 2 for s in (7, 8))
    for pos in {Tmax - 1, Tmax // 2, 0}:
        kqv, kc, vc = bf(B, (QH + 2 * KVH) * D, seed=1), bf(B, KVH, Tmax, D, seed=2), bf(B, KVH, Tmax, D, seed=3)
        x1, x2 = kqv[:, :(KVH + QH) * D].float().view(B, -1, 2, D // 2).unbind(2)
        c, s = cos[pos], sin[pos]
        rot = torch.cat([x1 * c - x2 * s, x2 * c + x1 * s], -1).bfloat16()
        kc1, vc1 = kc.clone(), vc.clone()
        kc1[:, :, pos], vc1[:, :, pos] = rot[:, :KVH], kqv[:, (KVH + QH) * D:].view(B, KVH, D)
        kd, vd, ln = kc.cuda(), vc.cuda(), torch.tensor(lens, dtype=torch.int32).cuda()
        out = F.decode_attn_append(kqv.cuda(), kd, vd, ln, pos, QH, KVH, cos.cuda(), sin.cuda(), D ** -0.5).double().cpu()
        assert torch.equal(kd.cpu(), kc1) and torch.equal(vd.cpu(), vc1)
        assert ((out - attention64(rot[:, KVH:], kc1, vc1, lens)).abs() <= attention_bound(out, Tmax)).all()


@pytest.mark.parametrize("Tmax,D", [(20, 64), (700, 128)])
def test_decode_attention_infinite_scores(Tmax, D):
    """Keys whose score is -infinity have no weight; if all are such, or one is +infinity, the result is not a number."""
    q, kc, vc = bf(4, 4, D, seed=1).abs(), bf(4, 2, Tmax, D, seed=2), bf(4, 2, Tmax, D, seed=3)
    kc[0] = -float("inf")
    kc[1, :, 7:] = -float("inf")
    kc[2, :, :Tmax - 3] = -float("inf")
    kc[3, :, 5] = float("inf")
    ln = torch.full((4,), Tmax, dtype=torch.int32)
    out = F.decode_attn(q.cuda(), kc.cuda(), vc.cuda(), ln.cuda()).float().cpu()
    ref = F.decode_attn(q.float(), kc.float(), vc.float(), ln)
    assert ref[[0, 3]].isnan().all() and out[[0, 3]].isnan().all()
    # half a bf16 ulp of the result, and fp32 sums over at most 7 weighted values (|v| < 6)
    assert ((out - ref)[1:3].abs() <= 2.0 ** -8 * ref[1:3].abs() + 6 * 7 * 2.0 ** -22).all()


@pytest.mark.parametrize("trans_b", [False, True])
@pytest.mark.parametrize("M,N,K", [
    (1, 1, 1), (1, 8, 8),                 # smallest
    (7, 63, 65), (8, 64, 64), (9, 65, 63),  # around one tile of columns, one stage of K, 8 rows
    (16, 200, 1000), (17, 768, 768),      # ragged K slices of a cluster; 3 row groups
    (33, 1290, 520), (64, 4104, 2050),    # the widest row count
    (3, 40000, 136),                      # more column tiles than resident CTAs: no K split
])
def test_skinny_gemm_edges(M, N, K, trans_b):
    pad = lambda n: (n + 7) // 8 * 8      # aligned pitches, ragged extents
    a = bf(M, pad(K), seed=1).cuda()[:, :K]
    b = (bf(N, pad(K), seed=2).cuda()[:, :K] if trans_b else bf(K, pad(N), seed=2).cuda()[:, :N])
    ref = a.double() @ (b.double().t() if trans_b else b.double())
    bound = a.double().abs() @ (b.double().abs().t() if trans_b else b.double().abs()) * (K * 2.0 ** -23) + 1e-30
    y = gemm(a, b, trans_b=trans_b, out_dtype=torch.float32, alpha=0.5)
    assert ((y.double() - 0.5 * ref).abs() <= bound).all()              # fp32 sums
    c = bf(M, N, seed=3).cuda()
    want = ref + c.double()
    z = gemm(a, b, trans_b=trans_b, add=c, out=c)                       # in place, bf16 result
    assert ((z.double() - want).abs() <= bound + 2.0 ** -8 * want.abs()).all()


@pytest.mark.parametrize("N", [65535 * 64, 65535 * 64 + 8])      # the most columns of the few-rows grid, and more
def test_gemm_of_few_rows_and_very_many_columns(N):
    a, b = bf(2, 8, seed=1).cuda(), bf(8, N, seed=2).cuda()
    ref, bound = a.double() @ b.double(), a.double().abs() @ b.double().abs() * (8 * 2.0 ** -23)
    assert ((gemm(a, b).double() - ref).abs() <= bound + 2.0 ** -8 * ref.abs()).all()


def test_skinny_gemm_reads_nothing_past_its_operands():
    a, b = torch.full((5, 72), float("nan")).bfloat16().cuda(), torch.full((72, 136), float("nan")).bfloat16().cuda()
    a[:3, :68], b[:68, :131] = 1.0, 1.0
    assert (gemm(a[:3, :68], b[:68, :131]) == 68).all()


@pytest.mark.parametrize("QH,KVH,D,Tmax,pos", [(3, 3, 32, 1, 0), (8, 2, 64, 70, 0), (8, 1, 64, 70, 69), (6, 3, 128, 600, 287),
                                              (12, 4, 64, 600, 288), (32, 8, 128, 300, 256)])
def test_decode_step_fused_append_matches_separate_kernels(QH, KVH, D, Tmax, pos):
    """The one-kernel form against rotation, cache copies and attention as separate kernels."""
    for B in (1, 3, 17):
        kqv = bf(B, (QH + 2 * KVH) * D, seed=1).cuda()
        kc, vc = bf(B, KVH, Tmax, D, seed=2).cuda(), bf(B, KVH, Tmax, D, seed=3).cuda()
        lens = torch.tensor([(pos + 1, pos, Tmax)[i % 3] for i in range(B)], dtype=torch.int32).cuda()   # pos outside / inside
        cos, sin = F.rope_table(Tmax, D, 10000.0, "cuda")
        kc1, vc1, row = kc.clone(), vc.clone(), kqv.clone()
        assert F.decode_append_fusable(kqv, kc, vc, lens, pos, QH, KVH)
        o = F.decode_attn_append(kqv, kc, vc, lens, pos, QH, KVH, cos, sin, D ** -0.5)
        assert torch.equal(kqv, row)
        F.rope_inplace(row, cos, sin, 1, KVH + QH, D, col0=0, pos0=pos)
        kc1[:, :, pos] = row[:, :KVH * D].view(B, KVH, D)
        vc1[:, :, pos] = row[:, (KVH + QH) * D:].view(B, KVH, D)
        assert torch.equal(vc, vc1)
        # a rotated element may round the other way where the compiler fuses the other product
        assert ((kc.float() - kc1.float()).abs() <= 2.0 ** -7 * kc1.float().abs()).all()
        o1 = F.decode_attn(row[:, KVH * D:(KVH + QH) * D].reshape(B, QH, D).contiguous(), kc1, vc1, lens)
        # one bf16 ulp of q or k moves a score by at most 2^-8 sum |q k| / sqrt(D) (< 0.05 here), values stay below 6
        assert (o.float() - o1.float()).abs().max() <= 0.05 and (o == o1).float().mean() > 0.9


def test_decode_append_form_is_left_where_it_does_not_apply():
    kqv, kc, vc = bf(2, 512, seed=1).cuda(), bf(2, 2, 40, 64, seed=2).cuda(), bf(2, 2, 40, 64, seed=3).cuda()
    lens = torch.ones(2, dtype=torch.int32, device="cuda")
    ok = lambda **kw: F.decode_append_fusable(**{**dict(kqv=kqv, kcache=kc, vcache=vc, lens=lens, pos=3, QH=4, KVH=2), **kw})
    assert ok()
    assert not ok(pos=40) and not ok(pos=-1) and not ok(kcache=kc.transpose(1, 2)) and not ok(kqv=kqv[:, ::2])
    assert not ok(kcache=kc.float()) and not ok(kcache=kc[:1]) and not ok(lens=lens.long()) and not ok(kqv=kqv.cpu())


@pytest.mark.parametrize("M,I,K", [(1, 8, 8), (3, 40, 72), (8, 2048, 768), (9, 5504, 2048), (17, 264, 130), (64, 1000, 512)])
def test_skinny_swiglu_edges(M, I, K):
    x, w = bf(M, (K + 7) // 8 * 8, seed=1).cuda()[:, :K], (bf(K, 2 * I, seed=2).float() * K ** -0.5).bfloat16().cuda()
    assert F.gemm_skinny_swiglu_fusable(x, w)
    g, v = (x.double() @ w.double()).chunk(2, 1)
    want = torch.nn.functional.silu(g) * v
    # the activation's slope is at most 1.1 |v| in the gate and |g| in the value, both fp32 sums over K terms below 30
    tol = 2.0 ** -8 * want.abs() + (1.1 * v.abs() + g.abs() + 1e-3) * 30 * K * 2.0 ** -23 + 1e-5 * want.abs()
    assert ((F.gemm_skinny_swiglu(x, w).double() - want).abs() <= tol).all()


@pytest.mark.parametrize("H", [264, 768, 1024])
@pytest.mark.parametrize("M", [1, 5, 148, 149])
def test_rmsnorm_few_rows(M, H):
    x, gamma = bf(M, H, seed=1).cuda(), bf(H, seed=2).cuda()
    y, rstd = F.rmsnorm_fwd(x, gamma)
    r = torch.rsqrt(x.double().square().mean(-1) + 1e-6)
    want = x.double() * r[:, None] * gamma.double()
    assert ((rstd.double() - r).abs() <= 1e-6 * r).all()
    assert ((y.double() - want).abs() <= (2.0 ** -8 + 1e-6) * want.abs()).all()


@pytest.mark.parametrize("B,H,QH,KVH,I", [(1, 64, 2, 1, 8), (3, 256, 4, 2, 264), (16, 768, 12, 4, 2048), (7, 512, 4, 4, 1365)])
def test_one_call_forms_match_the_separate_calls(B, H, QH, KVH, I, monkeypatch):
    from create_llm_by_cupy_b200.models.layers import GroupedQueryAttention, SwiGLU
    g = torch.Generator().manual_seed(0)
    gqa, mlp = GroupedQueryAttention(H, 40, QH, KVH, 2, device="cuda", generator=g), SwiGLU(H, 2, device="cuda", generator=g, ffn_size=I)
    x, res = bf(B, H, seed=1).cuda(), bf(B, 2 * H, seed=2).cuda()[:, :H]              # a residual with a pitch
    kc, vc = bf(B, KVH, 40, H // QH, seed=3).cuda(), bf(B, KVH, 40, H // QH, seed=4).cuda()
    lens = torch.full((B,), 18, dtype=torch.int32, device="cuda")
    for r in (None, res):
        k1, v1, k2, v2 = kc.clone(), vc.clone(), kc.clone(), vc.clone()
        o1, m1 = gqa.decode_step(x, 17, k1, v1, lens, residual=r), mlp.forward(x, residual=r, train_flg=False)
        with monkeypatch.context() as mp:
            mp.setattr(F, "decode_attn_block", lambda *a, **k: None)
            mp.setattr(F, "mlp_few_rows", lambda *a, **k: None)
            o2, m2 = gqa.decode_step(x, 17, k2, v2, lens, residual=r), mlp.forward(x, residual=r, train_flg=False)
        assert torch.equal(o1, o2) and torch.equal(m1, m2) and torch.equal(k1, k2) and torch.equal(v1, v2)
