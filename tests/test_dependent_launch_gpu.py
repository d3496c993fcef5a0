"""Kernels that start before their predecessor has finished read what it has written.

Pairs: every kind of kernel that lets its successor in early, directly followed by every kind that starts early, the first
one's result being an input of the second (activations, weights, gains, residuals, caches, lengths, statistics). The result
lands in memory that was filled with NaNs before, both are issued behind a delay so that the host has queued them up, and
the second one's outputs have to be those of the same two calls with the device synchronised in between, bit for bit.
Layers: forward and backward with weight gradients on their side stream, against the same with the device synchronised
behind every operator, issued directly and replayed from a CUDA graph."""
import pytest
import torch

from create_llm_by_cupy_b200.models.layers import GroupedQueryAttention, RMSNorm, SwiGLU
from create_llm_by_cupy_b200.ops import functional as F
from create_llm_by_cupy_b200.ops import gemm as G
from create_llm_by_cupy_b200.ops import native

pytestmark = pytest.mark.gpu
DEV = "cuda"
R, C = 512, 2048            # every consumer reads the last R rows of C columns of what was produced


def rnd(*shape, seed=0, std=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, device=DEV, generator=g) * std).bfloat16()


def flat(r):
    return [t for t in (r if isinstance(r, (tuple, list)) else [r]) if t is not None]


def poison(sizes):
    """Free blocks full of NaNs for the allocations that follow: one of each size in bytes."""
    blocks = [torch.full(((n + 1) // 2,), float("nan"), dtype=torch.bfloat16, device=DEV) for n in sizes]
    torch.cuda.synchronize()
    del blocks


# ------------------------------------------------------------------------------------------------- producers
def qkv(t, D):
    """(q, k, v) [1, R, heads, D] from R rows of C columns: 4 query heads to a KV head."""
    n = C // D
    h = t.view(1, -1, n, D)
    return h, h[:, :, :n // 4], h[:, :, n // 4:n // 2]


def _producers():
    x, g = rnd(16384, C, seed=1), rnd(C, seed=2)
    yield "norm", lambda: F.rmsnorm_fwd(x, g)[0]                                     # 592 CTAs that walk over all rows
    rstd = F.rmsnorm_fwd(x, g)[1]
    yield "norm_bwd", lambda: F.rmsnorm_bwd(x, x, g, rstd)[0]
    a, w = rnd(2048, 1024, seed=3), rnd(1024, C, seed=4, std=1 / 32)
    yield "gemm", lambda: F.gemm(a, w)
    yield "gemm_add", lambda: F.gemm(a, w, add=x[:2048])
    wide_w, small_w = rnd(1024, R * C // 8, seed=5, std=1 / 32), rnd(1024, 8192, seed=6, std=1 / 32)
    yield "gemm_few_rows", lambda: F.gemm(a[:8], wide_w).view(-1, C)
    yield "gemm_small", lambda: F.gemm(a[:200], small_w).view(-1, C)
    long_a, long_w, gate = rnd(8192, R, seed=7), rnd(8192, C, seed=8, std=1 / 90), rnd(1024, 2 * C, seed=9, std=1 / 32)
    assert G._splits(R, C, 8192, 0, None, False) > 1            # ranges in a workspace, then their sum
    yield "gemm_split_k", lambda: F.gemm(long_a, long_w, trans_a=True)
    assert G._splits(R, C, 2048, 0, None, True) == 1            # 32 tiles: two ranges each over the 33 clusters of a B200
    yield "gemm_cluster", lambda: F.gemm(x[:R], long_w[:2048])
    yield "gemm_swiglu", lambda: F.gemm_swiglu(a, gate)[1]
    ids = torch.arange(4096, dtype=torch.int32, device=DEV) * 3
    yield "embedding", lambda: F.embedding_fwd(x, ids, -1)

    def repitched():
        dst = torch.empty(4096, C, dtype=torch.bfloat16, device=DEV)
        return G.repitch(wide[:, 3:], dst, C, C)
    wide = rnd(4096, C + 5, seed=10)
    yield "repitch", repitched
    q, kk, v = qkv(rnd(2048, C, seed=11), 128)
    yield "flash_fwd", lambda: F.flash_attn_fwd(q, kk, v)[0].view(-1, C)
    o, lse = F.flash_attn_fwd(q, kk, v)
    yield "flash_bwd", lambda: F.flash_attn_bwd(o, q, kk, v, o, lse)[0].view(-1, C)
    # logits that are single weights: their fp32 words are a zero and a finite number when they are read as bf16
    hot, head = torch.eye(256, device=DEV).bfloat16().repeat(R // 256, 1), rnd(C // 2, 256, seed=12)
    t, tl = torch.zeros(R, dtype=torch.int32, device=DEV), torch.zeros(R, device=DEV)

    def stored():
        logits = torch.empty(R, C // 2, dtype=torch.float32, device=DEV)
        F.gemm_ce_stats(hot, head, t, tl, logits=logits)
        return logits.view(torch.bfloat16)
    yield "ce_stats", stored


# ------------------------------------------------------------------------------------------------- consumers
def _consumers():
    x, g, sq = rnd(R, C, seed=21), rnd(C, seed=22), rnd(C, C, seed=23, std=1 / 45)
    y, rstd = F.rmsnorm_fwd(x, g)
    yield "norm", lambda s: F.rmsnorm_fwd(s, g)
    yield "norm_gain", lambda s: F.rmsnorm_fwd(x, s[-1])
    yield "norm_bwd", lambda s: F.rmsnorm_bwd(s, x, g, rstd)
    yield "norm_bwd_x_add", lambda s: F.rmsnorm_bwd(x, s, s[-1], rstd, add=s)
    # few tiles: K over a cluster
    assert all(G.cluster_splits(R, N, C, 0) > 1 and G._splits(R, N, C, 0, None, True) == 1 for N in (256, R, 768, 1024))
    yield "gemm_cluster", lambda s: F.gemm(s, rnd(C, 768, seed=24))
    yield "gemm_cluster_weight_t", lambda s: F.gemm(x, s, trans_b=True)
    yield "gemm_cluster_add", lambda s: F.gemm(x, sq[:, :1024], add=s[:, :1024])
    # more of them, or a short K: one range
    assert G.cluster_splits(R, 3072, C, 0) == G.cluster_splits(4096, R, C, 0) == G.cluster_splits(R, C, 512, 0) == 1
    wide, tall = rnd(C, 3072, seed=28, std=1 / 45), rnd(4096, C, seed=29)
    yield "gemm", lambda s: F.gemm(s, wide)
    yield "gemm_weight", lambda s: F.gemm(x[:300, :R], s)
    yield "gemm_weight_t", lambda s: F.gemm(tall, s, trans_b=True)
    yield "gemm_weight_grad", lambda s: F.gemm(s, x, trans_a=True)
    yield "gemm_add", lambda s: F.gemm(x[:, :512], sq[:512], add=s)
    yield "gemm_fp32_add", lambda s: F.gemm(x, sq[:, :C // 2], add=s.view(torch.float32))
    yield "gemm_small", lambda s: F.gemm(s[-200:], sq)
    yield "gemm_few_rows", lambda s: F.gemm(s[-7:], sq)
    yield "gemm_few_rows_weight", lambda s: F.gemm(x[:7, :R], s, add=s[:7])
    yield "gemm_cluster_few", lambda s: F.gemm(s, sq[:, :256])
    yield "gemm_cluster_few_add", lambda s: F.gemm(x, sq[:, :256], add=s[:, :256])
    assert G._splits(R, 256, C, 0, None, False) > 1             # an fp32 result: ranges in a workspace, then their sum
    yield "gemm_split_k", lambda s: F.gemm(s, sq[:, :256], out_dtype=torch.float32)
    yield "gemm_split_k_add", lambda s: F.gemm(x, sq[:, :256], add=s.view(torch.float32)[:, :256])
    for D in (64, 128):
        cos, sin = F.rope_table(R, D, 10000.0, x.device)
        yield f"gemm_rope_{D}", lambda s, D=D, c=cos, sn=sin: F.gemm_rope(s, sq, c, sn, R, D, C // 2)
        q, k, v = (t.contiguous() for t in qkv(x, D))
        o, lse = F.flash_attn_fwd(q, k, v)
        yield f"flash_fwd_{D}", lambda s, D=D: F.flash_attn_fwd(*qkv(s, D))
        yield f"flash_bwd_{D}", lambda s, D=D, a=(q, k, v, o, lse): F.flash_attn_bwd(s.view(1, R, C // D, D), *a)
        delta = F.flash_delta(o, x.view(1, R, C // D, D), torch.empty(1, C // D, R, device=DEV))
        yield (f"flash_bwd_qkv_{D}", lambda s, D=D, a=(o, lse), d=delta:
               F.flash_attn_bwd(x.view(1, R, C // D, D), *qkv(s, D), *a, delta=d))
        yield f"gemm_delta_{D}", lambda s, D=D: F.gemm_delta(s, sq, x, R, D)
        yield f"gemm_delta_o_{D}", lambda s, D=D: F.gemm_delta(x, sq, s, R, D)

    w = rnd(C, 2 * 768, seed=25, std=1 / 45)
    yield "gemm_swiglu", lambda s: F.gemm_swiglu(s, w)
    yield "gemm_swiglu_weight", lambda s: F.gemm_swiglu(x[:, :R], s, False)
    gv = F.gemm_swiglu(x, w)[0]
    yield "gemm_swiglu_bwd", lambda s: F.gemm_swiglu_bwd(s, w.view(1536, C)[:768], gv)
    yield "gemm_swiglu_bwd_gv", lambda s: F.gemm_swiglu_bwd(x, sq[:C // 2], s)
    yield "few_rows_swiglu", lambda s: F.gemm_skinny_swiglu(s[-5:], w)
    yield "mlp_few_rows", lambda s: F.mlp_few_rows(s[-5:], w, w.view(1536, C)[:768], s[:5])
    half = w[:, :2 * R].contiguous()
    yield "mlp_few_rows_weight", lambda s: F.mlp_few_rows(x[:5], half, s, x[:5])
    t = torch.arange(R, dtype=torch.int32, device=DEV)
    tl = torch.zeros(R, device=DEV)
    yield "ce_stats", lambda s: F.gemm_ce_stats(s, sq[:1000], t, tl)
    yield "ce_stats_weight", lambda s: F.gemm_ce_stats(x, s, t, tl, logits=torch.empty(R, R, device=DEV))
    lse, coef = torch.full((R,), 9.0, device=DEV), torch.ones(R, device=DEV)
    yield "ce_dlogits", lambda s: F.gemm_ce_dlogits(s, sq[:1000], t, lse, coef)
    yield "ce_dlogits_rows", lambda s: F.gemm_ce_dlogits(x, sq[:1000], t, s.view(torch.float32)[0, :R], s.view(torch.float32)[1, :R])
    yield "ce_dlogits_kept", lambda s: F.ce_dlogits_kept(s.view(torch.float32), t, lse, coef, 0)
    yield "ce_dlogits_kept_rows", lambda s: F.ce_dlogits_kept(x.view(torch.float32), t, s.view(torch.float32)[0, :R], s.view(torch.float32)[1, :R], 0)
    ids = t[::3].contiguous()
    yield "embedding", lambda s: F.embedding_fwd(s, ids, -1)
    yield "repitch", lambda s: G.repitch(s, torch.empty(R, C + 3, dtype=torch.bfloat16, device=DEV)[:, 3:], C, C)
    cos, sin = F.rope_table(R, 64, 10000.0, x.device)
    lens = torch.full((8,), R, dtype=torch.int32, device=DEV)
    kqv, scale = x[:8, :16 * 64].contiguous(), 0.1
    # [8, 4, 512, 64]: caches of 8 sequences, 8 query heads. The last row is written by every call and read from its input.
    kc, vc = rnd(8, 4, R, 64, seed=26), rnd(8, 4, R, 64, seed=27)
    wq, wo = sq[:, :1024].contiguous(), sq[:512]
    a = lens, R - 1, 8, 4, cos, sin, scale
    yield "decode_keys", lambda s: F.decode_attn_append(kqv, s.view(kc.shape), vc, *a)
    yield "decode_values", lambda s: F.decode_attn_append(kqv, kc, s.view(kc.shape), *a)
    yield "decode_kqv", lambda s: F.decode_attn_append(s.view(-1, 1024)[:8], kc, vc, *a)
    yield "decode_query", lambda s: F.decode_attn(s.view(-1, 64)[:64].view(8, 8, 64), kc, vc, lens)
    yield "decode_whole", lambda s: F.decode_attn(kqv.view(-1, 64)[:64].view(8, 8, 64), s.view(kc.shape), s.view(kc.shape), lens)
    yield "decode_block", lambda s: F.decode_attn_block(s[-8:], wq, wo, kc, vc, *a, s[:8])
    yield "decode_block_keys", lambda s: F.decode_attn_block(x[:8], wq, wo, s.view(kc.shape), vc, *a)


@pytest.fixture(scope="module")
def consumers():
    made = list(_consumers())
    torch.cuda.synchronize()
    return made


PRODUCERS = ["norm", "norm_bwd", "gemm", "gemm_add", "gemm_few_rows", "gemm_small", "gemm_split_k", "gemm_cluster", "gemm_swiglu",
             "embedding", "repitch",
             "flash_fwd", "flash_bwd", "ce_stats"]


@pytest.mark.parametrize("producer", PRODUCERS)
def test_pairs(producer, consumers):
    make = dict(_producers())
    assert list(make) == PRODUCERS
    make = make[producer]
    first = make()
    rows, nbytes = first.shape[0], first.untyped_storage().nbytes()
    assert first.shape[1] == C and rows >= R and first.isfinite().all()
    del first
    torch.cuda.synchronize()
    for name, use in consumers:
        torch.cuda.synchronize()
        s = make()[rows - R:]
        torch.cuda.synchronize()
        want = [t.clone() for t in flat(use(s))]
        torch.cuda.synchronize()
        # the poison would show
        bad = flat(use(torch.full_like(s, float("nan"))))
        assert any(not torch.equal(a, b) for a, b in zip(bad, want)), name
        del s, bad
        for _ in range(2):
            poison([nbytes] + [t.untyped_storage().nbytes() for t in want])
            torch.cuda._sleep(200_000)                  # both calls are queued up behind this
            got = flat(use(make()[rows - R:]))
            for a, b in zip(got, want):
                assert torch.equal(a, b), name
    assert native.read_status() == (0, 0)


def test_lengths_written_by_the_kernel_before():
    """Lengths that a copy which lets its successor in early has only just written: shorter and longer than what stood there."""
    B, T, D = 8, 4096, 64
    kc, vc = rnd(B, 4, T, D, seed=1), rnd(B, 4, T, D, seed=2)
    kqv = rnd(B, 16 * D, seed=3)
    cos, sin = F.rope_table(T, D, 10000.0, kc.device)
    for was, now in ((1, T), (T, 1), (-5, 2000), (3000, 17)):
        lens, new = torch.full((4096, B), was, dtype=torch.int32, device=DEV), torch.full((4096, B), now, dtype=torch.int32, device=DEV)
        call = lambda n: F.decode_attn_append(kqv, kc.clone(), vc.clone(), n, T - 1, 8, 4, cos, sin, 0.1)        # noqa: E731
        want = call(new[-1])
        k, v = kc.clone(), vc.clone()
        torch.cuda.synchronize()
        torch.cuda._sleep(200_000)
        G.repitch(new.view(torch.bfloat16), lens.view(torch.bfloat16), 2 * B, 2 * B)
        assert torch.equal(F.decode_attn_append(kqv, k, v, lens[-1], T - 1, 8, 4, cos, sin, 0.1), want)


def test_one_call_forms_against_single_synchronised_operators():
    for B in (1, 3, 8):
        D, H, T, I = 64, 768, 256, 2048
        wq, wo, wg, w2 = (rnd(*s, seed=i, std=s[0] ** -0.5) for i, s in enumerate(((H, 20 * D), (H, H), (H, 2 * I), (I, H))))
        gains, (cos, sin) = rnd(2, H, seed=9), F.rope_table(T, D, 10000.0, wq.device)
        lengths = [torch.full((B,), pos + 1, dtype=torch.int32, device=DEV) for pos in range(6)]

        def tokens(single):
            sync = torch.cuda.synchronize if single else (lambda: None)
            x, outs = rnd(B, H, seed=5), []
            kc, vc = (torch.zeros(B, 4, T, D, device=DEV, dtype=torch.bfloat16) for _ in range(2))
            torch.cuda.synchronize()
            torch.cuda._sleep(2_000_000)
            for pos, lens in enumerate(lengths):
                h = F.rmsnorm_fwd(x, gains[0], keep_rstd=False)[0]
                sync()
                if single:
                    kqv = F.gemm(h, wq)
                    sync()
                    o = F.decode_attn_append(kqv, kc, vc, lens, pos, 12, 4, cos, sin, 0.125)
                    sync()
                    x = F.gemm(o.view(B, H), wo, add=x)
                else:
                    x = F.decode_attn_block(h, wq, wo, kc, vc, lens, pos, 12, 4, cos, sin, 0.125, x)
                sync()
                h = F.rmsnorm_fwd(x, gains[1], keep_rstd=False)[0]
                sync()
                if single:
                    act = F.gemm_skinny_swiglu(h, wg)
                    sync()
                    x = F.gemm(act, w2, add=x)
                else:
                    x = F.mlp_few_rows(h, wg, w2, x)
                sync()
                outs.append(x)
            return [*outs, kc, vc]

        want = tokens(True)
        for _ in range(3):
            for a, b in zip(tokens(False), want):
                assert torch.equal(a, b)


# ------------------------------------------------------------------------------------------------- layers, two streams
def _block(H, QH, KVH, I, B, T):
    gen = torch.Generator(device=DEV).manual_seed(1)
    kw = dict(device=DEV, generator=gen)
    return (RMSNorm(H, device=DEV), GroupedQueryAttention(H, T, QH, KVH, 2, **kw), SwiGLU(H, 2, ffn_size=I, **kw),
            rnd(B * T, H, seed=2), rnd(B * T, H, seed=3))


def _train(parts, B, T):
    norm, attn, mlp, x, dy = parts
    h = attn.forward(norm.forward(x), B, T, None, residual=x)
    y = mlp.forward(h, residual=h)
    dh = mlp.backward(dy)
    dx = norm.backward(attn.backward(dh))
    return [y, dh, dx, *mlp.grads, *attn.grads, *norm.grads]


@pytest.mark.parametrize("H,QH,KVH,I,B,T", [(768, 12, 4, 2048, 2, 300), (768, 12, 4, 2048, 8, 512), (1024, 8, 2, 2730, 1, 777)])
def test_layers_with_weight_gradients_on_their_stream(H, QH, KVH, I, B, T, monkeypatch):
    assert G.WGRAD_OVERLAP
    parts = _block(H, QH, KVH, I, B, T)
    with monkeypatch.context() as mp:
        count = []
        mp.setattr(native, "bump", lambda n=1: (count.append(n), torch.cuda.synchronize()))     # behind every operator
        want = [t.clone() for t in _train(parts, B, T)]
        assert len(count) > 12
    sizes = [t.untyped_storage().nbytes() for t in want]
    for _ in range(3):
        poison(sizes * 3)
        torch.cuda._sleep(2_000_000)
        got = _train(parts, B, T)
        G.wgrad_join()
        for a, b in zip(got, want):
            assert torch.equal(a, b)
        del got
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        _train(parts, B, T)
        G.wgrad_join()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = _train(parts, B, T)
        G.wgrad_join()
    for _ in range(3):
        for t in got:
            t.fill_(float("nan"))
        g.replay()
        for a, b in zip(got, want):
            assert torch.equal(a, b)
    assert native.read_status() == (0, 0)
