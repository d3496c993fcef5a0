"""Loss whose backward reads the logits that the forward stored: the same as with recomputed ones, whole and in part."""
import pytest
import torch

from create_llm_by_cupy_b200.models.layers import ChunkedCrossEntropy_Share
from create_llm_by_cupy_b200.ops import functional as F

pytestmark = pytest.mark.gpu


def run(x, t, W, chunk, keep, monkeypatch):
    monkeypatch.setattr(ChunkedCrossEntropy_Share, "KEEP_LOGITS_BYTES", keep)
    monkeypatch.setattr(ChunkedCrossEntropy_Share, "KEEP_LOGITS_WIDTH", 0)
    monkeypatch.setattr(ChunkedCrossEntropy_Share, "KEEP_LOGITS_WORK", 0)
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


M, H, V = 4096, 1024, 32000
SIZE = M * V * 4


@pytest.fixture
def limited():
    """Limits what the allocator may hold to ``limited(extra)`` bytes more than what is allocated now."""
    total = torch.cuda.mem_get_info()[1]

    def limit(extra):
        torch.cuda.empty_cache()
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_allocated() + extra) / total)

    yield limit
    torch.cuda.set_per_process_memory_fraction(1.0)


def retries():
    return torch.cuda.memory_stats()["num_alloc_retries"]


def inputs():
    g = torch.Generator(device="cuda").manual_seed(1)
    x, W = (torch.randn(n, H, device="cuda", generator=g).bfloat16() for n in (M, V))
    return x, torch.randint(1, V, (M,), device="cuda", generator=g, dtype=torch.int32), W


def step(layer, x, t, W):
    loss = layer.forward(x, t, W)
    kept = layer.cache[-1] is not None
    dx = layer.backward(W)
    return [kept, *(r.cpu() for r in (loss, dx, layer.dW))]


def same(got, want):
    assert abs(float(got[1] - want[1])) <= M * 2.0 ** -23 * float(want[1])
    for a, b in zip(got[2:], want[2:]):
        assert ((a.float() - b.float()).abs() <= 1e-30).all()


def test_nothing_is_kept_where_memory_is_short(limited):
    x, t, W = inputs()
    want = step(ChunkedCrossEntropy_Share(0, keep_logits_bytes=0), x, t, W)
    assert not want[0]
    layer = ChunkedCrossEntropy_Share(0)
    # enough for the step that recomputes (the gradients of x and W, one chunk of logit gradients twice), not for the logits
    # beside it; a buffer that fits alone is no reason to take it
    for extra in (SIZE // 2, SIZE + (100 << 20), 2 * SIZE):
        limited(extra)
        before = retries()
        for _ in range(3):
            got = step(layer, x, t, W)
            assert not got[0]
            same(got, want)
            del got
        assert retries() == before
    limited(4 * SIZE)
    got = step(layer, x, t, W)
    assert got[0]
    same(got, want)


def test_backward_gives_the_logits_back_when_memory_runs_out(limited, monkeypatch):
    x, t, W = inputs()
    want = step(ChunkedCrossEntropy_Share(0, keep_logits_bytes=0), x, t, W)
    monkeypatch.setattr(F.native, "memory_room", lambda device: (1 << 60, retries()))
    used, kernel = [], F.ce_dlogits_kept
    monkeypatch.setattr(F, "ce_dlogits_kept", lambda *a: (used.append(1), kernel(*a))[1])
    # MiB beside the logits: not enough for the gradient of W (62), then for that but not for a chunk (64) as well, then for all
    for extra, chunks in ((32, (0, 0)), (80, (0, 1)), (140, (0, 4)), (170, (0, 4)), (300, (4, 4))):
        limited(SIZE + (extra << 20))
        layer = ChunkedCrossEntropy_Share(0)
        del used[:]
        got = step(layer, x, t, W)
        assert got[0] and layer.cache is None and chunks[0] <= len(used) <= chunks[1]
        same(got, want)
        del got, layer


def test_a_buffer_that_cost_the_cache_is_not_asked_for_again(limited, monkeypatch):
    x, t, W = inputs()
    layer = ChunkedCrossEntropy_Share(0)
    monkeypatch.setattr(F.native, "memory_room", lambda device: (1 << 60, retries()))
    limited(SIZE + (300 << 20))
    cached = [torch.empty(n << 20, dtype=torch.uint8, device="cuda") for n in (250, 250)]      # in pieces that are too small
    del cached
    assert not step(layer, x, t, W)[0] and layer._refused == SIZE
    before = retries()
    assert not step(layer, x, t, W)[0] and retries() == before
    limited(SIZE // 2)
    refused = ChunkedCrossEntropy_Share(0)
    assert not step(refused, x, t, W)[0] and refused._refused == SIZE


def test_room_by_either_path(monkeypatch):
    keep = torch.empty(100 << 20, dtype=torch.uint8, device="cuda")
    F.native.status_tensor()
    got = F.native.memory_room(keep.device)
    monkeypatch.setattr(F.native, "host", None)
    assert got == F.native.memory_room(keep.device)
    assert got[0] <= torch.cuda.mem_get_info()[1] - torch.cuda.memory_allocated()


def test_two_forwards_hold_one_buffer_and_an_evaluation_none():
    x, t, W = inputs()
    layer = ChunkedCrossEntropy_Share(0)
    layer.forward(x, t, W)
    one = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    layer.forward(x, t, W)
    assert torch.cuda.memory_allocated() <= one + (1 << 20) and torch.cuda.max_memory_allocated() <= one + (64 << 20)
    ChunkedCrossEntropy_Share(0).forward(x, t, W, train_flg=False)
    assert torch.cuda.memory_allocated() <= one + (1 << 20)


@pytest.mark.parametrize("limit", [None, 0])
def test_captured_step(limit):
    x, t, W = inputs()
    layer = ChunkedCrossEntropy_Share(0, keep_logits_bytes=limit)
    want = step(layer, x, t, W)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step(layer, x, t, W)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        loss = layer.forward(x, t, W)
        kept = layer.cache[-1] is not None
        dx = layer.backward(W)
    assert kept == want[0] == (limit is None)
    for _ in range(2):
        dx.fill_(float("nan"))
        layer.dW.fill_(float("nan"))
        g.replay()
        same([kept, loss.cpu(), dx.cpu(), layer.dW.cpu()], want)
