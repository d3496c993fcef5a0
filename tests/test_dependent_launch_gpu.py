"""Kernels that start before their predecessor has finished: chains in which every kernel reads what the one before has
just written (weights, gains, lengths and caches among them) give bit for bit what the same chain gives with the device
synchronised between its calls, issued directly and replayed from a CUDA graph."""
import pytest
import torch

from create_llm_by_cupy_b200.ops import functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rand(*shape, seed, scale=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, device=DEV, generator=g) * scale).bfloat16()


def _chain(M, H, sync):
    """Norm, projection, attention or decode step, MLP and back, on weights that are rewritten right before their use."""
    step = torch.cuda.synchronize if sync else (lambda: None)
    D, KVH = 64, 2
    QH = H // D
    N = H + 2 * KVH * D
    x, outs = _rand(M, H, seed=1), []
    src = [_rand(H, N, seed=2, scale=H ** -0.5), _rand(H, H, seed=3, scale=H ** -0.5), _rand(H, 2 * H, seed=4, scale=H ** -0.5)]
    w = [torch.zeros_like(s) for s in src]
    gamma = torch.zeros(H, device=DEV, dtype=torch.bfloat16)
    cos, sin = F.rope_table(256, D, 10000.0, torch.device(DEV, torch.cuda.current_device()))
    kc, vc = (torch.zeros(M, KVH, 256, D, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    lens = torch.zeros(M, dtype=torch.int32, device=DEV)
    for it in range(3):
        big = _rand(2048, 2048, seed=9)
        y = F.gemm(big, big)                                    # keeps the GPU busy while the next calls are issued
        step()
        gamma.copy_(src[0][0, :H] + it)
        h, rstd = F.rmsnorm_fwd(x, gamma)
        step()
        F.add(src[0], src[0], out=w[0])
        if M <= 16:
            lens.fill_(it + 1)
            o = F.decode_attn_append(F.gemm(h, w[0]), kc, vc, lens, it, QH, KVH, cos, sin, 0.125)
        else:
            kqv = F.gemm(h, w[0]).view(1, M, N)
            step()
            k, q, v = (t.unflatten(-1, (-1, D)) for t in kqv.split([KVH * D, H, KVH * D], -1))
            o, lse = F.flash_attn_fwd(q, k, v)
            step()
            outs += F.flash_attn_bwd(o, q, k, v, o, lse)
        step()
        w[1].copy_(src[1])
        x2 = F.gemm(o.reshape(M, H), w[1], add=x)
        step()
        F.add(src[2], src[2], out=w[2])
        act = F.gemm_skinny_swiglu(x2, w[2]) if M <= 16 else F.gemm_swiglu(x2, w[2])[1]
        step()
        dx, dgamma = F.rmsnorm_bwd(act, x, gamma, rstd, add=x2)
        step()
        outs += [y[:4], h, o, x2, act, dx, dgamma]
        x = dx
    return outs + [kc, vc]


@pytest.mark.parametrize("M,H", [(1, 768), (13, 2048), (300, 512), (513, 2048)])
def test_chain_equals_synchronised_chain(M, H):
    want = _chain(M, H, True)
    for _ in range(3):
        for a, b in zip(_chain(M, H, False), want):
            assert torch.equal(a, b)


@pytest.mark.parametrize("M", [1, 300])
def test_chain_in_a_graph(M):
    x, w = _rand(M, 768, seed=1), _rand(768, 768, seed=2, scale=0.03)
    gamma, add = _rand(768, seed=3), _rand(M, 768, seed=4)

    def chain():
        y, acc = x, torch.zeros(M, 768, device=DEV, dtype=torch.bfloat16)      # a memset node before the first kernel
        for _ in range(4):
            y = F.gemm(F.rmsnorm_fwd(y, gamma)[0], w, add=add)
            acc = F.add(acc, y)
        return acc

    want = chain()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        chain()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = chain()
    for _ in range(3):
        got.zero_()
        g.replay()
        assert torch.equal(got, want)
