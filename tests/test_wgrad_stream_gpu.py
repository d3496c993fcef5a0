"""Lifetime of the operands of weight-gradient GEMMs on their side stream."""
import pytest
import torch

from create_llm_by_cupy_b200.ops import gemm as G

pytestmark = pytest.mark.gpu


def operands(seed, M=1024, K=256, N=512):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(M, n, generator=g, device="cuda").bfloat16() for n in (K, N))


def delay(stream=None):
    """Keep the GPU from starting anything on ``stream`` for some 50 ms, so that the host runs ahead."""
    with torch.cuda.stream(stream or torch.cuda.current_stream()):
        torch.cuda._sleep(100_000_000)


def test_memory_is_used_again_while_the_host_is_ahead():
    M, rounds = 1024, 40
    def work():
        a, b = (torch.zeros(M, 2048, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        G.wgrad_gemm(a, b)
        del a, b
        G.wgrad_join()
    work()
    torch.cuda.synchronize()
    before = torch.cuda.memory_reserved()
    delay()
    for _ in range(rounds):
        work()
    grown = torch.cuda.memory_reserved() - before
    torch.cuda.synchronize()
    assert grown <= 4 * M * 2048 * 2 + (32 << 20), grown          # 40 rounds of two such operands are 335 MB


def test_dropped_operands_are_not_overwritten():
    """Operands dropped before the side stream gets to them, with and without a join in reach: other tensors that are
    made meanwhile do not land on them."""
    n = 3 * G.WGRAD_HELD
    want = []
    for i in range(n):
        a, b = operands(i)
        want.append(a.double().t() @ b.double())
    torch.cuda.synchronize()
    ws = G._wgrad_stream(torch.device("cuda", torch.cuda.current_device()))
    for join_every in (1, 4, n):
        delay(ws)
        got = []
        for i in range(n):
            a, b = operands(i)
            got.append(G.wgrad_gemm(a, b))
            shapes = a.shape, b.shape
            del a, b
            noise = [torch.full(s, float("nan"), dtype=torch.bfloat16, device="cuda") for s in shapes]
            assert all(len(h) <= G.WGRAD_HELD for h in G._wgrad_held.values())
            if (i + 1) % join_every == 0:
                G.wgrad_join()
                noise += [torch.full(s, float("nan"), dtype=torch.bfloat16, device="cuda") for s in shapes]
            del noise
        G.wgrad_join()
        for y, w in zip(got, want):
            assert (y.double() - w).norm() <= 2.0 ** -8 * w.norm()
        key = torch.cuda.current_device(), torch.cuda.current_stream().cuda_stream
        assert key not in G._wgrad_held


def test_only_the_issuing_stream_releases_them():
    side = torch.cuda.Stream()
    key = torch.cuda.current_device(), side.cuda_stream
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        a, b = operands(1)
        G.wgrad_gemm(a, b)
    G.wgrad_join()
    assert [(x is a, y is b) for x, y in G._wgrad_held[key]] == [(True, True)]
    with torch.cuda.stream(side):
        G.wgrad_join()
    assert key not in G._wgrad_held
    torch.cuda.synchronize()
