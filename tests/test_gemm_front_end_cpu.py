"""Checks and choices of the GEMM front end that come before any launch. Tensors that call themselves CUDA tensors, and a
library that only records its calls, take the place of the device."""
import pytest
import torch

from create_llm_by_cupy_b200.models.layers import SwiGLU
from create_llm_by_cupy_b200.ops import gemm as G
from create_llm_by_cupy_b200.ops import native


class FakeCuda(torch.Tensor):
    is_cuda = property(lambda self: True)


def fake(*shape, dtype=torch.bfloat16):
    return torch.zeros(*shape, dtype=dtype).as_subclass(FakeCuda)


class Recorder:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda *args: self.calls.append((name, args)) or 0

    def names(self):
        return [name for name, _ in self.calls]


@pytest.fixture
def lib(monkeypatch):
    rec = Recorder()
    empty = torch.empty
    monkeypatch.setattr(torch, "empty", lambda *a, **k: empty(*a, **k).as_subclass(FakeCuda))
    monkeypatch.setattr(G, "_cta_pairs", lambda index: 74)
    monkeypatch.setattr(G, "cluster_splits", lambda M, N, K, dev: 1)
    monkeypatch.setattr(G, "WGRAD_OVERLAP", False)
    monkeypatch.setattr(native, "lib", lambda: rec)
    monkeypatch.setattr(native, "status_tensor", lambda device=None: None)
    monkeypatch.setattr(native, "stream_ptr", lambda: native.c_void_p(0))
    return rec


@pytest.mark.parametrize("K", [64, 192])                      # shorter and longer than the weight's 128
def test_fused_forms_refuse_differing_inner_dimensions(lib, K):
    w = fake(128, 512)                                        # [K, 2 I]
    wt = fake(512, 128)                                       # [N, K]
    few, many = fake(4, K), fake(256, K)
    targets, lse, coef = fake(256, dtype=torch.int32), fake(256, dtype=torch.float32), fake(256, dtype=torch.float32)
    cos = fake(256, 32, dtype=torch.float32)
    for call in (lambda: G.gemm(many, w), lambda: G.gemm_skinny_swiglu(few, w), lambda: G.gemm_swiglu(many, w),
                 lambda: G.gemm_rope(many, w, cos, cos, 256, 64, 128),
                 lambda: G.gemm_swiglu_bwd(many, wt, fake(256, 1024)), lambda: G.gemm_delta(many, wt, fake(256, 512), 256, 64),
                 lambda: G.gemm_ce_stats(many, wt, targets, lse), lambda: G.gemm_ce_dlogits(many, wt, targets, lse, coef)):
        with pytest.raises(ValueError, match="inner dims differ"):
            call()
    assert lib.calls == []


@pytest.mark.parametrize("rows", [4, 256])
@pytest.mark.parametrize("train", [True, False])
def test_swiglu_layer_refuses_an_input_of_another_width(lib, rows, train):
    layer = SwiGLU(128, 2, ffn_size=256)
    layer.params = [p.as_subclass(FakeCuda) for p in layer.params]
    layer.cache_gate = False
    with pytest.raises(ValueError, match="inner dims differ"):
        layer.forward(fake(rows, 192), train_flg=train)
    assert lib.calls == []


@pytest.mark.parametrize("out,error", [(fake(128, 514), None), (fake(128, 514, dtype=torch.float32), None),
                                       (fake(128, 514, dtype=torch.float16), TypeError), (fake(128, 520), AssertionError),
                                       (fake(64, 514), AssertionError), (fake(514, 128).t(), AssertionError)])
def test_gradient_of_a_padded_width_takes_what_the_plain_gemm_takes(lib, out, error):
    x, dgv, I = fake(256, 128), fake(256, 528), 257
    if error is None:
        assert G.wgrad_gemm_gate_value(x, dgv, I, out=out) is out
        return
    with pytest.raises(error):
        G.wgrad_gemm_gate_value(x, dgv, I, out=out)
    assert lib.calls == []


@pytest.mark.parametrize("K", [40, 1024])
def test_one_column_in_a_transposed_view_is_taken(lib, K):
    w = fake(1, K)                                            # w.t(): [K, 1] with strides (1, K)
    assert G.gemm(fake(5, K), w.t()).shape == (5, 1)
    assert G.gemm(w.t(), fake(K, 5), trans_a=True).shape == (1, 5)
    assert ("b200_repitch" in lib.names()) == (K >= 1024)     # the copy that refused such a view


@pytest.mark.parametrize("N,name", [(65535 * 64, "b200_gemm_skinny"), (65535 * 64 + 8, "b200_gemm_bf16")])
def test_more_columns_than_the_few_rows_grid_has(lib, N, name):
    G.gemm(fake(1, 8), fake(8, N))
    assert lib.names() == [name]
    assert G.gemm_skinny_swiglu_fusable(fake(1, 8), fake(8, (N + 15) // 16 * 16)) == (N == 65535 * 64)


@pytest.mark.parametrize("tiles,pending,side,split", [
    ((3, 4), False, None, True), ((3, 8), False, None, True),       # alone
    ((3, 4), True, None, True), ((2, 11), True, None, True), ((3, 8), True, None, False),     # beside weight gradients
    ((3, 4), True, False, False), ((3, 4), True, True, True), ((3, 8), True, True, True),     # a weight gradient itself
])
def test_split_k_beside_other_kernels(lib, monkeypatch, tiles, pending, side, split):
    M, N = (256 * t for t in tiles)
    monkeypatch.setitem(G._wgrad_pending, -1, pending)              # device index of these tensors
    G.gemm(fake(M, 8192), fake(8192, N), side=side)
    assert lib.names()[-1] == ("b200_gemm_bf16_2cta_split" if split else "b200_gemm_bf16_2cta")
    G.gemm(fake(M, 8192), fake(8192, N), side=side, out=fake(M, N + 1)[:, :N])                # through an aligned output
    assert lib.names()[-2] == ("b200_gemm_bf16_2cta_split" if split else "b200_gemm_bf16_2cta")


# us with K split over a cluster of that many pairs / over ranges in a workspace (the best number of them)
BOTH_SPLITS = [
    (256, 256, 2048, 4, 6.8, 11.3), (256, 256, 4096, 4, 8.4, 12.4), (256, 256, 8192, 4, 11.8, 13.8), (256, 256, 16384, 4, 18.5, 16.2),
    (256, 256, 65536, 4, 59.3, 30.6), (512, 512, 4096, 4, 9.3, 13.2), (512, 512, 8192, 4, 13.1, 15.3), (512, 512, 16384, 4, 20.6, 18.8),
    (512, 512, 32768, 4, 35.2, 25.7), (640, 768, 4096, 3, 11.3, 15.2), (768, 768, 8192, 3, 16.6, 18.1), (768, 768, 16384, 3, 26.4, 23.9),
    (768, 1024, 4096, 2, 13.2, 15.6), (768, 1024, 8192, 2, 20.7, 19.3), (768, 1280, 8192, 2, 20.9, 22.8),
    (256, 4096, 11008, 2, 28.4, 29.5), (256, 4096, 22016, 2, 52.4, 45.4), (512, 2048, 8192, 2, 21.3, 23.1),
    (256, 2048, 5504, 3, 13.0, 16.4), (256, 2048, 11008, 3, 19.9, 20.3), (300, 1544, 8192, 2, 20.5, 21.8),
    (777, 768, 32768, 2, 66.9, 41.6), (1024, 1024, 16384, 2, 36.1, 34.4), (400, 2048, 11008, 2, 25.5, 25.9)]


@pytest.mark.parametrize("M,N,K,cluster,us_cluster,us_workspace", BOTH_SPLITS)
def test_a_workspace_has_to_win_its_host_cost_beside_a_cluster_too(M, N, K, cluster, us_cluster, us_workspace):
    assert G.split_count(M, N, K, 74) > 1                    # without the cluster kernel each of them is split
    assert (G.split_count(M, N, K, 74, cluster) > 1) == (us_cluster - us_workspace > 4)


def test_an_addend_that_the_cluster_kernel_does_not_take_leaves_the_workspace_split(lib, monkeypatch):
    monkeypatch.setattr(G, "cluster_splits", lambda M, N, K, dev: 4)
    a, b = fake(256, 4096), fake(4096, 256)
    buf = fake(256 * 264 + 8)
    aligned, base = buf[:256 * 264].view(256, 264)[:, :256], buf[1:256 * 264 + 1].view(256, 264)[:, :256]
    for add, split in ((None, False), (aligned, False), (base, True), (fake(256, 257)[:, :256], True)):
        G.gemm(a, b, add=add)
        assert lib.names()[-1] == ("b200_gemm_bf16_2cta_split" if split else "b200_gemm_bf16_2cta"), add


@pytest.mark.parametrize("M,K,name", [(8, 64, "b200_gemm_skinny"), (9, 504, "b200_gemm_bf16"), (9, 512, "b200_gemm_skinny"),
                                      (64, 511, "b200_gemm_bf16"), (64, 512, "b200_gemm_skinny"), (65, 512, "b200_gemm_bf16")])
def test_few_rows_over_a_short_inner_dimension(lib, M, K, name):
    G.gemm(fake(M, 512)[:, :K], fake(K, 768))
    assert lib.names() == [name]


def test_an_explicit_implementation_holds_for_an_unaligned_output(lib, monkeypatch):
    monkeypatch.setattr(G, "GEMM_IMPL", "1cta")
    G.gemm(fake(256, 64), fake(64, 256), out=fake(256, 257)[:, :256], impl="2cta")
    assert [n for n in lib.names() if n.startswith("b200_gemm_bf16")] == ["b200_gemm_bf16_2cta"]
