"""GEMM operands and FFN widths whose rows do not start on 16-byte boundaries."""
import pytest
import torch

from create_llm_by_cupy_b200.models.layers import SwiGLU
from create_llm_by_cupy_b200.ops import functional as F
from create_llm_by_cupy_b200.ops import gemm as G

pytestmark = pytest.mark.gpu


def bf(*shape, seed, std=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * std).to(torch.bfloat16).cuda()


@pytest.mark.parametrize("R,nseg,C,W,extra", [(1, 1, 1, 1, 0), (3, 1, 8, 8, 1), (5, 2, 7, 8, 0), (300, 2, 1365, 1368, 0),
                                              (17, 1, 100, 104, 3), (2, 3, 16, 16, 5)])
def test_repitch(R, nseg, C, W, extra):
    src = bf(R, nseg * C + extra, seed=1)
    dst = torch.full((R, nseg * W), float("nan"), dtype=torch.bfloat16, device="cuda")
    G.repitch(src, dst, C, W, nseg, C, W)
    d3 = dst.view(R, nseg, W)
    assert torch.equal(d3[:, :, :C], src[:, :nseg * C].reshape(R, nseg, C)) and (d3[:, :, C:] == 0).all()
    back = torch.full_like(src, 7.0)
    G.repitch(dst, back, C, C, nseg, W, C)
    assert torch.equal(back[:, :nseg * C], src[:, :nseg * C]) and (back[:, nseg * C:] == 7.0).all()


@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("trans_a,trans_b", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K", [(5, 3, 7), (63, 65, 1031), (100, 301, 1203), (257, 259, 633), (300, 1365, 130)])
def test_gemm_with_odd_pitches(M, N, K, trans_a, trans_b, out_dtype):
    a, b = bf(*((K, M) if trans_a else (M, K)), seed=1), bf(*((N, K) if trans_b else (K, N)), seed=2)
    c = bf(M, N, seed=3).to(out_dtype)
    ref = (a.double().t() if trans_a else a.double()) @ (b.double().t() if trans_b else b.double())
    bound = (a.double().abs().t() if trans_a else a.double().abs()) @ (b.double().abs().t() if trans_b else b.double().abs())
    bound = bound * (K * 2.0 ** -23) + 2.0 ** -22
    ulp = 2.0 ** -8 if out_dtype == torch.bfloat16 else 2.0 ** -23
    for add in (None, c):
        want = ref if add is None else ref + c.double()
        y = G.gemm(a, b, trans_a=trans_a, trans_b=trans_b, add=add, out_dtype=out_dtype)
        assert y.is_contiguous() and ((y.double() - want).abs() <= bound + ulp * want.abs()).all()
    z = torch.full((M * N + 1,), 3.0, dtype=out_dtype, device="cuda")          # nothing is written past a misaligned output
    G.gemm(a, b, trans_a=trans_a, trans_b=trans_b, out=z[1:].view(M, N))
    assert z[0] == 3.0 and torch.equal(z[1:].view(M, N), G.gemm(a, b, trans_a=trans_a, trans_b=trans_b, out_dtype=out_dtype))


@pytest.mark.parametrize("M,H,I", [(256, 128, 257), (300, 512, 1365), (1000, 1024, 2730), (255, 512, 1365)])
def test_swiglu_layer_with_odd_width(M, H, I):
    layer = SwiGLU(H, 2, device="cuda", ffn_size=I, generator=torch.Generator().manual_seed(0))
    x, res, dout = bf(M, H, seed=1), bf(M, H, seed=2), bf(M, H, seed=3)
    cpu = SwiGLU(H, 2, dtype=torch.float32, ffn_size=I)
    cpu.params = [p.float().cpu() for p in layer.params]
    want = cpu.forward(x.float().cpu(), residual=res.float().cpu())
    wdx = cpu.backward(dout.float().cpu())
    for keep in (True, False):                     # gate kept from the forward, or recomputed in the backward
        layer.cache_gate = keep
        out = layer.forward(x, residual=res)
        into = [torch.full_like(p, float("nan")) for p in layer.params]
        dx = layer.backward(dout, grad_out=into if keep else None)
        F.wgrad_join(dx.device)
        for got, ref in zip((out, dx, *layer.grads), (want, wdx, *cpu.grads)):
            # three bf16 tensors lie between the inputs and a gradient: 2^-9 each, four times that for the norm
            assert got.is_contiguous() and got.shape == ref.shape
            assert (got.float().cpu() - ref).norm() <= 12 * 2.0 ** -9 * ref.norm()
        if keep:
            assert all(g.data_ptr() == i.data_ptr() for g, i in zip(layer.grads, into))
    assert layer.forward(x, train_flg=False).shape == (M, H)


@pytest.mark.parametrize("why", ["misaligned gradient", "epilogue switched off"])
@pytest.mark.parametrize("M,H,I", [(256, 128, 257), (1000, 512, 1365)])
def test_padded_width_backward_without_the_epilogue(M, H, I, why, monkeypatch):
    """The backward of a padded forward through a gradient of the activation in memory."""
    layer = SwiGLU(H, 2, device="cuda", ffn_size=I, generator=torch.Generator().manual_seed(0))
    x, dout = bf(M, H, seed=1), bf(M * H + 1, seed=3)[1:].view(M, H)
    cpu = SwiGLU(H, 2, dtype=torch.float32, ffn_size=I)
    cpu.params = [p.float().cpu() for p in layer.params]
    cpu.forward(x.float().cpu())
    wdx = cpu.backward(dout.float().cpu())
    if why == "epilogue switched off":
        dout = dout.clone()
    layer.forward(x)
    assert layer.cache[1].shape == (M, 2 * ((I + 7) // 8 * 8))
    if why == "epilogue switched off":
        monkeypatch.setattr(F, "SWIGLU_EPILOGUE", False)
    monkeypatch.setattr(F, "gemm_swiglu_bwd", None)                 # not called
    dx = layer.backward(dout)
    F.wgrad_join(dx.device)
    for got, ref in zip((dx, *layer.grads), (wdx, *cpu.grads)):
        # three bf16 tensors lie between the inputs and a gradient: 2^-9 each, four times that for the norm
        assert got.shape == ref.shape and (got.float().cpu() - ref).norm() <= 12 * 2.0 ** -9 * ref.norm()


@pytest.mark.parametrize("pitch", [0, 3])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_gate_value_gradient_into_a_given_matrix(dtype, pitch):
    M, H, I = 300, 512, 1365
    x, dgv = bf(M, H, seed=1), G.pad_gate_value(bf(M, 2 * I, seed=2), I)
    d = torch.cat([dgv[:, :I], dgv[:, 1368:1368 + I]], 1).double()
    ref, bound = x.double().t() @ d, x.double().abs().t() @ d.abs() * (M * 2.0 ** -23)     # fp32 sums
    buf = torch.full((H, 2 * I + pitch), 7.0, dtype=dtype, device="cuda")
    got = F.wgrad_gemm_gate_value(x, dgv, I, out=buf[:, :2 * I])
    F.wgrad_join(x.device)
    assert got.data_ptr() == buf.data_ptr() and got.dtype == dtype and (buf[:, 2 * I:] == 7.0).all()
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23
    assert ((got.double() - ref).abs() <= bound + ulp * ref.abs()).all()


def test_gemm_one_row_without_a_pitch():
    row = bf(1029, seed=1)[None].expand(1, -1).as_strided((1, 1029), (0, 1))      # row stride 0
    b = bf(1029, 37, seed=2)
    want = row.double() @ b.double()
    assert ((G.gemm(row, b).double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-3).all()


@pytest.mark.parametrize("M", [1, 5, 300])
@pytest.mark.parametrize("K", [40, 1024, 1029])
def test_gemm_with_one_column_in_a_transposed_view(M, K):
    a, w = bf(M, K, seed=1), bf(1, K, seed=2)
    want, bound = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t() * (K * 2.0 ** -23)
    for y in (G.gemm(a, w.t()), G.gemm(w.t(), a.t(), trans_a=True).t()):           # [K, 1] with strides (1, K), as B and as A
        assert ((y.double() - want).abs() <= bound + 2.0 ** -8 * want.abs()).all()


def at(t, first):
    """A contiguous copy of ``t`` that starts ``first`` elements behind a 16-byte boundary."""
    return torch.cat([t.new_zeros(first), t.reshape(-1)])[first:].view(t.shape)


# the smallest vector width, every vector kernel of the norms, and a width that none takes
@pytest.mark.parametrize("M,H", [(1, 8), (3, 256), (5, 768), (300, 1024), (300, 2048), (33, 4096), (5, 8192), (3, 8200), (7, 771)])
@pytest.mark.parametrize("first", [(1, 0, 0, 0), (0, 3, 0, 0), (0, 0, 2, 0), (0, 0, 0, 4), (7, 5, 6, 1)])
def test_norm_of_misaligned_bases(M, H, first):
    x, g, dy, add = (at(t, f) for t, f in zip((bf(M, H, seed=1), bf(H, seed=2), bf(M, H, seed=3), bf(M, H, seed=4)), first))
    xd, gd, dyd = x.double(), g.double(), dy.double()
    r = (xd.pow(2).mean(-1, keepdim=True) + 1e-6).rsqrt()
    y, rstd = F.rmsnorm_fwd(x, g)
    assert ((y.double() - xd * r * gd).abs() <= 2.0 ** -8 * (xd * r * gd).abs()).all()
    xh, w = xd * r, dyd * gd
    dx, dgamma = F.rmsnorm_bwd(dy, x, g, rstd, add=add)
    want = r * (w - xh * (w * xh).mean(-1, keepdim=True)) + add.double()
    sums = r * (w.abs() + xh.abs() * (w * xh).abs().mean(-1, keepdim=True)) + add.double().abs()
    assert ((dx.double() - want).abs() <= 2.0 ** -8 * want.abs() + (H + 8) * 2.0 ** -23 * sums).all()
    want, sums = (dyd * xh).sum(0), (dyd * xh).abs().sum(0)
    assert ((dgamma.double() - want).abs() <= 2.0 ** -8 * want.abs() + (M + H) * 2.0 ** -23 * sums).all()


@pytest.mark.parametrize("first", [0, 1, 2, 4, 7])
def test_elementwise_of_misaligned_bases(first):
    W, idx = bf(100, 64, seed=1), torch.tensor([0, 5, 99, 7, 5], dtype=torch.int32, device="cuda")
    want = W[idx.long()]
    want[0] = 0
    assert torch.equal(F.embedding_fwd(at(W, first), idx, 0), want)
    dW, dout = torch.zeros(100, 64, device="cuda"), bf(5, 64, seed=2)
    F.embedding_bwd(dW, idx, at(dout, first), 0)
    assert torch.equal(dW[99], dout[2].float()) and torch.equal(dW[5], dout[1].float() + dout[4].float()) and not dW[0].any()
    gv, dact = bf(300, 528, seed=3), bf(300, 264, seed=4)
    for a, b in ((first, 0), (0, first), (first, first)):
        for got, ref in ((F.swiglu_fwd(at(gv, a)), F.swiglu_fwd(gv)), (F.swiglu_bwd(at(dact, b), at(gv, a)), F.swiglu_bwd(dact, gv))):
            # two roundings of the same fp32 formula
            assert ((got.double() - ref.double()).abs() <= 2.0 ** -7 * ref.double().abs() + 1e-30).all()
        for n in (1, 8, 1027, 70000):
            p, q = bf(n, seed=5), bf(n, seed=6)
            out = at(torch.full((n,), 9.0, dtype=torch.bfloat16, device="cuda"), b)
            assert torch.equal(F.add(at(p, a), at(q, b), out=out), (p.float() + q.float()).bfloat16())
    cos, sin = F.rope_table(32, 64, 10000.0, gv.device)
    buf = bf(30, 256, seed=7)
    want = F.rope_inplace(buf.clone(), cos, sin, 30, 2, 64, 64).double()
    for c, f in (((cos, sin), first), ((at(cos, first), at(sin, first)), 0)):
        got = F.rope_inplace(at(buf, f), *c, 30, 2, 64, 64).double()
        assert ((got - want).abs() <= 2.0 ** -7 * want.abs() + 2.0 ** -22 * buf.double().abs().max()).all()


def test_strided_gains_and_ids():
    x, g2, dy = bf(5, 768, seed=1), bf(1536, seed=2), bf(5, 768, seed=3)
    g = g2[::2]
    y, rstd = F.rmsnorm_fwd(x, g.clone(memory_format=torch.contiguous_format))
    assert torch.equal(F.rmsnorm_fwd(x, g)[0], y)
    wide = torch.stack([rstd, torch.full_like(rstd, float("nan"))], 1)
    for a, b in zip(F.rmsnorm_bwd(dy, x, g, wide[:, 0]), F.rmsnorm_bwd(dy, x, g.clone(memory_format=torch.contiguous_format), rstd)):
        assert torch.equal(a, b)
    W, ids = bf(100, 64, seed=4), torch.tensor([3, 1, 4, 1, 5, 9], dtype=torch.int32, device="cuda")
    assert torch.equal(F.embedding_fwd(W, ids[::2], -1), W[ids[::2].long()])
    dW = F.embedding_bwd(torch.zeros(100, 64, device="cuda"), ids[::2], dy[:3, :64], -1)
    assert torch.equal(dW[ids[::2].long()], dy[:3, :64].float())


def test_embedding_gradient_at_an_odd_base_is_refused():
    idx, dout = torch.tensor([1], dtype=torch.int32, device="cuda"), bf(1, 64, seed=1)
    with pytest.raises(RuntimeError):
        F.embedding_bwd(at(bf(4, 64, seed=2), 1), idx, dout, 0)


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("which", range(3))
def test_attention_gradients_at_misaligned_bases_are_refused(D, which):
    B, T, QH, KVH = 1, 130, 4, 2
    q, k, v = bf(B, T, QH, D, seed=1), bf(B, T, KVH, D, seed=2), bf(B, T, KVH, D, seed=3)
    tabs = F.rope_table(T, D, 10000.0, q.device) if D == 32 else None
    o, lse = F.flash_attn_fwd(q, k, v, rope=tabs)
    out = [torch.empty_like(t) for t in (q, k, v)]
    F.flash_attn_bwd(o, q, k, v, o, lse, rope=tabs, out=out)
    out[which] = at(out[which], 4)
    with pytest.raises(RuntimeError):
        F.flash_attn_bwd(o, q, k, v, o, lse, rope=tabs, out=out)
    if D == 32:
        with pytest.raises(RuntimeError):
            F.flash_attn_fwd(q, k, v, rope=[at(t, int(i == which)) for i, t in enumerate(tabs)] if which < 2 else [at(t, 2) for t in tabs])
