"""tcgen05 attention forward and backward where their 128-row tiles end: one row, a tile and one row either way, an odd number
of tiles, keys cut inside a tile and at its edge, one and two key tiles to a CTA, sequences of up to 64 tokens."""
import math

import pytest
import torch

from create_llm_by_cupy_b200.ops import functional as F

pytestmark = pytest.mark.gpu
# bf16 rounding is 2^-9 relative at most, 2^-9 / sqrt(3) = 1.1e-3 in the 2-norm. The output carries its own rounding and that of
# P (1.6e-3 together), a gradient its own, that of P or dS, and through delta that of the output (2e-3 to 3e-3).
O_TOL, G_TOL = 4e-3, 8e-3


def _ref(q, k, v, do, valid):
    q, k, v = (t.double().requires_grad_(True) for t in (q, k, v))
    B, T, QH, D = q.shape
    R = QH // k.shape[2]
    s = torch.einsum("bthd,bshd->bhts", q, k.repeat_interleave(R, 2)) / math.sqrt(D)
    pos = torch.arange(T, device=q.device)
    ok = (pos[None, :] <= pos[:, None])[None] & (pos[None, None, :] < valid[:, None, None])
    s = s.masked_fill(~ok[:, None], float("-inf"))
    o = torch.einsum("bhts,bshd->bthd", torch.softmax(s, -1), v.repeat_interleave(R, 2))
    return [o.detach(), torch.logsumexp(s, -1).detach(), *torch.autograd.grad(o, (q, k, v), do.double())]


def _inputs(B, T, QH, KVH, D, lens):
    g = torch.Generator(device="cuda").manual_seed(T + D)
    packed = torch.randn(B, T, (QH + 2 * KVH) * D, device="cuda", generator=g).to(torch.bfloat16)
    k = packed[:, :, :KVH * D].unflatten(2, (KVH, D))
    q = packed[:, :, KVH * D:(KVH + QH) * D].unflatten(2, (QH, D))
    v = packed[:, :, (KVH + QH) * D:].unflatten(2, (KVH, D))
    do = torch.randn(B, T, QH, D, device="cuda", generator=g).to(torch.bfloat16)
    return q, k, v, do, torch.tensor(lens or [T] * B, dtype=torch.int32, device="cuda")


def _check(got, ref, T, names=("o", "lse", "dq", "dk", "dv"), tols=(O_TOL, 1e-5, G_TOL, G_TOL, G_TOL)):
    for name, a, b, tol in zip(names, got, ref, tols):
        err = (a.double() - b).norm() / b.norm().clamp_min(1e-6)
        # one key per row: dq and dk are differences of equal numbers, zero up to their rounding
        if T == 1 and name in ("dq", "dk"):
            assert a.double().abs().max() < 0.1, (name, a)
        else:
            assert err < tol, (name, float(err))


@pytest.fixture(params=[0, 1], ids=["a tile", "two tiles"])
def key_tiles_of_a_cta(request):
    """Of the dK/dV kernels: the second of two tiles runs over the barriers, rings and staging tiles that the first one left."""
    old = F.set_flash_bwd_pairing(request.param)
    yield
    F.set_flash_bwd_pairing(old)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,T,vl", [(1, 1, None), (2, 127, None), (2, 128, [128, 1]), (3, 129, [129, 128, 127]), (1, 255, None),
                                    (2, 257, [256, 130]), (2, 385, [385, 64]), (1, 641, None), (2, 641, [500, 100])])
def test_tile_edges(B, T, vl, D, key_tiles_of_a_cta):
    q, k, v, do, valid = _inputs(B, T, 6, 2, D, vl)
    o, lse = F.flash_attn_fwd(q, k, v, valid_len=valid if vl else None)
    got = [o, lse, *F.flash_attn_bwd(do, q, k, v, o, lse, valid_len=valid if vl else None)]
    _check(got, _ref(q, k, v, do, valid), T)


def _rotated(x, cos, sin, back=False):
    """Half-split pairs of x [B, T, heads, D], turned by their position's angle (or back)."""
    a, b = x.double().chunk(2, -1)
    c, s = (t.double()[:x.shape[1]][None, :, None, :] for t in (cos, sin))
    s = -s if back else s
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _backward_with_rotation(B, T, QH, KVH, D, lens):
    """Gradients as they are and turned back, which is how a layer asks for them, against fp64."""
    q, k, v, do, valid = _inputs(B, T, QH, KVH, D, lens)
    tabs = F.rope_table(T, D, 10000.0, q.device)
    o, lse = F.flash_attn_fwd(q, k, v, valid_len=valid)
    ref = _ref(q, k, v, do, valid)
    _check([o, lse, *F.flash_attn_bwd(do, q, k, v, o, lse, valid_len=valid)], ref, T)
    assert F.flash_bwd_can_unrotate(q)
    got = F.flash_attn_bwd(do, q, k, v, o, lse, valid_len=valid, unrotate=tabs)
    want = [_rotated(ref[2], *tabs, back=True), _rotated(ref[3], *tabs, back=True), ref[4]]
    _check(got, want, T, ("dq", "dk", "dv"), (G_TOL,) * 3)
    for b, n in enumerate(valid.tolist()):                   # keys past the length have no gradient at all
        assert (got[1][b, n:] == 0).all() and (got[2][b, n:] == 0).all()


# Up to 64 tokens head_dim 64 runs 64-query iterations: part of a tile, and a length inside it
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,T,lens", [(1, 2, [2]), (2, 2, [2, 1]), (3, 33, [33, 32, 5]), (2, 63, [63, 1]), (4, 64, [64, 63, 33, 1]),
                                      (2, 65, [65, 64])])
@pytest.mark.parametrize("QH,KVH", [(6, 2), (4, 4), (8, 1)])
def test_short_sequences(B, T, lens, QH, KVH, D):
    _backward_with_rotation(B, T, QH, KVH, D, lens)


# 149 to 443 key tiles: two of them to a CTA without being told, the short sequences' second ones with no query left (a length
# of 40 leaves one key tile, of 600 five of eight); an odd number of tiles, whose middle one is alone
@pytest.mark.parametrize("B,T,lens", [(8, 1024, [1024, 1000, 600, 40, 897, 896, 1, 513]), (10, 641, [641, 600, 129, 1] + [641] * 6)])
def test_two_key_tiles_of_a_cta_by_number(B, T, lens):
    KVH = 4
    assert 148 < -(-T // 128) * KVH * B < 3 * 148
    _backward_with_rotation(B, T, 12, KVH, 64, lens)
