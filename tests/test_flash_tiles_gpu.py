"""tcgen05 attention forward and backward where their 128-row tiles end: one row, a tile and one row either way, an odd number
of tiles, keys cut inside a tile and at its edge."""
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


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,T,vl", [(1, 1, None), (2, 127, None), (2, 128, [128, 1]), (3, 129, [129, 128, 127]), (1, 255, None),
                                    (2, 257, [256, 130]), (2, 385, [385, 64]), (1, 641, None)])
def test_tile_edges(B, T, vl, D):
    QH, KVH = 6, 2
    g = torch.Generator(device="cuda").manual_seed(T + D)
    packed = torch.randn(B, T, (QH + 2 * KVH) * D, device="cuda", generator=g).to(torch.bfloat16)
    k = packed[:, :, :KVH * D].unflatten(2, (KVH, D))
    q = packed[:, :, KVH * D:(KVH + QH) * D].unflatten(2, (QH, D))
    v = packed[:, :, (KVH + QH) * D:].unflatten(2, (KVH, D))
    do = torch.randn(B, T, QH, D, device="cuda", generator=g).to(torch.bfloat16)
    valid = torch.tensor(vl or [T] * B, dtype=torch.int32, device="cuda")
    o, lse = F.flash_attn_fwd(q, k, v, valid_len=valid if vl else None)
    got = [o, lse, *F.flash_attn_bwd(do, q, k, v, o, lse, valid_len=valid if vl else None)]
    for name, a, b, tol in zip(("o", "lse", "dq", "dk", "dv"), got, _ref(q, k, v, do, valid),
                               (O_TOL, 1e-5, G_TOL, G_TOL, G_TOL)):
        err = (a.double() - b).norm() / b.norm().clamp_min(1e-6)
        # one key per row: dq and dk are differences of equal numbers, zero up to their rounding
        if T == 1 and name in ("dq", "dk"):
            assert a.double().abs().max() < 0.1, (name, a)
        else:
            assert err < tol, (name, float(err))
