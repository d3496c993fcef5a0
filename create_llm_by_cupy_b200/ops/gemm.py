"""bf16 GEMM front end: tcgen05 kernel on CUDA tensors, fp32 torch restatement on CPU tensors.

Replaces the ``cp.matmul`` (cuBLAS) call sites of the reference
(model/fast_layers.py:217,341,420,423,457,458,736,748,794,797,813,815,1328,1351,1435,1464,1471).
"""
from __future__ import annotations

import collections
import ctypes
import functools
import threading

import torch

from . import native

c_void_p, c_float = ctypes.c_void_p, ctypes.c_float

GEMM_OUT_F32 = 1
GEMM_ADD_C = 2
# Few rows: the skinny kernel (weights streamed once, K split over a cluster) instead of 128-row tensor-core tiles.
# Up to 8 rows it always wins (skinny / tiles in us: 768 x 768: 3.6 / 6.8, 2048 x 11008: 11 / 18, 4096 x 22016: 34 / 43).
# Beyond that every 64-column CTA reads the activations again, so the line lies at rows x columns: 16 rows, K x 11008 wins
# (K = 768 9.6 / 10.3, 2048 14.8 / 20, 4096 24.6 / 24.8) but K x 16384 does not (768 15 / 11.5, 2048 25 / 20.6); 32 rows,
# K x 6144 wins (768 8.2 / 9.0, 2048 12.4 / 14.4, 11008 41 / 54), K x 8192 does not (768 10.3 / 9.5, 2048 16.5 / 14.5, 11008
# 60 / 55); 64 rows, K x 3072 wins (768 10.3 / 10.3, 2048 12.4 / 15, 11008 32 / 54), K x 5120 does not (768 10.8 / 10.3,
# 2048 16.5 / 15.6, 11008 55.6 / 54.8). K alone moves it only where it is short, and then the tiles win: K = 256, 32 rows,
# 256 x 2048 8.2 / 6.2; 64 rows 10.3 / 6.2; from K = 512 on 6.2 / 8.0 and 8.2 / 8.2. (The SwiGLU form and the one-call forms
# save launches as well and take a short K too.)
SKINNY_ROWS = 64
SKINNY_AREA = 1 << 18
SKINNY_K = 512
SKINNY_COLS = 65535 * 64        # its grid has one row per 64 columns


def _skinny(M: int, N: int) -> bool:
    if M <= 8:
        return N <= SKINNY_COLS
    return M <= SKINNY_ROWS and (16 if M <= 16 else 32 if M <= 32 else 64) * N < SKINNY_AREA


GEMM_WHOLE_TILES = 8      # CTA-pair kernel: do not split the tiles of a part-filled last round
GEMM_WHOLE_K = 16         # CTA-pair kernel: do not split K over a cluster
_ROUTE_TILES, _ROUTE_SKINNY, _ROUTE_SMALL = range(3)      # kernels of ``native.host.gemm``

# Code-path switches (module attributes; tests and the benchmark's baseline arm set them).
# "1cta": single-CTA 128x256 tiles; "2cta": CTA pairs (cta_group::2) on 256x256 tiles where the
# problem is large enough, single-CTA otherwise.
GEMM_IMPL = "2cta"
# Tile hand-out of the CTA-pair kernel: 1 = tiles beyond each pair's first come from a device
# counter (pairs that start late draw fewer), 0 = fixed round-robin assignment.
GEMM_DYNAMIC_TILES = 1
_dynamic_applied = None
# 1: when the last round of 256x256 tiles would fill less than half of the CTA pairs, those tiles
# are split into 256x128 halves so that twice as many pairs work on it; 0: whole tiles only.
GEMM_HALF_TILES = 1
_half_applied = None


def set_dynamic_tiles(on: bool) -> None:
    global GEMM_DYNAMIC_TILES
    GEMM_DYNAMIC_TILES = int(on)


def set_half_tiles(on: bool) -> None:
    global GEMM_HALF_TILES
    GEMM_HALF_TILES = int(on)


def _apply_dynamic():
    global _dynamic_applied, _half_applied
    if _dynamic_applied != GEMM_DYNAMIC_TILES:
        native.lib().b200_gemm_2cta_dynamic_tiles(int(GEMM_DYNAMIC_TILES))
        _dynamic_applied = GEMM_DYNAMIC_TILES
    if _half_applied != GEMM_HALF_TILES:
        native.lib().b200_gemm_2cta_half_tiles(int(GEMM_HALF_TILES))
        _half_applied = GEMM_HALF_TILES


def _rowmajor_2d(t: torch.Tensor) -> tuple[torch.Tensor, int]:
    """Return (tensor, pitch) for a 2-D view whose last dim is contiguous; copy if it is not."""
    assert t.dim() == 2
    rows, cols = t.shape
    s0, s1 = t.stride()
    if s1 != 1 or (rows > 1 and s0 < cols):
        t = t.contiguous()
        if t.stride(1) != 1:             # one column: contiguous whatever that stride says, so it came back as it was
            t = t.as_strided((rows, cols), (cols, 1))
        s0 = t.stride(0)
    return t, (s0 if rows > 1 else max(cols, s0))


# Operands whose rows do not start on 16-byte boundaries (an FFN width of int(8 H / 3), say) are copied into a pitch
# that is a multiple of 8 and multiplied on the tensor cores: up to three more launches, about 7 us. The CUDA-core kernel
# takes such operands as they are, at 0.27 us per 16 of K and 4.7e12 multiply-adds per second: 128 x 128 x 65 3.1 against
# 9.2 us with the copies, 256 x 256 x 33 3.0 / 11.4, but 2048 x 5460 x 1024 2430 / 50. It stays below both limits.
PAD_WORK = 1 << 25
PAD_K = 1024
# An output of the CTA-pair kernel (256 x 256 and larger) with such a base or pitch goes through an aligned one and a copy:
# the kernel's epilogue would store it element by element (over K = 1024, 256 x 257: 64 us, 18.5 with the copy; 2048 x 2730:
# 97 / 35).


def repitch(src: torch.Tensor, dst: torch.Tensor, cols: int, width: int, nseg: int = 1, sseg: int = 0, dseg: int = 0):
    """Copy ``cols`` columns of each of ``nseg`` column segments of ``src`` [R, ...] to ``dst`` [R, ...] (bf16; segment s at
    columns ``s * sseg`` / ``s * dseg``), zeros in the columns up to ``width`` of a segment of ``dst``."""
    assert src.is_cuda and src.element_size() == dst.element_size() == 2 and src.stride(1) == dst.stride(1) == 1
    native.status_tensor()
    native.check(native.lib().b200_repitch(
        native.ptr(src), native.ptr(dst), src.shape[0], nseg, cols, width, sseg, dseg, ctypes.c_longlong(src.stride(0)),
        ctypes.c_longlong(dst.stride(0)), native.stream_ptr()), "repitch")
    native.bump()
    return dst


def _padded(t: torch.Tensor, ld: int) -> tuple[torch.Tensor, int]:
    """(``t``, pitch) in rows that start on 16-byte boundaries (a copy when they do not already)."""
    if ld % 8 == 0 and t.data_ptr() % 16 == 0:
        return t, ld
    rows, cols = t.shape
    buf = torch.empty((rows, (cols + 7) // 8 * 8), dtype=t.dtype, device=t.device)
    return repitch(t, buf, cols, buf.shape[1])[:, :cols], buf.shape[1]


def _copy_rows(src: torch.Tensor, dst: torch.Tensor) -> torch.Tensor:
    """``dst.copy_(src)`` for 2-D matrices of one dtype (bf16 or fp32) and any pitch."""
    if src.dtype == torch.float32:
        src, dst = src.view(torch.bfloat16), dst.view(torch.bfloat16)
    repitch(src, dst, src.shape[1], src.shape[1])
    return dst


# 1: GEMMs with too few tiles for the CTA pairs run as several K ranges per tile, over a cluster or over a workspace; 0: every
# tile walks K once, so that the sums are those of the other tile kernels (the one that gathers its weight among them).
GEMM_SPLIT_K = 1


def _whole_flags(dev: int, side: bool | None) -> int:
    """Flags of a CTA-pair GEMM on device ``dev`` that keep its tiles or its K whole (``side``: see ``_splits``)."""
    whole = GEMM_WHOLE_TILES if _wgrad_pending.get(dev, False) else 0
    return whole if GEMM_SPLIT_K and side is not False else whole | GEMM_WHOLE_K


@functools.lru_cache(maxsize=4096)
def split_count(M: int, N: int, K: int, pairs: int, cluster: int = 1) -> int:
    """K ranges per 256 x 256 tile (1: no split), by the time each number takes: 0.29 us per 64-deep block of K that one
    pair walks and, for a split, the second kernel with 2 us of launch and the fp32 sums read at about 4 TB/s. A split
    has to win 4 us, what its workspace and second launch cost the host. Measured, one range against the rule's:
    768 x 1280 over K = 8192 44.3 / 22.4 us, 768 x 768 over 8192 44.4 / 17.6, 256 x 4096 over 11008 57.0 / 29.4. Left whole:
    777 x 768 over 2048 (16.6 / 14.2 with 3), 768 x 768 over 1024 (12.0 / 12.4 with 4).

    ``cluster``: ranges of the kernel that splits K over a cluster, if the call takes it (1: it does not). That one has neither
    cost, so a split has to win the same 4 us against it, and 4 more, by which ``cost`` is short of what a split takes (256 x
    4096 over 11008: 24 us more than its launch and tail, ``cost`` says 19). us over the cluster / split: 768 x 768 over 8192 16.6 /
    18.1, 768 x 1280 20.9 / 22.8, 768 x 1024 20.7 / 19.3, 256 x 4096 over 11008 28.4 / 29.5, 512 x 512 over 16384 20.6 / 18.8, all
    left to the cluster; split are 512 x 512 over 32768 35.2 / 25.7, 777 x 768 66.9 / 41.6, 256 x 4096 over 22016 52.4 / 45.4."""
    tiles = -(-M // 256) * -(-N // 256)
    kb = -(-K // 64)
    whole, gain = (0.29 * kb, 4.0) if cluster <= 1 else (0.23 * -(-kb // cluster) + 0.8, 8.0)

    def cost(n):
        return whole if n == 1 else 0.29 * -(-kb // n) + 2.0 + 1e-6 * n * M * N

    best = min(range(1, max(1, min(pairs // tiles, kb // 4, 16)) + 1), key=cost)
    return best if cost(best) < whole - gain else 1


@functools.lru_cache(maxsize=4096)
def cluster_splits(M: int, N: int, K: int, dev: int) -> int:
    """Ranges of K that the CTA-pair kernel splits a bf16 product with a row-major ``a`` into by itself (1: none) on the
    current device ``dev``."""
    return native.lib().b200_gemm_2cta_cluster_splits(M, N, K)


def _cluster_result(N: int, out_dtype: torch.dtype, add: torch.Tensor | None) -> bool:
    """Whether the kernel that splits K over a cluster takes such a result and addend: bf16 in whole 16-byte pieces (an output
    that is not goes through one that is)."""
    return (N % 8 == 0 and out_dtype is torch.bfloat16
            and (add is None or (add.stride(0) % 8 == 0 and add.data_ptr() % 16 == 0)))


def _splits(M: int, N: int, K: int, dev: int, side: bool | None, cluster: bool) -> int:
    """K ranges per tile for one call. ``split_count`` gives the GEMM the GPU to itself; beside another kernel the idle
    pairs are not idle, and what remains of its gain depends on who waits for the result:
      * while weight gradients are pending (``side`` None) a split pays up to three tenths of the pairs in tiles: 777 x 768
        over 4096 (12 tiles), MLP forward + backward 82.8 / 81.5 us whole / split; 1024 x 1280 over 6832 (20) 170.6 / 163.1;
        but 2048 x 768 over 4096 (24) 101.8 / 105.0, 2048 x 1024 over 5472 (32) 165.6 / 169.1;
      * a weight gradient on the side stream that the issuing stream has long work to hide (``side`` False) stays whole:
        split it delays that work (768 x 768 over 8192 beside the attention backward: attention layer 308 / 316 us, 125M
        training pass 8582 / 8671; 2048 x 768 over 8192 beside the MLP's backward: pass 8582 / 8602);
      * one that is waited for soon (``side`` True) is split: 768 x 1280 over 8192 at the end of the attention layer 308 /
        290 us, pass 8582 / 8571 (at 5600 rows 6346 / 6393)."""
    if not GEMM_SPLIT_K or side is False:
        return 1
    pairs = _cta_pairs(dev)
    if side is None and _wgrad_pending.get(dev, False) and -(-M // 256) * -(-N // 256) * 10 > pairs * 3:
        return 1
    return split_count(M, N, K, pairs, cluster_splits(M, N, K, dev) if cluster else 1)


_pairs: dict = {}


def _cta_pairs(index: int) -> int:
    n = _pairs.get(index)
    if n is None:
        n = _pairs[index] = torch.cuda.get_device_properties(index).multi_processor_count // 2
    return n


def gemm(a: torch.Tensor, b: torch.Tensor, *, trans_a: bool = False, trans_b: bool = False,
         out: torch.Tensor | None = None, add: torch.Tensor | None = None,
         out_dtype: torch.dtype | None = None, alpha: float = 1.0, bn: int = 0,
         max_ctas: int = 0, force_fallback: bool = False, impl: str | None = None,
         side: bool | None = None) -> torch.Tensor:
    """``out = alpha * op(a) @ op(b) (+ add)``.

    ``a`` is ``[M, K]`` (``[K, M]`` with ``trans_a``); ``b`` is ``[K, N]`` (``[N, K]`` with
    ``trans_b``). Inputs are bf16 on CUDA; ``out``/``add`` are bf16 or fp32 (same dtype) and
    ``add`` may alias ``out`` (accumulation). Accumulation is fp32 in TMEM. ``side`` marks a weight gradient on the
    side stream (see ``_splits``).
    """
    M, K = (a.shape[1], a.shape[0]) if trans_a else (a.shape[0], a.shape[1])
    Kb, N = (b.shape[1], b.shape[0]) if trans_b else (b.shape[0], b.shape[1])
    if K != Kb:
        raise ValueError(f"gemm: inner dims differ ({K} vs {Kb})")
    if out_dtype is None:
        out_dtype = out.dtype if out is not None else (add.dtype if add is not None else a.dtype)
    if (native.host is not None and (impl or GEMM_IMPL) == "2cta" and bn == 0 and max_ctas == 0 and not force_fallback
            and out_dtype in (torch.bfloat16, torch.float32)):
        splits, whole = 1, 0
        if M <= SKINNY_ROWS and not trans_a and (M <= 8 or K >= SKINNY_K) and _skinny(M, N):
            route = _ROUTE_SKINNY
        elif M >= 256 and N >= 256:
            route = _ROUTE_TILES
            dev = torch._C._cuda_getDevice()
            splits = _splits(M, N, K, dev, side, not trans_a and _cluster_result(N, out_dtype, add))
            if splits == 1:
                _apply_dynamic()
                whole = _whole_flags(dev, side)
        else:
            route = _ROUTE_SMALL
        res = native.host.gemm(a, b, trans_a, trans_b, out, add, out_dtype is torch.float32, alpha, whole, route, splits)
        if res is not None:
            native.bump(2 if splits > 1 else 1)
            return res

    if not a.is_cuda:
        af = a.float().t() if trans_a else a.float()
        bf = b.float().t() if trans_b else b.float()
        res = (af @ bf) * alpha
        if add is not None:
            res = res + add.float()
        res = res.to(out_dtype)
        if out is not None:
            out.copy_(res)
            return out
        return res

    if a.dtype != torch.bfloat16 or b.dtype != torch.bfloat16:
        raise TypeError("gemm: CUDA operands must be bf16")
    if out_dtype not in (torch.bfloat16, torch.float32):
        raise TypeError("gemm: out dtype must be bf16 or fp32")
    a, lda = _rowmajor_2d(a)
    b, ldb = _rowmajor_2d(b)
    if out is None:
        out = torch.empty((M, N), dtype=out_dtype, device=a.device)
    assert out.dim() == 2 and out.shape == (M, N) and out.stride(1) == 1 and out.dtype == out_dtype
    ldd = out.stride(0) if M > 1 else max(N, out.stride(0))
    flags = GEMM_OUT_F32 if out_dtype == torch.float32 else 0
    ldc = 0
    if add is not None:
        assert add.shape == (M, N) and add.stride(1) == 1 and add.dtype == out_dtype
        ldc = add.stride(0) if M > 1 else max(N, add.stride(0))
        flags |= GEMM_ADD_C
    native.status_tensor()
    impl = impl or GEMM_IMPL
    lib = native.lib()
    if impl == "2cta" and not force_fallback and bn == 0 and max_ctas == 0:
        pa, pb = a.data_ptr(), b.data_ptr()
        ok = (lda | ldb) % 8 == 0 and (pa | pb) % 16 == 0
        if not ok and M * N > 0 and (M * N * K >= PAD_WORK or K >= PAD_K):
            (a, lda), (b, ldb) = _padded(a, lda), _padded(b, ldb)
            pa, pb, ok = a.data_ptr(), b.data_ptr(), True
        if ok and M <= SKINNY_ROWS and not trans_a and (M <= 8 or K >= SKINNY_K) and _skinny(M, N):
            rc = lib.b200_gemm_skinny(
                c_void_p(pa), c_void_p(pb), native.ptr(out), native.ptr(add), M, N, K, lda, ldb, ldd, ldc,
                int(not trans_b), flags & GEMM_OUT_F32, c_float(alpha), native.stream_ptr())
            native.check(rc, "b200_gemm_skinny")
            native.bump()
            return out
        if ok and M >= 256 and N >= 256:
            po = out.data_ptr()
            if po % 16 or ldd * (4 if flags & GEMM_OUT_F32 else 2) % 16:
                tmp = torch.empty((M, (N + 7) // 8 * 8), dtype=out_dtype, device=a.device)[:, :N]
                if add is not None:
                    _copy_rows(add, tmp)
                gemm(a, b, trans_a=trans_a, trans_b=trans_b, out=tmp, add=None if add is None else tmp, alpha=alpha,
                     impl=impl, side=side)
                _copy_rows(tmp, out)
                return out
            dev = a.get_device()
            splits = _splits(M, N, K, dev, side, not trans_a and _cluster_result(N, out_dtype, add))
            if splits > 1:
                ws = torch.empty(splits * (-(-M // 256) * 256) * (-(-N // 4) * 4), dtype=torch.float32, device=a.device)
                rc = lib.b200_gemm_bf16_2cta_split(
                    c_void_p(pa), c_void_p(pb), c_void_p(po), native.ptr(add), M, N, K, lda, ldb, ldd, ldc, int(trans_a),
                    int(not trans_b), flags, c_float(alpha), native.ptr(ws), splits, native.stream_ptr())
                native.check(rc, "b200_gemm_bf16_2cta_split")
                native.bump(2)
                return out
            _apply_dynamic()
            # Half tiles shorten the tail of a GEMM that has the GPU to itself. While weight-gradient GEMMs
            # are in flight on the side stream the tail is filled by the other kernel's CTAs, and narrower
            # tiles only cost efficiency (measured on the 1.3 B step: 1.1 ms faster alone, 1.2 ms slower beside).
            flags |= _whole_flags(dev, side)
            rc = lib.b200_gemm_bf16_2cta(
                c_void_p(pa), c_void_p(pb), c_void_p(po), native.ptr(add), M, N, K, lda, ldb, ldd, ldc, int(trans_a),
                int(not trans_b), flags, c_float(alpha), native.stream_ptr())
            native.check(rc, "b200_gemm_bf16_2cta")
            native.bump()
            return out
    rc = lib.b200_gemm_bf16(
        native.ptr(a), native.ptr(b), native.ptr(out), native.ptr(add),
        M, N, K, lda, ldb, ldd, ldc, int(trans_a), int(not trans_b), flags,
        ctypes.c_float(alpha), bn, max_ctas, int(force_fallback), native.stream_ptr())
    native.check(rc, "b200_gemm_bf16")
    native.bump()
    return out


# Rotary embedding in the epilogue of the CTA-pair kernel instead of an in-place pass over the output.
GEMM_ROPE_EPILOGUE = True


_rope_t_cache: dict = {}


def rope_tables_transposed(cos: torch.Tensor, sin: torch.Tensor):
    """([D/2, T] cos, [D/2, T] sin) copies of the [T, D/2] rotary tables, cached per table. The kernels'
    epilogues own one row (position) per thread, so a warp reads consecutive words from this layout."""
    key = (cos.data_ptr(), sin.data_ptr(), tuple(cos.shape))
    tt = _rope_t_cache.get(key)
    if tt is None:
        if len(_rope_t_cache) > 16:
            _rope_t_cache.clear()
        tt = _rope_t_cache[key] = (cos.t().contiguous(), sin.t().contiguous(), cos, sin)   # keeps the sources alive
    return tt


def gemm_rope_fusable(a: torch.Tensor, b: torch.Tensor, head_dim: int, rope_cols: int) -> bool:
    """True when ``gemm_rope(a, b, ...)`` (``a`` [M, K], ``b`` [K, N], both row-major bf16) runs with the
    rotation fused into the GEMM epilogue."""
    if not (GEMM_ROPE_EPILOGUE and a.is_cuda and GEMM_IMPL == "2cta" and head_dim in (64, 128)):
        return False
    M, N = a.shape[0], b.shape[1]
    return bool(M >= 256 and N >= 256 and N % 8 == 0 and rope_cols % head_dim == 0 and 0 < rope_cols <= N and _tma_ok(a, b))


def gemm_rope(a: torch.Tensor, b: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, T: int, head_dim: int,
              rope_cols: int) -> torch.Tensor:
    """``a @ b`` whose first ``rope_cols`` output columns are heads of width ``head_dim`` rotated by the
    rotary embedding of position ``row % T`` (half-split pairing, tables fp32 [>= T, head_dim / 2]).
    Only where ``gemm_rope_fusable`` holds."""
    M, K = a.shape
    N = b.shape[1]
    _same_inner("gemm_rope", K, b.shape[0])
    assert gemm_rope_fusable(a, b, head_dim, rope_cols)
    assert cos.dtype == torch.float32 and sin.dtype == torch.float32 and cos.is_contiguous() and sin.is_contiguous()
    assert cos.shape[0] >= T and cos.shape[1] == head_dim // 2
    native.status_tensor()
    _apply_dynamic()
    flags = GEMM_WHOLE_TILES if _wgrad_pending.get(a.device.index, False) else 0
    # the epilogue reads the tables transposed ([head_dim / 2][positions]): a thread owns a row, so a warp
    # then reads consecutive words
    tt = rope_tables_transposed(cos, sin)
    if native.host is not None:
        out = native.host.gemm_rope(a, b, tt[0], tt[1], T, head_dim, rope_cols, flags)
        if out is not None:
            native.bump()
            return out
    out = torch.empty((M, N), dtype=torch.bfloat16, device=a.device)
    rc = native.lib().b200_gemm_bf16_2cta_rope(
        native.ptr(a), native.ptr(b), native.ptr(out), M, N, K, a.stride(0), b.stride(0), N, 0, 1, flags,
        native.ptr(tt[0]), native.ptr(tt[1]), T, tt[0].shape[1], rope_cols, head_dim, native.stream_ptr())
    native.check(rc, "b200_gemm_bf16_2cta_rope")
    native.bump()
    return out


def _tma_ok(*ts) -> bool:
    if native.host is not None:
        ok = native.host.tma_ok(*ts)
        if ok is not None:
            return ok
    return all(t.is_cuda and t.dtype == torch.bfloat16 and t.dim() == 2 and t.stride(1) == 1 and t.stride(0) % 8 == 0
               and t.data_ptr() % 16 == 0 for t in ts)


def _same_inner(what: str, K: int, Kb: int) -> None:
    """The kernels take one inner dimension for both operands: a shorter one would be read past its end."""
    if K != Kb:
        raise ValueError(f"{what}: inner dims differ ({K} vs {Kb})")


def _whole_tiles_flag(device) -> int:
    return GEMM_WHOLE_TILES if _wgrad_pending.get(device.index, False) else 0


def gemm_swiglu_fusable(x: torch.Tensor, w_gate_val: torch.Tensor) -> bool:
    """True when ``gemm_swiglu(x, w_gate_val)`` runs as one kernel (``x`` [M, K], ``w_gate_val`` [K, 2 I], bf16)."""
    if not (x.is_cuda and GEMM_IMPL == "2cta" and _tma_ok(x, w_gate_val)):
        return False
    I = w_gate_val.shape[1] // 2
    return x.shape[0] >= 256 and I >= 128 and w_gate_val.shape[1] == 2 * I and I % 8 == 0


def gemm_swiglu(x: torch.Tensor, w_gate_val: torch.Tensor, keep_gv: bool = True):
    """``gv = x @ [W_gate | W_value]`` and ``act = silu(gate) * value`` from ONE GEMM whose epilogue applies the
    activation to the fp32 accumulator (a tile holds 128 gate columns beside the matching 128 value columns).
    Returns ``(gv [M, 2 I] or None, act [M, I])``; ``gv`` is only written when ``keep_gv`` (the backward reads it).
    Only where ``gemm_swiglu_fusable`` holds."""
    M, K = x.shape
    I = w_gate_val.shape[1] // 2
    _same_inner("gemm_swiglu", K, w_gate_val.shape[0])
    assert gemm_swiglu_fusable(x, w_gate_val)
    native.status_tensor()
    _apply_dynamic()
    if native.host is not None:
        r = native.host.gemm_swiglu(x, w_gate_val, keep_gv, _whole_tiles_flag(x.device))
        if r is not None:
            native.bump()
            return r
    act = torch.empty((M, I), dtype=torch.bfloat16, device=x.device)
    gv = torch.empty((M, 2 * I), dtype=torch.bfloat16, device=x.device) if keep_gv else None
    rc = native.lib().b200_gemm_bf16_2cta_swiglu(
        native.ptr(x), native.ptr(w_gate_val), native.ptr(gv), native.ptr(act), M, I, K, x.stride(0),
        w_gate_val.stride(0), 2 * I, I, _whole_tiles_flag(x.device), native.stream_ptr())
    native.check(rc, "b200_gemm_bf16_2cta_swiglu")
    native.bump()
    return gv, act


def gemm_skinny_swiglu_fusable(x: torch.Tensor, w_gate_val: torch.Tensor) -> bool:
    """True when ``gemm_skinny_swiglu(x, w_gate_val)`` runs: few rows (``x`` [M, K], ``w_gate_val`` [K, 2 I], bf16)."""
    return (x.is_cuda and GEMM_IMPL == "2cta" and x.dim() == 2 and w_gate_val.shape[1] % 16 == 0
            and 0 < x.shape[0] and _skinny(x.shape[0], w_gate_val.shape[1]) and _tma_ok(x, w_gate_val))


def gemm_skinny_swiglu(x: torch.Tensor, w_gate_val: torch.Tensor) -> torch.Tensor:
    """``silu(x @ W_gate) * (x @ W_value)`` [M, I] for few rows, in one kernel that stores only the activation. Only where
    ``gemm_skinny_swiglu_fusable`` holds."""
    M, K = x.shape
    I = w_gate_val.shape[1] // 2
    _same_inner("gemm_skinny_swiglu", K, w_gate_val.shape[0])
    assert gemm_skinny_swiglu_fusable(x, w_gate_val)
    act = torch.empty((M, I), dtype=torch.bfloat16, device=x.device)
    native.status_tensor()
    native.check(native.lib().b200_gemm_skinny_swiglu(
        native.ptr(x), native.ptr(w_gate_val), native.ptr(act), M, I, K, x.stride(0), w_gate_val.stride(0), I,
        native.stream_ptr()), "b200_gemm_skinny_swiglu")
    native.bump()
    return act


def gemm_swiglu_bwd_fusable(dout: torch.Tensor, w_out: torch.Tensor, gv: torch.Tensor) -> bool:
    """True when ``gemm_swiglu_bwd`` runs as one kernel (``dout`` [M, H], ``w_out`` [I, H], ``gv`` [M, 2 I], bf16; I of
    ``gv`` may be the width of ``w_out`` rounded up to a multiple of 8)."""
    if not (dout.is_cuda and GEMM_IMPL == "2cta" and _tma_ok(dout, w_out, gv)):
        return False
    I = (w_out.shape[0] + 7) // 8 * 8
    return dout.shape[0] >= 256 and I >= 256 and I % 8 == 0 and gv.shape == (dout.shape[0], 2 * I)


def gemm_swiglu_bwd(dout: torch.Tensor, w_out: torch.Tensor, gv: torch.Tensor) -> torch.Tensor:
    """``d[gate | value]`` [M, 2 I] from ``dout`` [M, H], the down projection ``w_out`` [I, H] and the forward's
    projection ``gv``: the gradient of the activation, ``dout @ w_out^T``, exists only in tensor memory; the GEMM's
    epilogue reads the gate / value tiles and writes the two gradients. Only where ``gemm_swiglu_bwd_fusable``."""
    M, K = dout.shape
    I = gv.shape[1] // 2
    _same_inner("gemm_swiglu_bwd", K, w_out.shape[1])
    assert gemm_swiglu_bwd_fusable(dout, w_out, gv)
    dgv = torch.empty_like(gv)
    native.status_tensor()
    _apply_dynamic()
    rc = native.lib().b200_gemm_bf16_2cta_swiglu_bwd(
        native.ptr(dout), native.ptr(w_out), native.ptr(gv), native.ptr(dgv), M, I, K, dout.stride(0), w_out.stride(0),
        gv.stride(0), dgv.stride(0), w_out.shape[0], native.stream_ptr())
    native.check(rc, "b200_gemm_bf16_2cta_swiglu_bwd")
    native.bump()
    return dgv


def gemm_delta_fusable(dout: torch.Tensor, w_o: torch.Tensor, o: torch.Tensor, T: int, head_dim: int) -> bool:
    """True when ``gemm_delta`` runs as one kernel (``dout`` [M, H], ``w_o`` [heads * head_dim, H], ``o`` [M, heads *
    head_dim], bf16; M = batch * T)."""
    if not (dout.is_cuda and GEMM_IMPL == "2cta" and _tma_ok(dout, w_o, o)):
        return False
    N = w_o.shape[0]
    return (head_dim in (64, 128) and N % head_dim == 0 and dout.shape[0] >= 256 and N >= 256 and T > 0
            and dout.shape[0] % T == 0 and o.shape == (dout.shape[0], N))


def gemm_delta(dout: torch.Tensor, w_o: torch.Tensor, o: torch.Tensor, T: int, head_dim: int):
    """Gradient of the attention output and the row sums the attention backward needs, from ONE GEMM:
    ``do = dout @ w_o^T`` [M, heads * head_dim] and ``delta[b, head, t] = sum_d do * o`` (fp32, [batch, heads, T]); the
    epilogue reads the forward's output ``o`` tile by tile. Only where ``gemm_delta_fusable`` holds."""
    M, K = dout.shape
    N = w_o.shape[0]
    _same_inner("gemm_delta", K, w_o.shape[1])
    assert gemm_delta_fusable(dout, w_o, o, T, head_dim)
    do = torch.empty((M, N), dtype=torch.bfloat16, device=dout.device)
    delta = torch.empty((M // T, N // head_dim, T), dtype=torch.float32, device=dout.device)
    native.status_tensor()
    _apply_dynamic()
    rc = native.lib().b200_gemm_bf16_2cta_delta(
        native.ptr(dout), native.ptr(w_o), native.ptr(do), native.ptr(o), native.ptr(delta), M, N, K, dout.stride(0),
        w_o.stride(0), N, o.stride(0), T, head_dim, _whole_tiles_flag(dout.device), native.stream_ptr())
    native.check(rc, "b200_gemm_bf16_2cta_delta")
    native.bump()
    return do, delta


def gemm_ce_fusable(x: torch.Tensor, w: torch.Tensor) -> bool:
    """True when the LM-head GEMMs with the loss epilogues run for ``x`` [M, K] and ``w`` [V, K] (bf16)."""
    return bool(x.is_cuda and GEMM_IMPL == "2cta" and _tma_ok(x, w) and x.shape[0] >= 256 and w.shape[0] >= 256)


def gemm_ce_stats(x: torch.Tensor, w: torch.Tensor, targets: torch.Tensor, tlogit: torch.Tensor, col0: int = 0,
                  vocab: int = 0, logits: torch.Tensor | None = None):
    """Logits ``x @ w^T`` that need not be stored: returns per-tile row statistics ``(pmax, psum)``, each
    ``[ceil(V / 256), M]`` fp32 (maximum and sum of exp(logit - maximum) over the tile's columns), and writes the
    target's logit of every row whose target lies in ``[col0, col0 + V)`` into ``tlogit`` [M] fp32. ``vocab``
    (size of the whole vocabulary, 0: unknown) lets the bounds-checking build report targets beyond it. ``logits``
    ([M, keep] fp32 rows on 16-byte boundaries, ``keep`` a multiple of 32 or V) receives the leading columns."""
    M, K = x.shape
    V = w.shape[0]
    keep = 0 if logits is None else logits.shape[1]
    if logits is not None:
        assert (logits.shape[0] == M and logits.dtype == torch.float32 and logits.is_cuda and 0 < keep <= V
                and (keep % 32 == 0 or keep == V) and logits.stride(1) == 1 and logits.stride(0) % 4 == 0
                and logits.stride(0) >= keep and logits.data_ptr() % 16 == 0)
    _same_inner("gemm_ce_stats", K, w.shape[1])
    assert gemm_ce_fusable(x, w) and targets.dtype == torch.int32 and targets.numel() == M
    nt = (V + 255) // 256
    pmax = torch.empty((nt, M), dtype=torch.float32, device=x.device)
    psum = torch.empty((nt, M), dtype=torch.float32, device=x.device)
    native.status_tensor()
    _apply_dynamic()
    rc = native.lib().b200_gemm_bf16_2cta_ce_stats(
        native.ptr(x), native.ptr(w), M, V, K, x.stride(0), w.stride(0), native.ptr(targets), native.ptr(pmax),
        native.ptr(psum), native.ptr(tlogit), col0, 0, int(vocab), native.ptr(logits),
        0 if logits is None else logits.stride(0), keep, native.stream_ptr())
    native.check(rc, "b200_gemm_bf16_2cta_ce_stats")
    native.bump()
    return pmax, psum


def gemm_ce_dlogits(x: torch.Tensor, w: torch.Tensor, targets: torch.Tensor, lse: torch.Tensor, coef: torch.Tensor,
                    col0: int = 0) -> torch.Tensor:
    """``(exp(x @ w^T - lse[row]) - onehot(target)) * coef[row]`` as bf16 [M, V_chunk]: the gradient of the loss
    w.r.t. the logits of vocabulary rows ``col0 .. col0 + V_chunk``, formed in the GEMM epilogue."""
    M, K = x.shape
    C = w.shape[0]
    _same_inner("gemm_ce_dlogits", K, w.shape[1])
    assert gemm_ce_fusable(x, w) and C % 8 == 0
    out = torch.empty((M, C), dtype=torch.bfloat16, device=x.device)
    native.status_tensor()
    _apply_dynamic()
    rc = native.lib().b200_gemm_bf16_2cta_ce_dlogits(
        native.ptr(x), native.ptr(w), native.ptr(out), M, C, K, x.stride(0), w.stride(0), C, native.ptr(targets),
        native.ptr(lse), native.ptr(coef), col0, native.stream_ptr())
    native.check(rc, "b200_gemm_bf16_2cta_ce_dlogits")
    native.bump()
    return out


def gemm_allgather(a: torch.Tensor, unit_buf: torch.Tensor, b_offset: int, b_shape: tuple, *, trans_b: bool,
                   peer_slices, seg: torch.Tensor, epoch: int, n_copy: int = 8, add: torch.Tensor | None = None,
                   out: torch.Tensor | None = None, trans_a: bool = False, only_b: bool = False) -> torch.Tensor:
    """``out = op(a) @ op(B) (+ add)`` where B is the weight ``b_shape`` stored at element offset
    ``b_offset`` of the local ZeRO unit buffer ``unit_buf`` — and the unit buffer is being filled
    by this same kernel: ``n_copy`` CTAs pull every rank's slice (``peer_slices`` = W device
    pointers, one per rank, same length) over NVLink while the remaining CTAs run the GEMM, each
    waiting only for the rows of B it is about to load. When the kernel finishes the whole unit
    buffer is valid. ``seg`` = this buffer's progress counters (int64 zeros, one per MiB),
    ``epoch`` = 1, 2, ... per use of the buffer. With ``only_b`` the kernel copies just the 32 KiB
    chunks that hold B (``ag_region`` gives their byte range; the caller gathers the rest of the
    unit with ``FusedCollectives.all_gather(..., skip=range)``); ``seg`` must then be zeroed and
    ``epoch`` be 1 for every call, because the range differs from use to use."""
    W = len(peer_slices)
    M, K = (a.shape[1], a.shape[0]) if trans_a else (a.shape[0], a.shape[1])
    if trans_b:
        N, Kb = b_shape
    else:
        Kb, N = b_shape
    if K != Kb:
        raise ValueError(f"gemm_allgather: inner dims differ ({K} vs {Kb})")
    assert a.is_cuda and a.dtype == torch.bfloat16 and unit_buf.dtype == torch.bfloat16
    assert unit_buf.numel() % W == 0
    a, lda = _rowmajor_2d(a)
    if out is None:
        out = torch.empty((M, N), dtype=torch.bfloat16, device=a.device)
    flags, ldc = 0, 0
    if add is not None:
        assert add.shape == (M, N) and add.stride(1) == 1 and add.dtype == out.dtype
        ldc = add.stride(0)
        flags |= GEMM_ADD_C
    native.status_tensor()
    src = (ctypes.c_void_p * W)(*[ctypes.c_void_p(int(p)) for p in peer_slices])
    rc = native.lib().b200_gemm_bf16_allgather(
        native.ptr(a), native.ptr(out), native.ptr(add), M, N, K, lda, out.stride(0), ldc, int(trans_a),
        int(not trans_b), flags, ctypes.c_float(1.0), src, native.ptr(unit_buf), native.ptr(seg),
        ctypes.c_ulonglong(unit_buf.numel() // W * 2), ctypes.c_ulonglong(b_offset * 2), W, n_copy,
        ctypes.c_uint(epoch), int(only_b), native.stream_ptr())
    native.check(rc, "b200_gemm_bf16_allgather")
    native.bump()
    return out


def ag_region(slice_bytes: int, world: int, b_offset_bytes: int, b_bytes: int) -> tuple[int, int]:
    """Byte range of the unit buffer that ``gemm_allgather(..., only_b=True)`` fills itself."""
    out = (ctypes.c_ulonglong * 3)()
    native.check(native.lib().b200_ag_region(ctypes.c_ulonglong(slice_bytes), world, ctypes.c_ulonglong(b_offset_bytes),
                                             ctypes.c_ulonglong(b_bytes), out), "ag_region")
    return int(out[0]), int(out[1])


# ---------------------------------------------------------------------------------------------
# Weight-gradient GEMMs on a second stream. Every GEMM here is a persistent kernel that fills the
# GPU, so two of them never run side by side; but on one stream the next kernel cannot start until
# the LAST tile of the previous one has finished, and several training shapes end with a
# part-filled wave (e.g. 2048 x 3072 x 8192 is 1.3 waves of CTA pairs). The weight-gradient GEMMs
# do not feed the activation-gradient chain, so issuing them on a side stream lets their first
# CTAs start on SMs the other kernel has already left.
WGRAD_OVERLAP = True
_wgrad_streams: dict = {}
_wgrad_pending: dict = {}     # device index -> a side-stream GEMM has been issued and not joined yet


def _wgrad_stream(device):
    key = device.index if device.index is not None else torch.cuda.current_device()
    st = _wgrad_streams.get(key)
    if st is None:
        st = _wgrad_streams[key] = torch.cuda.Stream(device=device)
    return st


def wgrad_gemm(a: torch.Tensor, b: torch.Tensor, out: torch.Tensor | None = None, last: bool = False) -> torch.Tensor:
    """``a^T @ b`` for a weight gradient; runs on the side stream when overlap is enabled. The
    caller must call ``wgrad_join()`` before the result is consumed on the main stream. ``last``: little follows on the
    main stream before that join."""
    if not (WGRAD_OVERLAP and a.is_cuda):
        return gemm(a, b, trans_a=True, out=out)
    return _on_wgrad_stream(lambda: gemm(a, b, trans_a=True, out=out, side=last), a, b)


# Operands of side-stream GEMMs stay referenced until the stream that issued them waits for the side stream: from then on
# their memory may be used again in that stream's order. ``record_stream`` gives a block back only when the host has seen
# its event complete, so a host that runs ahead takes new device memory on every pass (125M, 8 x 1024 tokens: 12.0 GB
# reserved in place of 3.2, and cudaMalloc calls of milliseconds between the launches). It remains for a stream that issues
# more than WGRAD_HELD of them without joining (a model's block issues four).
WGRAD_HELD = 8
_wgrad_held: dict = {}        # (device index, raw stream) -> deque of operand pairs
_wgrad_lock = threading.Lock()


def _on_wgrad_stream(compute, a: torch.Tensor, b: torch.Tensor) -> torch.Tensor:
    """``compute()``, which reads ``a`` and ``b``, on the side stream behind everything issued on the current one."""
    ws = _wgrad_stream(a.device)
    index = a.device.index
    _wgrad_pending[index] = True
    issuer = torch._C._cuda_getCurrentRawStream(index)
    try:
        if index == torch._C._cuda_getDevice():
            # what ``ws.wait_stream`` and ``with torch.cuda.stream(ws)`` do, without their device checks and stream
            # objects (about 25 us of host time per weight gradient)
            prev = torch._C._cuda_getCurrentStream(index)
            ev = torch.cuda.Event()
            ev.record(torch.cuda.Stream(stream_id=prev[0], device_index=prev[1], device_type=prev[2]))
            ws.wait_event(ev)
            torch._C._cuda_setStream(stream_id=ws.stream_id, device_index=ws.device_index, device_type=ws.device_type)
            try:
                return compute()
            finally:
                torch._C._cuda_setStream(stream_id=prev[0], device_index=prev[1], device_type=prev[2])
        ws.wait_stream(torch.cuda.current_stream(a.device))
        with torch.cuda.stream(ws):
            return compute()
    finally:
        # after the launch, so that whoever takes the pair out waits behind it
        with _wgrad_lock:
            held = _wgrad_held.setdefault((index, issuer), collections.deque())
            held.append((a, b))
            if len(held) > WGRAD_HELD:
                for t in held.popleft():
                    t.record_stream(ws)


def pad_gate_value(w: torch.Tensor, I: int) -> torch.Tensor:
    """``[gate | value]`` [R, 2 I] with both halves padded by zero columns to a multiple of 8: [R, 2 Ip]."""
    Ip = (I + 7) // 8 * 8
    out = torch.empty((w.shape[0], 2 * Ip), dtype=w.dtype, device=w.device)
    return repitch(w, out, I, Ip, 2, I, Ip)


def wgrad_gemm_gate_value(x: torch.Tensor, dgv: torch.Tensor, I: int, out: torch.Tensor | None = None) -> torch.Tensor:
    """``x^T @ dgv`` without the padding columns of ``dgv`` [M, 2 Ip] (see ``pad_gate_value``): [K, 2 I], on the
    weight-gradient stream like ``wgrad_gemm``. ``out`` may be bf16 or fp32, as there."""
    if out is not None:
        assert out.shape == (x.shape[1], 2 * I) and out.stride(1) == 1
        if out.dtype not in (torch.bfloat16, torch.float32):
            raise TypeError("wgrad_gemm_gate_value: out dtype must be bf16 or fp32")

    def compute():
        dst = torch.empty((x.shape[1], 2 * I), dtype=x.dtype, device=x.device) if out is None else out
        full = gemm(x, dgv, trans_a=True, out_dtype=dst.dtype, side=False if WGRAD_OVERLAP else None)
        w = dst.element_size() // 2                        # fp32 moves as pairs of 2-byte words
        repitch(*(t.view(torch.bfloat16) for t in (full, dst)), I * w, I * w, 2, dgv.shape[1] // 2 * w, I * w)
        return dst

    return _on_wgrad_stream(compute, x, dgv) if WGRAD_OVERLAP else compute()


def wgrad_event(device):
    """An event after everything issued so far on the weight-gradient side stream of ``device`` (None when
    that stream has never been used): what a consumer on a third stream waits for instead of joining."""
    dev = torch.device(device)
    if not WGRAD_OVERLAP or dev.type != "cuda":
        return None
    key = dev.index if dev.index is not None else torch.cuda.current_device()
    ws = _wgrad_streams.get(key)
    if ws is None:
        return None
    ev = torch.cuda.Event()
    ev.record(ws)
    return ev


def wgrad_join(device=None) -> None:
    if not WGRAD_OVERLAP or not torch.cuda.is_available():
        return
    dev = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    if dev.type != "cuda":
        return
    key = dev.index if dev.index is not None else torch.cuda.current_device()
    ws = _wgrad_streams.get(key)
    if ws is not None:
        cur = torch.cuda.current_stream(dev)
        with _wgrad_lock:
            held = _wgrad_held.pop((key, cur.cuda_stream), None)
        cur.wait_stream(ws)
        del held                          # not before the wait
    _wgrad_pending[key] = False
