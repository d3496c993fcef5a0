// Epilogue shared by the tcgen05 attention-backward kernels (head_dim 128 or 64): store one fp32 accumulator
// row from tensor memory as bf16, applying the inverse rotary embedding on the way.
//
// The kernels work on rotated Q and K, so their dQ and dK are gradients of the rotated tensors. The
// gradient of the un-rotated one is the inverse rotation of the same row (pairs (j, j + D/2), angle of
// the row's position): y1 = x1 c + x2 s, y2 = x2 c - x1 s. Doing it here, on the fp32 accumulator a
// thread already holds, removes the separate in-place pass over the [dK | dQ] columns.
#pragma once
#include "common.cuh"
#include "ptx.cuh"

namespace b200 {

// Pairs j in [j0, j0 + nj) (nj a multiple of 16) of the row at TMEM address `taddr` (column 0 of the
// kD-wide accumulator). The tables are fp32 and TRANSPOSED, [kD / 2][ld]: cs_row / sn_row point at this row's
// position in line 0 and element j is at [j * ld], so the lanes of a warp (consecutive positions) read
// consecutive words. The TMEM loads are warp-collective: every lane calls this, `active` only predicates
// the global stores.
template <int kD>
__device__ __forceinline__ void store_row_unrot_from_tmem(uint32_t taddr, bf16* grow, int j0, int nj,
                                                          const float* cs_row, const float* sn_row, int ld,
                                                          bool active) {
#pragma unroll 1
  constexpr int kHalf = kD / 2;
  for (int j = j0; j < j0 + nj; j += 16) {
    uint32_t a[16], b[16];
    tmem_ld_32x32b_x16(taddr + j, a);
    tmem_ld_32x32b_x16(taddr + kHalf + j, b);
    tmem_ld_wait();
    if (!active) continue;
    uint32_t y1[8], y2[8];
#pragma unroll
    for (int i = 0; i < 16; i += 4) {
      float cc[4], ss[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        cc[e] = cs_row[size_t(j + i + e) * ld];
        ss[e] = sn_row[size_t(j + i + e) * ld];
      }
      float o1[4], o2[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float x1 = __uint_as_float(a[i + e]), x2 = __uint_as_float(b[i + e]);
        o1[e] = fmaf(x1, cc[e], x2 * ss[e]);
        o2[e] = fmaf(x2, cc[e], -x1 * ss[e]);
      }
#pragma unroll
      for (int e = 0; e < 4; e += 2) {
        const bf162 t1 = __floats2bfloat162_rn(o1[e], o1[e + 1]);
        const bf162 t2 = __floats2bfloat162_rn(o2[e], o2[e + 1]);
        y1[(i + e) >> 1] = *reinterpret_cast<const uint32_t*>(&t1);
        y2[(i + e) >> 1] = *reinterpret_cast<const uint32_t*>(&t2);
      }
    }
    *reinterpret_cast<uint4*>(grow + j) = make_uint4(y1[0], y1[1], y1[2], y1[3]);
    *reinterpret_cast<uint4*>(grow + j + 8) = make_uint4(y1[4], y1[5], y1[6], y1[7]);
    *reinterpret_cast<uint4*>(grow + kHalf + j) = make_uint4(y2[0], y2[1], y2[2], y2[3]);
    *reinterpret_cast<uint4*>(grow + kHalf + j + 8) = make_uint4(y2[4], y2[5], y2[6], y2[7]);
  }
}

// The same rows, through shared memory: a warp gathers 128 bytes of each of its 32 rows in `buf` (4 KiB of its own, 16-byte
// chunks swizzled by the row) and writes them out eight lanes to a row. A store instruction whose lanes are in 32 rows takes 32
// turns in the load-store unit; with two of these per pass the dK/dV kernel's epilogue took 4600 clocks at head_dim 64 and
// 8300 at 128, and the first shared-memory reads of the next pass queued behind it for up to 10000 more.
__device__ __forceinline__ void row_chunk_put(uint8_t* buf, int lane, int chunk, const uint32_t* v) {
  *reinterpret_cast<uint4*>(buf + lane * 128 + ((chunk ^ (lane & 7)) << 4)) = make_uint4(v[0], v[1], v[2], v[3]);
}

// Rows [0, live) of `buf` to `base` + row * ts: their first 64 bytes to column c0, the others to column c1.
__device__ __forceinline__ void flush_rows(const uint8_t* buf, int lane, bf16* base, long long ts, int c0, int c1, int live) {
  __syncwarp();
  const int c = lane & 7, col = c < 4 ? c0 + c * 8 : c1 + (c - 4) * 8;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = i * 4 + (lane >> 3);
    const uint4 v = *reinterpret_cast<const uint4*>(buf + r * 128 + ((c ^ (r & 7)) << 4));
    if (r < live) *reinterpret_cast<uint4*>(base + r * ts + col) = v;
  }
  __syncwarp();
}

// 64 columns from `col` of the accumulator at `taddr`, as they are. (Rolled loops here and below: the code is fetched once per
// pass, cold.)
__device__ __forceinline__ void store_rows_plain(uint32_t taddr, int col, uint8_t* buf, int lane, bf16* base, long long ts,
                                                 int live) {
#pragma unroll 1
  for (int hh = 0; hh < 2; ++hh) {
    uint32_t r[32], y[16];
    tmem_ld_32x32b_x32(taddr + col + 32 * hh, r);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      const bf162 t = __floats2bfloat162_rn(__uint_as_float(r[i]), __uint_as_float(r[i + 1]));
      y[i >> 1] = *reinterpret_cast<const uint32_t*>(&t);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) row_chunk_put(buf, lane, 4 * hh + k, &y[4 * k]);
  }
  flush_rows(buf, lane, base, ts, col, col + 32, live);
}

// cos and sin of pairs [j0, j0 + 16) at this row's position; tables as above.
struct RowTables {
  float c[16], s[16];
};
__device__ __forceinline__ void load_row_tables(RowTables& t, const float* cs_row, const float* sn_row, int ld, int j0) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    t.c[i] = cs_row[size_t(j0 + i) * ld];
    t.s[i] = sn_row[size_t(j0 + i) * ld];
  }
}

// Pairs [j0, j0 + 16) of the kD-wide accumulator at `taddr`, rotated back, into `buf`: chunks k0, k0 + 1 take their first
// elements, k0 + 4, k0 + 5 their second ones.
template <int kD>
__device__ __forceinline__ void put_rows_unrot(uint32_t taddr, int j0, const RowTables& t, uint8_t* buf, int lane, int k0) {
  uint32_t a[16], b[16], y1[8], y2[8];
  tmem_ld_32x32b_x16(taddr + j0, a);
  tmem_ld_32x32b_x16(taddr + kD / 2 + j0, b);
  tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    float o1[2], o2[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float x1 = __uint_as_float(a[i + e]), x2 = __uint_as_float(b[i + e]);
      o1[e] = fmaf(x1, t.c[i + e], x2 * t.s[i + e]);
      o2[e] = fmaf(x2, t.c[i + e], -x1 * t.s[i + e]);
    }
    const bf162 t1 = __floats2bfloat162_rn(o1[0], o1[1]);
    const bf162 t2 = __floats2bfloat162_rn(o2[0], o2[1]);
    y1[i >> 1] = *reinterpret_cast<const uint32_t*>(&t1);
    y2[i >> 1] = *reinterpret_cast<const uint32_t*>(&t2);
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    row_chunk_put(buf, lane, k0 + k, &y1[4 * k]);
    row_chunk_put(buf, lane, k0 + 4 + k, &y2[4 * k]);
  }
}

// Pairs [j0, j0 + 32), from the tables to the rows at `base`.
template <int kD>
__device__ __forceinline__ void store_rows_unrot(uint32_t taddr, int j0, const float* cs_row, const float* sn_row, int ld,
                                                 uint8_t* buf, int lane, bf16* base, long long ts, int live) {
#pragma unroll 1
  for (int hh = 0; hh < 2; ++hh) {
    RowTables t;
    load_row_tables(t, cs_row, sn_row, ld, j0 + 16 * hh);
    put_rows_unrot<kD>(taddr, j0 + 16 * hh, t, buf, lane, 2 * hh);
  }
  flush_rows(buf, lane, base, ts, j0, kD / 2 + j0, live);
}

}  // namespace b200
