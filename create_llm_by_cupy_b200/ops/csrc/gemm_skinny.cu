// D[M, N] = alpha * A B (+ C) for few rows (M <= 64): the projections of a decoded token and of short prompts.
//
// What bounds it: the weight matrix B is read once and nothing is computed for long, so the time is how fast the
// whole GPU can stream it. A 128-row tensor-core tile per 128 columns leaves most SMs without a tile (N = 768:
// 6 CTAs that walk all of K one after the other). Here
//   * a CTA owns 64 columns and a slice of K; the CTAs that share a column tile form a cluster along K and add
//     their fp32 sums through distributed shared memory, so a 768 x 768 weight is 48 CTAs and there is no
//     workspace and no second launch;
//   * 64 x 64 weight tiles (8 KiB) arrive through a ring of cp.async stages, several CTAs per SM, so that tens of
//     KiB per SM are in flight; with SwiGLU 32 k x (64 gate + 64 value columns), so that a row is read 128 bytes at a time
//     there too (64 k x (32 + 32): 4096 x 22016, eight rows, 38.0 us where this takes 35.5; 2048 x 11008, 16 rows, 16.1 / 14.4);
//   * the product runs as W^T x^T on mma.sync (16 weight columns x 8 tokens x 16 k, fp32 accumulation): one token
//     costs the same instructions as eight, and both weight layouts feed the same fragments through ldmatrix.
// One row, weights not in L2 (before: 128-row tiles): 768 x 768 6.8 -> 3.6 us, 2048 x 3072 13.3 -> 5.6, 2048 x 11008
// 19.2 -> 10.9 (4.1 TB/s), 11008 x 4096 52 -> 17 (5.2 TB/s), 4096 x 22016 44 -> 34 (5.3 TB/s).
#include <cooperative_groups.h>

#include "common.cuh"

namespace b200 {
namespace cg = cooperative_groups;

constexpr int SK_TN = 64;                  // weight columns per CTA
constexpr int SK_TK = 64;                  // k per stage
constexpr int SK_W_BYTES = SK_TN * SK_TK * 2;
constexpr int SK_THREADS = 128;            // warp w owns columns 16 w .. 16 w + 15

struct SkinnyParams {
  const bf16* A;      // [M, K], pitch lda
  const bf16* B;      // [K, N] (K_ROWS) or [N, K], pitch ldb
  const void* C;
  void* D;
  int M, N, K, lda, ldb, ldd, ldc;
  int out_f32, kslice;                     // kslice: k range of one CTA, a multiple of SK_TK
  int I;                                   // GLU: B = [gate | value], N = 2 I, D [M, I] = silu(gate) * value
  float alpha;
};

template <int MT, bool GLU>
struct SkinnySmem {
  static constexpr int kTk = GLU ? 32 : SK_TK;                     // k per stage
  static constexpr int kCols = GLU ? 2 * SK_TN : SK_TN;            // weight columns of a CTA
  static constexpr int kStages = MT <= 2 ? 6 : (MT == 4 ? 5 : 4);
  static constexpr int kABytes = MT * 8 * SK_TK * 2;
  static constexpr int kStageBytes = SK_W_BYTES + kABytes;
  static constexpr int kSum = MT * 8 * kCols * 4;                  // fp32 [rows][columns] for the cluster's sum
  static constexpr int kTotal = kStages * kStageBytes > kSum ? kStages * kStageBytes : kSum;
  static constexpr int kPerSm = 228 * 1024 / (kTotal + 1024);      // CTAs that fit an SM: 4 up to 8 rows, then 3
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// 128-byte rows of eight 16-byte chunks, chunk index XORed with the row: ldmatrix reads eight rows without conflict
__device__ __forceinline__ uint32_t sw_addr(uint32_t base, int row, int chunk) {
  return base + uint32_t(row) * 128u + uint32_t((chunk ^ (row & 7)) * 16);
}

// One stage: 8 KiB of weights (64 k x 64 columns; GLU: 32 k x 64 gate columns, then the 64 value columns of the same index: 128
// bytes of a row at a time either way) and the tokens' tile at k0. Bytes past K, N or M arrive as zeros
// (cp.async with a short source size; the address of a skipped chunk is the matrix base).
template <int MT, bool K_ROWS, bool GLU>
__device__ __forceinline__ void skinny_load(const SkinnyParams& p, uint32_t stage, int n0, int k0, int k_end) {
  const int tid = threadIdx.x;
#pragma unroll
  for (int i = 0; i < SK_W_BYTES / 16 / SK_THREADS; ++i) {
    const int idx = tid + i * SK_THREADS, row = idx >> 3, chunk = idx & 7;
    const int k = GLU ? k0 + (row & 31) : (K_ROWS ? k0 + row : k0 + chunk * 8);
    int n = K_ROWS ? n0 + chunk * 8 : n0 + row;
    int left;                                             // elements of this chunk inside the matrix
    if (GLU) {
      left = k < k_end ? p.I - n : 0;
      n += row < 32 ? 0 : p.I;
    } else if (K_ROWS) left = k < k_end ? p.N - n : 0;
    else left = n < p.N ? k_end - k : 0;
    left = left < 0 ? 0 : (left > 8 ? 8 : left);
    const bf16* src = left > 0 ? (K_ROWS ? p.B + size_t(k) * p.ldb + n : p.B + size_t(n) * p.ldb + k) : p.B;
    cp_async16(sw_addr(stage, row, chunk), src, left * 2);
  }
  const uint32_t sa = stage + SK_W_BYTES;
  constexpr int kChunks = SkinnySmem<MT, GLU>::kTk / 8;
  for (int idx = tid; idx < MT * 8 * kChunks; idx += SK_THREADS) {
    const int row = idx / kChunks, chunk = idx % kChunks, k = k0 + chunk * 8;
    int left = row < p.M ? k_end - k : 0;
    left = left < 0 ? 0 : (left > 8 ? 8 : left);
    cp_async16(sw_addr(sa, row, chunk), left > 0 ? p.A + size_t(row) * p.lda + k : p.A, left * 2);
  }
}

// grid (k slices, column tiles), cluster (k slices, 1, 1)
template <int MT, bool K_ROWS, bool GLU>
__global__ void __launch_bounds__(SK_THREADS)
gemm_skinny_kernel(const SkinnyParams p) {
  using S = SkinnySmem<MT, GLU>;
  extern __shared__ __align__(128) uint8_t smem[];
  cg::cluster_group cluster = cg::this_cluster();
  const int ks = int(gridDim.x), rank = int(blockIdx.x);
  const int n0 = int(blockIdx.y) * SK_TN;       // output columns of a CTA: 64
  const int k_begin = rank * p.kslice, k_end = min(p.K, k_begin + p.kslice);
  const int steps = k_end > k_begin ? (k_end - k_begin + S::kTk - 1) / S::kTk : 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(smem));

  constexpr int kHalves = GLU ? 2 : 1;           // gate and value columns
  float acc[kHalves][MT][4];
#pragma unroll
  for (int h = 0; h < kHalves; ++h)
#pragma unroll
    for (int t = 0; t < MT; ++t)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[h][t][e] = 0.f;

  pdl_wait();
  // No pdl_trigger(): the next kernel's CTAs then start as these end. Let in before that, they land unevenly among this one's,
  // take shared memory and issue slots from what is still running and run unevenly themselves. us with the trigger here for
  // slices of up to 12 stages and behind the loop for longer ones / without: a 7B block of 8 sequences 113.2 / 104.3, of one
  // 88.9 / 86.6, a 1.3B block of one 43.4 / 40.8, of 16 54.4 / 52.9, one token through the 125M model 349 / 337 on the device,
  // a training pass of 64 tokens 2027 / 2022.
#pragma unroll
  for (int s = 0; s < S::kStages - 1; ++s) {
    if (s < steps) skinny_load<MT, K_ROWS, GLU>(p, base + s * S::kStageBytes, n0, k_begin + s * S::kTk, k_end);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  const int mi = lane >> 3, mr = lane & 7;       // ldmatrix: matrix and row that this lane addresses
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(S::kStages - 2) : "memory");
    __syncthreads();                             // stage s has landed; everyone has left stage s - 1
    const int nx = s + S::kStages - 1;
    if (nx < steps)
      skinny_load<MT, K_ROWS, GLU>(p, base + (nx % S::kStages) * S::kStageBytes, n0, k_begin + nx * S::kTk, k_end);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const uint32_t sw = base + (s % S::kStages) * S::kStageBytes, sa = sw + SK_W_BYTES;
    uint32_t w[SK_TK / 16][4];                   // GLU: gate k 0-15, 16-31, then value
#pragma unroll
    for (int kk = 0; kk < SK_TK / 16; ++kk) {
      // A fragment of 16 weight columns x 16 k: matrices (columns 0-7, k 0-7), (8-15, 0-7), (0-7, 8-15), (8-15, 8-15)
      if (K_ROWS) ldsm4t(w[kk], sw_addr(sw, kk * 16 + (mi >> 1) * 8 + mr, warp * 2 + (mi & 1)));
      else ldsm4(w[kk], sw_addr(sw, warp * 16 + (mi & 1) * 8 + mr, kk * 2 + (mi >> 1)));
    }
#pragma unroll
    for (int t = 0; t < MT; ++t) {
      uint32_t x0[4], x1[4];                     // tokens 8 t .. 8 t + 7, k 0-31 and 32-63
      constexpr bool kAhead = MT == 8;           // both before the products (64 x 768 over 768 6.7 us, 7.0 one after the other;
      ldsm4(x0, sw_addr(sa, t * 8 + mr, mi));    // five rows 3.6, 3.5)
      if (!GLU && kAhead) ldsm4(x1, sw_addr(sa, t * 8 + mr, 4 + mi));
      mma16816(acc[0][t], w[0], x0[0], x0[1]);
      mma16816(acc[0][t], w[1], x0[2], x0[3]);
      if (GLU) {
        mma16816(acc[kHalves - 1][t], w[2], x0[0], x0[1]);
        mma16816(acc[kHalves - 1][t], w[3], x0[2], x0[3]);
      } else {
        if (!kAhead) ldsm4(x1, sw_addr(sa, t * 8 + mr, 4 + mi));
        mma16816(acc[0][t], w[2], x1[0], x1[1]);
        mma16816(acc[0][t], w[3], x1[2], x1[3]);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();

  // fp32 partial sums as [token][columns]; the CTAs of the cluster each finish a share of the outputs
  float* sum = reinterpret_cast<float*>(smem);
#pragma unroll
  for (int h = 0; h < kHalves; ++h)
#pragma unroll
    for (int t = 0; t < MT; ++t)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        sum[(t * 8 + (lane & 3) * 2 + (e & 1)) * S::kCols + h * SK_TN + warp * 16 + (lane >> 2) + (e >> 1) * 8] = acc[h][t][e];
  cluster.sync();
  const int rows = min(p.M, MT * 8);
  for (int i = rank * SK_THREADS + int(threadIdx.x); i < rows * SK_TN; i += ks * SK_THREADS) {
    const int row = i / SK_TN, col = n0 + i % SK_TN, at = row * S::kCols + i % SK_TN;
    if (col >= (GLU ? p.I : p.N)) continue;
    float v = 0.f;
    for (int c = 0; c < ks; ++c) v += cluster.map_shared_rank(sum, c)[at];
    if constexpr (GLU) {
      float u = 0.f;
      for (int c = 0; c < ks; ++c) u += cluster.map_shared_rank(sum, c)[at + SK_TN];
      static_cast<bf16*>(p.D)[size_t(row) * p.ldd + col] = __float2bfloat16(v / (1.f + __expf(-v)) * u);
      continue;
    }
    v *= p.alpha;
    if (p.out_f32) {
      if (p.C) v += static_cast<const float*>(p.C)[size_t(row) * p.ldc + col];
      static_cast<float*>(p.D)[size_t(row) * p.ldd + col] = v;
    } else {
      if (p.C) v += __bfloat162float(static_cast<const bf16*>(p.C)[size_t(row) * p.ldc + col]);
      static_cast<bf16*>(p.D)[size_t(row) * p.ldd + col] = __float2bfloat16(v);
    }
  }
  cluster.sync();                                // peers read this CTA's sums until here
}

template <int MT, bool K_ROWS, bool GLU>
static int launch_skinny(SkinnyParams p, cudaStream_t st) {
  using S = SkinnySmem<MT, GLU>;
  auto kern = gemm_skinny_kernel<MT, K_ROWS, GLU>;
  if (S::kTotal > 48 * 1024) B200_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kTotal));
  const int tiles = ((GLU ? p.I : p.N) + SK_TN - 1) / SK_TN, ksteps = (p.K + S::kTk - 1) / S::kTk;
  if (tiles > 65535) return static_cast<int>(cudaErrorInvalidValue);
  // k slices: as many as fill the GPU's resident CTAs once, at most 8 (a portable cluster) and at least 2 stages each
  int ks = 1;
  while (ks < 8 && long(tiles) * ks * 2 <= long(S::kPerSm) * num_sms() && ksteps >= 4 * ks) ks *= 2;
  p.kslice = (ksteps + ks - 1) / ks * S::kTk;
  return static_cast<int>(launch_pdl(kern, dim3(ks, tiles), dim3(SK_THREADS), S::kTotal, st, ks, p));
}

template <bool K_ROWS, bool GLU>
static int launch_skinny_rows(const SkinnyParams& p, cudaStream_t st) {
  if (p.M <= 8) return launch_skinny<1, K_ROWS, GLU>(p, st);
  if (p.M <= 16) return launch_skinny<2, K_ROWS, GLU>(p, st);
  if (p.M <= 32) return launch_skinny<4, K_ROWS, GLU>(p, st);
  return launch_skinny<8, K_ROWS, GLU>(p, st);
}

}  // namespace b200

using namespace b200;

// Same contract as b200_gemm_bf16 for a row-major A [M, K] with M <= 64, 16-byte aligned A and B bases and pitches
// that are multiples of 8. b_k_rows = 1: B is [K, N]; 0: B is [N, K]. C may alias D (each element is read by the
// thread that writes it). out_f32: D and C are fp32, else bf16.
B200_API int b200_gemm_skinny(const void* A, const void* B, void* D, const void* C, int M, int N, int K, int lda, int ldb,
                              int ldd, int ldc, int b_k_rows, int out_f32, float alpha, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || M > 64 || ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & 15) != 0 ||
      (lda % 8) != 0 || (ldb % 8) != 0)
    return static_cast<int>(cudaErrorInvalidValue);
  SkinnyParams p = {static_cast<const bf16*>(A), static_cast<const bf16*>(B), C, D, M, N, K, lda, ldb, ldd, ldc,
                    out_f32, 0, 0, alpha};
  return b_k_rows ? launch_skinny_rows<true, false>(p, stream) : launch_skinny_rows<false, false>(p, stream);
}

// ACT[M, I] = silu(A W_gate) * (A W_value) for B = [W_gate | W_value] ([K, 2 I] row-major), M <= 64, I a multiple of 8:
// the activation in the epilogue of the few-rows GEMM (one launch and one round trip of the projection less per block of
// a decoded token).
B200_API int b200_gemm_skinny_swiglu(const void* A, const void* B, void* ACT, int M, int I, int K, int lda, int ldb,
                                     int ldact, cudaStream_t stream) {
  if (M <= 0 || I <= 0) return 0;
  if (K <= 0 || M > 64 || (I % 8) != 0 || ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & 15) != 0 ||
      (lda % 8) != 0 || (ldb % 8) != 0)
    return static_cast<int>(cudaErrorInvalidValue);
  SkinnyParams p = {static_cast<const bf16*>(A), static_cast<const bf16*>(B), nullptr, ACT, M, 2 * I, K, lda, ldb, ldact,
                    0, 0, 0, I, 1.f};
  return launch_skinny_rows<true, true>(p, stream);
}
