// One-token attention against a KV cache (causal GQA decode).
//
// What bounds it: the K and V rows of the valid prefix are read once; at small batch the time is latency - how
// many loads are in flight - not bandwidth. So:
//   * one cluster of CTAs per (sequence, KV head), every CTA and every warp of it taking its own 32-key tiles
//     (a prefix of n keys is n / 32 independent chains instead of four);
//   * all query heads of the group share each K / V row that was loaded (up to 4 heads per CTA). A tile is one run of bytes
//     in the cache: a warp asks for K and V of its first tile with two bulk copies as soon as its inputs are ready and for the
//     next one when it has read them (through registers a tile was four round trips one after the other);
//   * the scores of a tile are mma.sync products (rows = heads, columns = keys, fp32 sums): a lane's 16-byte pieces of
//     q and of the keys are fragments as they stand, because a dot product does not care in which order the head
//     dimension is walked as long as both sides walk it alike. No exchange between lanes is left before the softmax
//     (summing a key's product over lanes cost 5 shuffles in a chain per pair of keys). The weights stay fp32 and
//     multiply V on the FMA units;
//   * the partial softmax states (maximum, sum, weighted values) meet in shared memory, first over the warps of
//     a CTA, then over the CTAs of the cluster through distributed shared memory: no workspace, no second launch.
// Device time inside a block, us, tiles through registers -> shared memory: B = 8, 32 / 8 heads of 128, 3001 keys (98 MB of
// cache, 15 us at the copy rate) 35.0 -> 26.2, B = 16, 4001 keys 73.9 -> 51.9, B = 2, 65 keys 21.7 -> 11.4; B = 1, 16 / 4 heads
// of 128, 1801 keys 11.7 -> 10.0, B = 16, 1001 keys 17.8 -> 16.3; 12 / 4 heads of 64 6.8 to 8.5 before and after.
#include <cooperative_groups.h>

#include <atomic>

#include "common.cuh"
#include "ptx.cuh"
#include "tile_rows.h"

namespace b200 {
namespace cg = cooperative_groups;

constexpr int DA_MAX_WARPS = 16;
constexpr int DA_TILE = 32;          // keys per warp and step
constexpr int DA_PREFETCH = 4;       // tiles per warp that are on their way to L2 before the kernel's inputs are ready

struct DecodeParams {
  const bf16* q;        // [B, QH, D]
  const bf16* kc;       // [B, KVH, Tmax, D]
  const bf16* vc;
  bf16* out;            // [B, QH, D]
  const int* lens;      // [B]
  int QH, KVH, Tmax, groups;    // groups: CTA groups per KV head (RT query heads each)
  float scale;
  // APPEND: q, k, v come from the packed projection row [K | Q | V] of the new token, k and q un-rotated; its k
  // (rotated) and v are also written to position `pos` of the caches
  const bf16* kqv;
  bf16* kcw;
  bf16* vcw;
  const float* cosr;            // rotary table rows of `pos`, [D / 2]
  const float* sinr;
  int ld, pos;
  int* status;
};

__device__ __forceinline__ void unpack16B(const uint4& u, float (&f)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}

__device__ __forceinline__ void mma_scores(float (&d)[4], uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(0u), "r"(a2), "r"(0u), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint4 pack16B(const float (&f)[8]) {
  uint4 u;
  uint32_t* w = reinterpret_cast<uint32_t*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const bf162 h = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    w[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return u;
}

// 8-element chunk `dl` of a head at `x`, rotated (half-split pairs, partner chunk D / 16 away) and rounded to bf16
template <int D>
__device__ __forceinline__ uint4 rotated_chunk(const bf16* x, int dl, const float* cosr, const float* sinr) {
  constexpr int HC = D / 16;                              // chunks per half head
  float a[8], b[8], y[8];
  unpack16B(reinterpret_cast<const uint4*>(x)[dl], a);
  unpack16B(reinterpret_cast<const uint4*>(x)[dl ^ HC], b);
  const int j = (dl % HC) * 8;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float c = cosr[j + e], sn = sinr[j + e];
    y[e] = dl < HC ? a[e] * c - b[e] * sn : a[e] * c + b[e] * sn;
  }
  return pack16B(y);
}

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(dst)), "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

template <int RT>
struct alignas(RT * 4) HeadRow {     // one key's scores / weights, one vector load
  float v[RT];
};

// grid (cluster size, KVH * groups, B), cluster (cluster size, 1, 1), block 32 * warps (any number up to 16), dynamic shared
// memory warps * 2 tiles.
template <int D, int RT, bool APPEND>
__global__ void __maxnreg__(128)
decode_attn_kernel(const DecodeParams p) {
  constexpr int LPK = D / 8;                 // lanes per key, 16 bytes each
  constexpr int KPS = 32 / LPK;              // keys per load step
  constexpr int STEPS = DA_TILE / KPS;       // 16 / 8 / 4 for D = 128 / 64 / 32
  constexpr int TB = DA_TILE * D * 2;        // bytes of a tile of K or V
  extern __shared__ __align__(128) uint8_t tiles[];     // [warp]: a tile of K, a tile of V; then the warp's weighted values
  __shared__ uint64_t full[DA_MAX_WARPS][2];            // K, V of the warp's tile have arrived
  __shared__ int abort_flag;
  __shared__ HeadRow<RT> s_p[DA_MAX_WARPS][DA_TILE];
  __shared__ float s_m[DA_MAX_WARPS][RT], s_l[DA_MAX_WARPS][RT];
  __shared__ float c_m[RT], c_l[RT], c_o[RT][D];        // this CTA's state, read by the cluster

  cg::cluster_group cluster = cg::this_cluster();
  const int cs = int(gridDim.x), rank = int(blockIdx.x);
  const int nw = int(blockDim.x) >> 5, warp = int(threadIdx.x) >> 5, lane = int(threadIdx.x) & 31;
  const int b = blockIdx.z, kvh = int(blockIdx.y) / p.groups, g = int(blockIdx.y) % p.groups;
  const int R = p.QH / p.KVH;
  const int h0 = kvh * R + g * RT, nh = min(RT, R - g * RT);
  const int kl = lane / LPK, dl = lane % LPK;           // key slot and 8-element column of this lane
  if (APPEND && lane < 2) {
    // The first tiles of this warp travel to L2 while the projection before this kernel runs: keys up to the new token's,
    // which the host knows. The lengths may only be being written, so they are not read here; a shorter one costs a
    // useless prefetch.
    const bf16* rows = (lane == 0 ? p.kc : p.vc) + (size_t(b) * p.KVH + kvh) * size_t(p.Tmax) * D;
    for (int i = 0, t = rank + warp * cs; i < DA_PREFETCH && t * DA_TILE <= p.pos; ++i, t += nw * cs)
      l2_prefetch(rows + size_t(t) * DA_TILE * D, uint32_t(min(DA_TILE, p.pos + 1 - t * DA_TILE)) * D * 2);
  }
  if (lane < 2) mbar_init(&full[warp][lane], 1);
  if (threadIdx.x == 0) abort_flag = 0;
  mbar_fence_init();
  __syncthreads();
  pdl_wait();
  const int len = min(p.lens[b], p.Tmax);
  uint8_t* kt = tiles + size_t(warp) * 2 * TB;
  uint8_t* vt = kt + TB;
  const bf16* kb = p.kc + (size_t(b) * p.KVH + kvh) * size_t(p.Tmax) * D;
  const bf16* vb = p.vc + (size_t(b) * p.KVH + kvh) * size_t(p.Tmax) * D;
  // A tile of K (which 0) or V (1), by the first lane: its valid keys are one run of bytes, or two with the new token's row
  // between them. That row is being written by the first CTA and comes from s_new.
  auto fetch = [&](int t, int which) {
    if (t * DA_TILE >= len) return;
    const TileRows rows = tile_rows(t * DA_TILE, DA_TILE, len, APPEND ? p.pos : -1);
    uint64_t* bar = &full[warp][which];
    uint8_t* dst = which == 0 ? kt : vt;
    const bf16* src = (which == 0 ? kb : vb) + size_t(t) * DA_TILE * D;
    if (rows.first + rows.rest == 0) {                   // the new token's row alone: nothing to wait for
      mbar_arrive(bar);
      return;
    }
    mbar_expect_tx(bar, uint32_t(rows.first + rows.rest) * D * 2);
    if (rows.first > 0) bulk_load(dst, src, uint32_t(rows.first) * D * 2, bar);
    if (APPEND && rows.rest > 0)
      bulk_load(dst + (rows.first + 1) * D * 2, src + (rows.first + 1) * D, uint32_t(rows.rest) * D * 2, bar);
  };
  if (lane == 0) {
    fetch(rank + warp * cs, 0);
    fetch(rank + warp * cs, 1);
  }

  __shared__ uint4 s_new[2][LPK];                       // the new token's rotated k and v
  const bf16* new_row = nullptr;
  if constexpr (APPEND) {
    new_row = p.kqv + size_t(b) * p.ld;
    if (threadIdx.x < 2 * LPK) {
      const int which = threadIdx.x / LPK, c = threadIdx.x % LPK;
      const uint4 u = which == 0 ? rotated_chunk<D>(new_row + kvh * D, c, p.cosr, p.sinr)
                                 : reinterpret_cast<const uint4*>(new_row + (p.KVH + p.QH + kvh) * D)[c];
      s_new[which][c] = u;
      // nobody reads this cache row in this launch: every CTA takes it from its s_new, and no copy covers it
      if (rank == 0 && g == 0)
        reinterpret_cast<uint4*>((which == 0 ? p.kcw : p.vcw) + ((size_t(b) * p.KVH + kvh) * p.Tmax + p.pos) * D)[c] = u;
    }
    __syncthreads();
  }

  const int hl = lane >> 2, tl = lane & 3;              // fragment coordinates: head (or key) row, quad
  constexpr int QC = D / 32;                            // 16-byte pieces of a row per lane: chunks tl, tl + 4, ...
  uint32_t qa[QC][4];
#pragma unroll
  for (int i = 0; i < QC; ++i) {
    uint4 u = make_uint4(0u, 0u, 0u, 0u);
    if (hl < nh) {
      if constexpr (APPEND) u = rotated_chunk<D>(new_row + (p.KVH + h0 + hl) * D, tl + 4 * i, p.cosr, p.sinr);
      else u = reinterpret_cast<const uint4*>(p.q + (size_t(b) * p.QH + h0 + hl) * D)[tl + 4 * i];
    }
    qa[i][0] = u.x; qa[i][1] = u.y; qa[i][2] = u.z; qa[i][3] = u.w;
  }
  float acc[RT][8], m = -INFINITY, l = 0.f;             // m, l: of head hl
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[r][e] = 0.f;
  // 16 bytes of a key's row, from the warp's tile or, for the new token, from this launch
  auto piece = [&](const uint8_t* tile, int which, int key0, int k, int chunk) {
    const uint4* at = reinterpret_cast<const uint4*>(tile + k * D * 2) + chunk;
    if (APPEND && key0 + k == p.pos) at = &s_new[which][chunk];
    return *at;
  };

  // tile t goes to CTA t % cs, warp (t / cs) % nw: neighbouring tiles on different SMs
  uint32_t phase = 0;
  for (int t = rank + warp * cs; t * DA_TILE < len; t += nw * cs, phase ^= 1) {
    const int key0 = t * DA_TILE;
    float sc[4][4];                                     // keys 8 nb + 2 tl, + 1 of head hl in [nb][0], [nb][1]
    if (!__all_sync(0xffffffffu, mbar_wait(&full[warp][0], phase, &abort_flag))) break;
#pragma unroll
    for (int nb = 0; nb < 4; ++nb) {
#pragma unroll
      for (int e = 0; e < 4; ++e) sc[nb][e] = 0.f;
#pragma unroll
      for (int i = 0; i < QC; ++i) {
        const uint4 kf = piece(kt, 0, key0, nb * 8 + hl, tl + 4 * i);      // past the length: masked below
        mma_scores(sc[nb], qa[i][0], qa[i][1], kf.x, kf.y);
        mma_scores(sc[nb], qa[i][2], qa[i][3], kf.z, kf.w);
      }
    }
    __syncwarp();                                       // the tile of K has been read
    if (lane == 0) fetch(t + nw * cs, 0);
    float mx = -INFINITY;
#pragma unroll
    for (int nb = 0; nb < 4; ++nb)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        sc[nb][e] = key0 + nb * 8 + tl * 2 + e < len ? sc[nb][e] * p.scale : -INFINITY;
        mx = fmaxf(mx, sc[nb][e]);
      }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float mn = fmaxf(m, mx), ref = mn == -INFINITY ? 0.f : mn;
    const float corr = __expf(m - ref);                 // 0 on the first tile
    m = mn;
    l *= corr;
#pragma unroll
    for (int nb = 0; nb < 4; ++nb)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int k = nb * 8 + tl * 2 + e;
        const float pe = key0 + k < len ? __expf(sc[nb][e] - ref) : 0.f;
        l += pe;                                        // this lane's keys; summed over the quad at the end
        if (hl < RT) s_p[warp][k].v[hl] = pe;
      }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      const float cr = __shfl_sync(0xffffffffu, corr, r * 4);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[r][e] *= cr;
    }
    if (!__all_sync(0xffffffffu, mbar_wait(&full[warp][1], phase, &abort_flag))) break;
#pragma unroll
    for (int st = 0; st < STEPS; ++st) {
      const int k = st * KPS + kl;
      uint4 u = piece(vt, 1, key0, k, dl);
      if (key0 + k >= len) u = make_uint4(0u, 0u, 0u, 0u);     // never written: its weight is 0, but 0 times anything is not
      float vf[8];
      unpack16B(u, vf);
      const HeadRow<RT> w = s_p[warp][k];
#pragma unroll
      for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[r][e] += w.v[r] * vf[e];
    }
    __syncwarp();                                       // the next tile overwrites s_p and the tile of V
    if (lane == 0) fetch(t + nw * cs, 1);
  }

  // No pdl_trigger(), as in gemm_skinny.cu: a 7B block of 8 sequences 104.9 us with it here, 102.2 without; one of a 125M model,
  // 4 sequences, 27.7 / 26.8.
  // over the key slots of the warp, then the warps of the CTA
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  if (tl == 0 && hl < RT) { s_m[warp][hl] = m; s_l[warp][hl] = l; }
#pragma unroll
  for (int r = 0; r < RT; ++r) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
#pragma unroll
      for (int o = LPK; o < 32; o <<= 1) acc[r][e] += __shfl_xor_sync(0xffffffffu, acc[r][e], o);
      if (kl == 0) reinterpret_cast<float*>(kt)[r * D + dl * 8 + e] = acc[r][e];      // every copy into it has been waited for
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < RT * D; i += blockDim.x) {
    const int r = i / D, d = i % D;
    float mx = -INFINITY;
    for (int w = 0; w < nw; ++w) mx = fmaxf(mx, s_m[w][r]);
    const float ref = mx == -INFINITY ? 0.f : mx;
    float ls = 0.f, o = 0.f;
    for (int w = 0; w < nw; ++w) {
      const float f = __expf(s_m[w][r] - ref);
      ls += s_l[w][r] * f;
      o += reinterpret_cast<const float*>(tiles + size_t(w) * 2 * TB)[r * D + d] * f;
    }
    c_o[r][d] = o;
    if (d == 0) { c_m[r] = mx; c_l[r] = ls; }
  }
  // over the CTAs of the cluster: every CTA finishes its share of the outputs
  cluster.sync();
  for (int i = rank * int(blockDim.x) + int(threadIdx.x); i < RT * D; i += cs * int(blockDim.x)) {
    const int r = i / D, d = i % D;
    if (r >= nh) break;
    float mx = -INFINITY;
    for (int c = 0; c < cs; ++c) mx = fmaxf(mx, *cluster.map_shared_rank(&c_m[r], c));
    const float ref = mx == -INFINITY ? 0.f : mx;
    float ls = 0.f, o = 0.f;
    for (int c = 0; c < cs; ++c) {
      const float f = __expf(*cluster.map_shared_rank(&c_m[r], c) - ref);
      ls += *cluster.map_shared_rank(&c_l[r], c) * f;
      o += *cluster.map_shared_rank(&c_o[r][d], c) * f;
    }
    // no valid key: zeros. ls == 0 with valid keys: every score is -infinity, and 0 / 0 is what the softmax of those is
    p.out[(size_t(b) * p.QH + h0 + r) * D + d] = __float2bfloat16(len <= 0 ? 0.f : o / ls);
  }
  cluster.sync();                                       // peers still read this CTA's state until here
  if (threadIdx.x == 0 && abort_flag != 0 && p.status != nullptr && atomicCAS(p.status, 0, abort_flag) == 0) p.status[1] = 330;
}

// What one of the decode attention's kernels may use and how much of it fits, per device of the process (nothing is kept of a
// request that failed).
struct DecodeDevice {
  std::atomic<bool> allowed{false};       // its dynamic shared memory: more than 48 KiB from head_dim 128's 4 warps on
  std::atomic<int> fit[5] = {};           // 1 + the CTAs of 1 to 4 warps that run at the same time
  std::atomic<int> clusters[4][DA_MAX_WARPS + 1] = {};      // 1 + the clusters of 1, 2, 4, 8 CTAs of that many warps
};

template <int D, int RT>
static int launch_decode(DecodeParams p, int B, cudaStream_t st) {
  p.groups = (p.QH / p.KVH + RT - 1) / RT;
  const long pairs = long(B) * p.KVH * p.groups;
  if (p.KVH * p.groups > 65535 || B > 65535) return static_cast<int>(cudaErrorInvalidValue);
  constexpr int kTiles = 2 * DA_TILE * D * 2;
  constexpr int kMaxWarps = 131072 / kTiles < DA_MAX_WARPS ? 131072 / kTiles : DA_MAX_WARPS;
  const auto kern = p.kqv != nullptr ? decode_attn_kernel<D, RT, true> : decode_attn_kernel<D, RT, false>;
  // With the shared memory asked for on the first device alone, a launch on a second one would be refused.
  static DecodeDevice devices[2][64];
  int dev = 0;
  B200_CHECK(cudaGetDevice(&dev));
  DecodeDevice* known = dev >= 0 && dev < 64 ? &devices[p.kqv != nullptr][dev] : nullptr;
  if (known == nullptr || !known->allowed.load(std::memory_order_acquire)) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxWarps * kTiles);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return static_cast<int>(e);
    }
    if (known != nullptr) known->allowed.store(true, std::memory_order_release);
  }
  auto once = [](std::atomic<int>* kept, auto query) -> long {        // a count that the device is asked for once, 0: not known
    int n = kept != nullptr ? kept->load(std::memory_order_relaxed) : 0;
    if (n == 0) {
      if (query(&n) != cudaSuccess) {
        cudaGetLastError();
        return 0;
      }
      ++n;
      if (kept != nullptr) kept->store(n, std::memory_order_relaxed);
    }
    return n - 1;
  };
  auto fit = [&](int warps) -> long {      // CTAs of that many warps (up to 4) that run at the same time
    return once(known != nullptr ? &known->fit[warps] : nullptr, [&](int* n) {
      const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, kern, 32 * warps, warps * kTiles);
      *n *= num_sms();
      return e;
    });
  };
  auto fit_clusters = [&](int cs, int warps) -> long {
    return once(known != nullptr ? &known->clusters[cs == 8 ? 3 : cs >> 1][warps] : nullptr, [&](int* n) {
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = cs;
      at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(cs);
      cfg.blockDim = dim3(32 * warps);
      cfg.dynamicSmemBytes = warps * kTiles;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      return cudaOccupancyMaxActiveClusters(n, kern, &cfg);
    });
  };
  const int keys = p.kqv != nullptr ? p.pos + 1 : p.Tmax;       // what the lengths are expected to be, at most; longer ones work too
  const int tiles = (keys + DA_TILE - 1) / DA_TILE;
  // Up to 8 CTAs per (sequence, KV head): doubled while there are more tiles than CTAs, one CTA per SM of head_dim 128 (two
  // of 64, four of 32: the same bytes) is not exceeded yet and twice as many still run at the same time. At least four warps
  // (they also form the result), up to 128 KiB of tiles while at most one CTA per SM exists. Swept for the attention alone, us:
  // 8 sequences, 8 KV heads of 128, 3001 keys 34.8 with 256 CTAs of four warps (45.1 with 512, 36.9 with 512 of two); 16 x 4
  // heads, 1001 keys 21.2 with 256 of four (28.7 with 512 of four); 4 x 4 heads, 301 keys 14.3 with four warps (22.5 with eight:
  // their 128 KiB have to wait for an empty SM); 32 x 4 heads of 32, 301 keys 6.4 with 512 of four (11.2 with 1024).
  int cs = 1;
  while (cs < 8 && cs < tiles && pairs * cs * kTiles <= 16384L * num_sms() && 2 * pairs * cs <= fit(4)) cs *= 2;
  int warps = (tiles + cs - 1) / cs;
  const int cap = pairs * cs <= num_sms() ? kMaxWarps : 4;
  if (warps > cap) warps = cap;
  if (warps < 4) warps = 4;
  // More than four only where all clusters still run at once: CTAs of which an SM holds one leave no room for the last of 16
  // clusters of eight (a 1.3B block of 4 sequences, 2048 keys 53.4 us with eight warps, 47.3 with four; 125M, 3001 keys 35.1 with
  // twelve, 29.9 with eight).
  while (warps > 4 && pairs > fit_clusters(cs, warps)) warps = (warps - 1) / 4 * 4 < 4 ? 4 : (warps - 1) / 4 * 4;
  // Fewer where only they all run at once, with a twentieth to spare for an uneven spread: 512 CTAs of head_dim 128, 31 keys
  // 12.4 us with two warps (18.9 with four, of which 296 fit), 3001 keys 131 (142); 1024 16.7 and 252 with one (36 and 283).
  auto one_round = [&](int w) { return 20 * pairs * cs <= 19 * fit(w); };
  if (warps == 4 && pairs * cs > num_sms() && one_round(1))
    while (!one_round(warps)) --warps;
  p.status = status_ptr();
  return static_cast<int>(launch_pdl(kern, dim3(cs, p.KVH * p.groups, B), dim3(32 * warps), warps * kTiles, st, cs, p));
}

template <int D>
static int launch_decode_heads(const DecodeParams& p, int B, cudaStream_t st) {
  const int R = p.QH / p.KVH;
  if (R == 1) return launch_decode<D, 1>(p, B, st);
  if (R == 2) return launch_decode<D, 2>(p, B, st);
  return launch_decode<D, 4>(p, B, st);
}

static int launch_decode_dim(const DecodeParams& p, int B, int D, cudaStream_t st) {
  switch (D) {
    case 32: return launch_decode_heads<32>(p, B, st);
    case 64: return launch_decode_heads<64>(p, B, st);
    case 128: return launch_decode_heads<128>(p, B, st);
    default: return static_cast<int>(cudaErrorInvalidValue);
  }
}

}  // namespace b200

using namespace b200;

// out[b, h] = softmax(q[b, h] K^T * scale) V over the first lens[b] (at most Tmax) keys of the caches
// [B, KVH, Tmax, D]; zeros where lens[b] <= 0.
B200_API int b200_decode_attn(const void* q, const void* kcache, const void* vcache, void* out, const void* lens,
                              int B, int QH, int KVH, int Tmax, int D, float scale, cudaStream_t st) {
  if (B <= 0) return 0;
  const uintptr_t all = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(kcache) |
                        reinterpret_cast<uintptr_t>(vcache);
  if (QH <= 0 || KVH <= 0 || QH % KVH != 0 || (all & 15) != 0) return static_cast<int>(cudaErrorInvalidValue);
  DecodeParams p = {};
  p.q = static_cast<const bf16*>(q);
  p.kc = static_cast<const bf16*>(kcache);
  p.vc = static_cast<const bf16*>(vcache);
  p.out = static_cast<bf16*>(out);
  p.lens = static_cast<const int*>(lens);
  p.QH = QH; p.KVH = KVH; p.Tmax = Tmax; p.scale = scale;
  return launch_decode_dim(p, B, D, st);
}

// The same for the token whose projection is kqv[b] = [K | Q | V] (pitch ld, K and Q un-rotated): rotates K and Q by
// the angle of position pos (cos / sin: table rows of that position, [D / 2] fp32), writes K and V to position pos
// of the caches and attends over the first lens[b] keys, position pos included with its new values. One launch in
// place of two rotations, two or three cache copies and the attention (12 -> 8 launches per block; 1.3B, one token,
// device time of the five steps 23 -> 13 us; the block 217 -> 165 us, host included).
B200_API int b200_decode_attn_append(const void* kqv, void* kcache, void* vcache, void* out, const void* lens,
                                     const void* cosr, const void* sinr, int B, int QH, int KVH, int Tmax, int D, int ld,
                                     int pos, float scale, cudaStream_t st) {
  if (B <= 0) return 0;
  const uintptr_t all = reinterpret_cast<uintptr_t>(kqv) | reinterpret_cast<uintptr_t>(kcache) |
                        reinterpret_cast<uintptr_t>(vcache);
  if (QH <= 0 || KVH <= 0 || QH % KVH != 0 || (all & 15) != 0 || (ld % 8) != 0 || pos < 0 || pos >= Tmax ||
      kqv == nullptr || cosr == nullptr || sinr == nullptr)
    return static_cast<int>(cudaErrorInvalidValue);
  DecodeParams p = {};
  p.kc = p.kcw = static_cast<bf16*>(kcache);
  p.vc = p.vcw = static_cast<bf16*>(vcache);
  p.out = static_cast<bf16*>(out);
  p.lens = static_cast<const int*>(lens);
  p.QH = QH; p.KVH = KVH; p.Tmax = Tmax; p.scale = scale;
  p.kqv = static_cast<const bf16*>(kqv);
  p.cosr = static_cast<const float*>(cosr);
  p.sinr = static_cast<const float*>(sinr);
  p.ld = ld; p.pos = pos;
  return launch_decode_dim(p, B, D, st);
}

// gemm_skinny.cu
B200_API int b200_gemm_skinny(const void* A, const void* B, void* D, const void* C, int M, int N, int K, int lda, int ldb,
                              int ldd, int ldc, int b_k_rows, int out_f32, float alpha, cudaStream_t stream);
B200_API int b200_gemm_skinny_swiglu(const void* A, const void* B, void* ACT, int M, int I, int K, int lda, int ldb,
                                     int ldact, cudaStream_t stream);

// The attention half of a block for one token per sequence, three launches from one call (at a few microseconds of
// device time each, a call into this library from Python costs as much as a launch):
//   kqv = x W_kqv;  o = rotate, append to the caches, attend;  out = o W_o (+ residual)
// x [B, H] (pitch ldx), W_kqv [H, (QH + 2 KVH) D], W_o [QH D, H] contiguous, kqv / o: caller's scratch.
B200_API int b200_decode_attn_block(const void* x, const void* w_kqv, const void* w_o, const void* residual, void* out,
                                    void* kqv, void* o, void* kcache, void* vcache, const void* lens, const void* cosr,
                                    const void* sinr, int B, int H, int QH, int KVH, int Tmax, int D, int ldx, int ldr,
                                    int pos, float scale, cudaStream_t st) {
  const int N = (QH + 2 * KVH) * D, HO = QH * D;
  int rc = b200_gemm_skinny(x, w_kqv, kqv, nullptr, B, N, H, ldx, N, N, 0, 1, 0, 1.f, st);
  if (rc == 0)
    rc = b200_decode_attn_append(kqv, kcache, vcache, o, lens, cosr, sinr, B, QH, KVH, Tmax, D, N, pos, scale, st);
  if (rc == 0) rc = b200_gemm_skinny(o, w_o, out, residual, B, H, HO, HO, H, H, ldr, 1, 0, 1.f, st);
  return rc;
}

// The MLP half for few rows, two launches from one call: out = (silu(x W_gate) * (x W_value)) W_out (+ residual);
// W_gate_val [H, 2 I] and W_out [I, H] contiguous, act: caller's scratch [M, I].
B200_API int b200_mlp_few_rows(const void* x, const void* w_gate_val, const void* w_out, const void* residual, void* out,
                               void* act, int M, int H, int I, int ldx, int ldr, cudaStream_t st) {
  const int rc = b200_gemm_skinny_swiglu(x, w_gate_val, act, M, I, H, ldx, 2 * I, I, st);
  if (rc != 0) return rc;
  return b200_gemm_skinny(act, w_out, out, residual, M, H, I, I, H, H, ldr, 1, 0, 1.f, st);
}
