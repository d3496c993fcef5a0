// Causal GQA flash-attention forward on tcgen05 (head_dim 128 or 64).
//
// A CTA owns one or two consecutive 128-row query tiles of one (batch, head) and walks the key tiles once. Each query
// tile has its own softmax warpgroup, its own score buffer and its own output accumulator in tensor memory:
//
//   head_dim 128: one CTA per SM, two query tiles          head_dim 64: two CTAs per SM, one query tile each
//     columns   0..127  S_0 (fp32 scores of query tile 0;    columns   0..127  S
//                       P_0 as bf16 overwrites 0..63)                128..191  O
//             128..255  S_1                                          192..255  P (bf16)
//             256..383  O_0 (fp32, accumulated by P V)
//             384..511  O_1
//
// A thread of a softmax warpgroup owns one query row (one TMEM lane) and all 128 key columns of the tile, so the row
// maximum and the row sum never leave the thread. While one warpgroup of an SM is in its exp2 pass the tensor core runs
// the other one's P V and next S; neither side waits for the other except through the data it needs.
//
// What bounds it: a tile's chain scores -> maximum -> exp2 -> P V -> next scores. head_dim 64 has the columns for a P of
// its own, so its next scores start as soon as the present ones are in registers; head_dim 128 hands P over in two halves
// instead. With two query tiles per CTA for head_dim 64 too, both warpgroups went through their exponentials at the same
// time (16 a clock and SM) and an SM stood still while a CTA started and stored; a CTA each lets them drift apart.
// 8 x 1024 tokens, 12 / 4 heads of 64: 46.4 us -> 36.2 (4 x 4096: 203 -> 161, 1 x 777: 17.8 -> 13.2); 4 x 2048, 16 / 4 heads
// of 128: 98 -> 90. Tried and slower: half a row per thread with four warpgroups (43 / 104 us), turns for the exponentials
// (44), part of them on the FMA units by a polynomial (37 to 39 where the present form takes 36).
//
// The running maximum is applied lazily: the reference point m of a row only moves when the new
// tile maximum exceeds it by more than 8 (log2 units), so exp2(s - m) stays below 2^8 and the
// output accumulator has to be rescaled (TMEM load, multiply, TMEM store by the row's own thread)
// only on the rare tiles where that happens. The final 1 / l normalisation uses the same m.
//
// K and V travel through separate 2-deep rings: the K slot of tile j is free as soon as its
// S(j) MMAs have run, long before the V slot, so the TMA load of K(j+2) gets a full iteration of
// lead. The output tile is staged in the (by then unused) Q tile in the 128-byte swizzle and
// stored with cp.async.bulk.tensor. Every wait is bounded (see ptx.cuh). head_dim 64 has one 64-column box per
// Q / K / V / O tile instead of two, four k-steps in S = Q K^T and N = 64 in O += P V.
#include "common.cuh"
#include "ptx.cuh"

namespace b200 {

constexpr float kF3Log2e = 1.4426950408889634f;
constexpr float kF3RescaleStep = 8.f;

struct Flash3Params {
  float* lse;
  const int* valid_len;
  int B, T, QH, KVH;
  int bchunk;            // batch elements whose K and V stay in L2 together
  float scale;
  int* status;
};

template <int kD>
struct F3 {
  static constexpr int kW = kD == 128 ? 2 : 1;                         // query tiles of a CTA
  static constexpr int kCtas = kD == 128 ? 1 : 2;                      // CTAs of an SM
  static constexpr int kThreads = 64 + 128 * kW;                       // warp 0: TMA; 1: MMA, tensor memory; then a warpgroup per tile
  static constexpr int kTile = 128 * kD * 2;
  static constexpr int kQ = 0;                                         // Q_w
  static constexpr int kK = kW * kTile;                                // K ring [2]
  static constexpr int kV = kK + 2 * kTile;                            // V ring [2]
  static constexpr int kBar = kV + 2 * kTile;
  // q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_full[2], pv_done[2], stage_bar[2], early[2] = 19
  static constexpr int kSmem = kBar + 19 * 8 + 16 + 1024;
  // tensor-memory columns
  static constexpr bool kOwnP = kD == 64;                              // P_w beside S_w, not over it
  static constexpr int kCols = kD == 128 ? 512 : 256;
  static constexpr int kColS = 0, kColO = kW * 128, kColP = kOwnP ? kColO + kD : 0;
};

__device__ __forceinline__ void tma_store_4d(const CUtensorMap* m, const void* smem_src, int c0, int c1, int c2,
                                             int c3) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(smem_src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}

__device__ __forceinline__ void tmem_st_32x32b_x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
      "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
      "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}

struct TrueTag { static constexpr bool value = true; };
struct FalseTag { static constexpr bool value = false; };

__device__ __forceinline__ float f3_max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Raw maximum of the 128 scores of one row; masked keys (beyond the diagonal or the valid length) are
// set to -inf in place so that the exponential pass needs no mask.
// Four chains: one chain of 64 dependent maxima took 490 clocks of a tile, these take 400.
template <bool kMask>
__device__ __forceinline__ float f3_row_max(uint32_t (&sc)[128], int key0, int row, int vlen) {
  float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
  for (int e = 0; e < 128; e += 2) {
    if (kMask) {
      const int key = key0 + e;
      if (key > row || key >= vlen) sc[e] = 0xff800000u;
      if (key + 1 > row || key + 1 >= vlen) sc[e + 1] = 0xff800000u;
    }
    mx[(e >> 1) & 3] = f3_max3(mx[(e >> 1) & 3], __uint_as_float(sc[e]), __uint_as_float(sc[e + 1]));
  }
  return fmaxf(f3_max3(mx[0], mx[1], mx[2]), mx[3]);
}

// P = exp2(s * sl2 - m_ref) for scores [kLo, kHi) of one row, packed to bf16 pairs IN PLACE (pair e / 2 lands in
// register e / 2, which has been consumed by then); adds to the two partial row sums.
template <int kLo, int kHi>
__device__ __forceinline__ void f3_row_p(uint32_t (&sc)[128], float sl2, float m_ref, float& rs0, float& rs1) {
#pragma unroll
  for (int e = kLo; e < kHi; e += 2) {
    const float p0 = exp2f(fmaf(__uint_as_float(sc[e]), sl2, -m_ref));
    const float p1 = exp2f(fmaf(__uint_as_float(sc[e + 1]), sl2, -m_ref));
    rs0 += p0;
    rs1 += p1;
    const bf162 t = __floats2bfloat162_rn(p0, p1);
    sc[e >> 1] = *reinterpret_cast<const uint32_t*>(&t);
  }
}

template <int kD>
__global__ void __launch_bounds__(F3<kD>::kThreads, F3<kD>::kCtas)
flash_fwd_tc3_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO,
                     const Flash3Params p) {
  using L = F3<kD>;
  constexpr int kW = L::kW;
  constexpr bool kOwnP = L::kOwnP;
  constexpr uint32_t kTile = L::kTile;
  extern __shared__ uint8_t f3_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(f3_smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBar);
  uint64_t* q_full = bars;
  uint64_t* k_full = bars + 1;
  uint64_t* k_empty = bars + 3;
  uint64_t* v_full = bars + 5;
  uint64_t* v_empty = bars + 7;
  uint64_t* s_full = bars + 9;       // [w]: S_w of the current key tile is in TMEM
  uint64_t* p_full = bars + 11;      // [w]: warpgroup w has written P_w (128 arrivals)
  uint64_t* pv_done = bars + 13;     // [w]: O_w includes the key tile whose P V was committed last
  uint64_t* stage_bar = bars + 15;   // [w]: the output tile of warpgroup w is staged in shared memory
  uint64_t* early = bars + 17;       // [w]: head_dim 64: warpgroup w holds S_w in registers; 128: it has written half of P_w
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 19);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // 1-D grid over chunks of p.bchunk batch elements; inside a chunk the longest rows come first: every (head, batch) of the
  // last query tiles, then of those before. An SM takes three or four CTAs of 2 to 16 key tiles in a training shape: with all
  // the query tiles of one head in a row the SMs were busy for 72 to 110 us (mean 86) of 113.
  int pt, h, b;
  {
    const int n_pairs = (p.T + 128 * kW - 1) / (128 * kW);
    const int per_chunk = n_pairs * p.QH * p.bchunk;
    const int chunk = int(blockIdx.x) / per_chunk, r = int(blockIdx.x) - chunk * per_chunk;
    const int hb = p.QH * min(p.bchunk, p.B - chunk * p.bchunk);
    pt = n_pairs - 1 - r / hb;
    h = (r % hb) % p.QH;
    b = chunk * p.bchunk + (r % hb) / p.QH;
  }
  const int kvh = h / (p.QH / p.KVH);
  const int T = p.T;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
      mbar_init(&s_full[s], 1);
      mbar_init(&p_full[s], 128);
      mbar_init(&pv_done[s], 1);
      mbar_init(&stage_bar[s], 128);
      mbar_init(&early[s], 128);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmO);
  }
  if (warp == 1) tmem_alloc(tmem_slot, L::kCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  constexpr uint32_t kColS = L::kColS, kColO = L::kColO, kColP = L::kColP;
  pdl_wait();                            // by every role: their bounded waits start counting behind it
  pdl_trigger();
  const int vlen = p.valid_len ? checked_index(p.valid_len[b], T, p.status, 301) : T;
  const int kv_tiles = (max(vlen, 1) + 127) / 128;
  int nt[2] = {0, 0};
#pragma unroll
  for (int w = 0; w < kW; ++w) {
    const int mt = kW * pt + w;
    nt[w] = (mt * 128 < T) ? min(mt + 1, kv_tiles) : 0;
  }
  const int nmax = max(nt[0], nt[1]);

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0) {
      mbar_expect_tx(q_full, (nt[1] > 0 ? 2 : 1) * kTile);
      for (int w = 0; w < kW; ++w) {
        if (nt[w] == 0) continue;
        uint8_t* sQ = smem + L::kQ + w * kTile;
        tma_load_4d(sQ, &tmQ, q_full, 0, h, (kW * pt + w) * 128, b);
        if (kD == 128) tma_load_4d(sQ + 16384, &tmQ, q_full, 64, h, (kW * pt + w) * 128, b);
      }
      for (int j = 0; j < nmax; ++j) {
        const int s = j & 1;
        const uint32_t par = ((j >> 1) & 1) ^ 1;
        if (!mbar_wait(&k_empty[s], par, abort_flag)) break;
        uint8_t* sK = smem + L::kK + s * kTile;
        mbar_expect_tx(&k_full[s], kTile);
        tma_load_4d(sK, &tmK, &k_full[s], 0, kvh, j * 128, b);
        if (kD == 128) tma_load_4d(sK + 16384, &tmK, &k_full[s], 64, kvh, j * 128, b);
        if (!mbar_wait(&v_empty[s], par, abort_flag)) break;
        uint8_t* sV = smem + L::kV + s * kTile;
        mbar_expect_tx(&v_full[s], kTile);
        tma_load_4d(sV, &tmV, &v_full[s], 0, kvh, j * 128, b);
        if (kD == 128) tma_load_4d(sV + 16384, &tmV, &v_full[s], 64, kvh, j * 128, b);
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    {
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, 128, 0, 0);
      constexpr uint32_t idesc_pv = umma_idesc_bf16(128, kD, 0, 1);
      auto issue_s = [&](int w, int j) {
        const uint64_t dQ = umma_smem_desc(smem_u32(smem + L::kQ + w * kTile), 16, 1024);
        const uint64_t dK = umma_smem_desc(smem_u32(smem + L::kK + (j & 1) * kTile), 16, 1024);
#pragma unroll
        for (int kk = 0; kk < kD / 16; ++kk) {
          const uint32_t off = ((kk >> 2) * 16384 + (kk & 3) * 32) >> 4;      // in the descriptors' 16-byte units
          umma_bf16_ss_warp(tmem_base + kColS + w * 128, dQ + off, dK + off, idesc_s, kk != 0);
        }
        umma_commit_warp(&s_full[w]);
      };
      bool ok = mbar_wait_warp(q_full, 0, abort_flag);
      if (ok && nmax > 0) {
        ok = mbar_wait_warp(&k_full[0], 0, abort_flag);
        if (ok) {
          tc_fence_after();
          for (int w = 0; w < kW; ++w)
            if (nt[w] > 0) issue_s(w, 0);
          umma_commit_warp(&k_empty[0]);
        }
      }
      // O_w += P_w V for k-steps [lo, hi) of key tile j
      auto issue_pv = [&](int w, int j, int lo, int hi) {
        const uint64_t dV = umma_smem_desc(smem_u32(smem + L::kV + (j & 1) * kTile), 16384, 1024);
        const uint32_t tP = tmem_base + kColP + w * 128;
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          if (kk >= lo && kk < hi)
            umma_bf16_ts_warp(tmem_base + kColO + w * 128, tP + kk * 8, dV + kk * 128, idesc_pv, (j | kk) != 0);
      };
      for (int j = 0; j < nmax && ok; ++j) {
        bool v_ready = false, k_ready = false;
        // The next scores of query tile w: with a P of its own (head_dim 64) as soon as the warpgroup has read the present
        // ones, else behind the P V whose P lies over them.
        auto next_s = [&](int w) {
          if (!k_ready && !mbar_wait_warp(&k_full[(j + 1) & 1], ((j + 1) >> 1) & 1, abort_flag)) return false;
          k_ready = true;
          tc_fence_after();
          issue_s(w, j + 1);
          return true;
        };
        if (kOwnP) {
          for (int w = 0; w < kW && ok; ++w) {
            if (j + 1 >= nt[w]) continue;
            ok = mbar_wait_warp(&early[w], j & 1, abort_flag) && next_s(w);
          }
          if (!ok) break;
          if (j + 1 < nmax) umma_commit_warp(&k_empty[(j + 1) & 1]);
        }
        for (int w = 0; w < kW && ok; ++w) {
          if (j >= nt[w]) continue;
          if (!mbar_wait_warp(kOwnP ? &p_full[w] : &early[w], j & 1, abort_flag)) { ok = false; break; }
          if (!v_ready) {
            if (!mbar_wait_warp(&v_full[j & 1], (j >> 1) & 1, abort_flag)) { ok = false; break; }
            v_ready = true;
          }
          tc_fence_after();
          if (kOwnP) {
            issue_pv(w, j, 0, 8);
          } else {
            issue_pv(w, j, 0, 4);
            if (!mbar_wait_warp(&p_full[w], j & 1, abort_flag)) { ok = false; break; }
            tc_fence_after();
            issue_pv(w, j, 4, 8);
          }
          umma_commit_warp(&pv_done[w]);
          if (!kOwnP && j + 1 < nt[w] && !next_s(w)) { ok = false; break; }
        }
        if (!ok) break;
        if (!kOwnP && j + 1 < nmax) umma_commit_warp(&k_empty[(j + 1) & 1]);
        umma_commit_warp(&v_empty[j & 1]);
      }
    }
  } else {
    // ---------------------------------------------------------------- softmax warpgroup w: one query tile
    const int w = (warp - 2) >> 2;
    const int q = warp & 3;
    const int rloc = q * 32 + lane;
    const int mt = kW * pt + w;
    const int row = mt * 128 + rloc;
    const int my_tiles = nt[w];
    const uint32_t lane_sel = uint32_t(q * 32) << 16;
    const uint32_t tS = tmem_base + lane_sel + kColS + w * 128;
    const uint32_t tO = tmem_base + lane_sel + kColO + w * 128;
    const uint32_t tP = tmem_base + lane_sel + kColP + w * 128;
    const float sl2 = p.scale * kF3Log2e;
    float m_ref = 0.f, l_run = 0.f;          // reference maximum (log2 units) and the row sum relative to it
    bool ok = true;
    for (int j = 0; j < my_tiles && ok; ++j) {
      if (!mbar_wait(&s_full[w], j & 1, abort_flag)) { ok = false; break; }
      tc_fence_after();
      const bool need_mask = (j == mt) || (j * 128 + 128 > vlen);
      const int key0 = j * 128;
      // The whole row (128 raw scores) is read in one go: four loads, one wait. A tensor-memory load queues
      // behind the MMAs the other warpgroup has in flight, so every separate round trip costs that wait again.
      uint32_t sc[128];
      tmem_ld_32x32b_x32(tS, *reinterpret_cast<uint32_t(*)[32]>(&sc[0]));
      tmem_ld_32x32b_x32(tS + 32, *reinterpret_cast<uint32_t(*)[32]>(&sc[32]));
      tmem_ld_32x32b_x32(tS + 64, *reinterpret_cast<uint32_t(*)[32]>(&sc[64]));
      tmem_ld_32x32b_x32(tS + 96, *reinterpret_cast<uint32_t(*)[32]>(&sc[96]));
      tmem_ld_wait();
      if (kOwnP) {                       // the tensor core may write the next scores over these
        tc_fence_before();
        mbar_arrive(&early[w]);
      }
      float mx = (need_mask ? f3_row_max<true>(sc, key0, row, vlen) : f3_row_max<false>(sc, key0, row, vlen)) * sl2;
      // The reference maximum is set by the first tile and afterwards moves only when a tile exceeds it by
      // more than 2^8; then O_w and the row sum are rescaled by the row's own thread.
      if (j == 0) {
        m_ref = (mx == -INFINITY) ? 0.f : mx;
      } else {
        const bool need = mx > m_ref + kF3RescaleStep;
        if (__any_sync(0xffffffffu, need)) {
          // O_w holds the key tiles up to j - 1 once their P V has completed
          if (!mbar_wait(&pv_done[w], (j - 1) & 1, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const float corr = need ? exp2f(m_ref - mx) : 1.f;
          l_run *= corr;
#pragma unroll 1
          for (int c = 0; c < kD / 16; ++c) {
            uint32_t t[16];
            tmem_ld_32x32b_x16(tO + c * 16, t);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 16; ++e) t[e] = __float_as_uint(__uint_as_float(t[e]) * corr);
            tmem_st_32x32b_x16(tO + c * 16, t);
          }
          tmem_st_wait();
          if (need) m_ref = mx;
        }
      }
      // P = exp2(s * scale - m_ref) as bf16 pairs, packed in place over the first 64 registers, and its row sum
      float rs0 = 0.f, rs1 = 0.f;
      if (kOwnP) {
        f3_row_p<0, 128>(sc, sl2, m_ref, rs0, rs1);
        if (j > 0 && !mbar_wait(&pv_done[w], (j - 1) & 1, abort_flag)) { ok = false; break; }   // P_w has been read
        tc_fence_after();
      } else {
        // head_dim 128: the next scores wait for this P V, so its first half is handed over early
        f3_row_p<0, 64>(sc, sl2, m_ref, rs0, rs1);
        tmem_st_32x32b_x16(tP, *reinterpret_cast<const uint32_t(*)[16]>(&sc[0]));
        tmem_st_32x32b_x16(tP + 16, *reinterpret_cast<const uint32_t(*)[16]>(&sc[16]));
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive(&early[w]);
        f3_row_p<64, 128>(sc, sl2, m_ref, rs0, rs1);
      }
#pragma unroll
      for (int c = kOwnP ? 0 : 2; c < 4; ++c)
        tmem_st_32x32b_x16(tP + c * 16, *reinterpret_cast<const uint32_t(*)[16]>(&sc[16 * c]));
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&p_full[w]);
      l_run += rs0 + rs1;
    }
    if (ok && my_tiles > 0) {
      if (mbar_wait(&pv_done[w], (my_tiles - 1) & 1, abort_flag)) {
        tc_fence_after();
        // all MMAs of this query tile have completed: its Q tile in shared memory is free and becomes
        // the staging area of the output (two 128 x 64 boxes, 128-byte swizzle)
        const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
        uint8_t* stg = smem + L::kQ + w * kTile;
        const uint32_t swz = uint32_t(rloc & 7);
#pragma unroll 1
        for (int c = 0; c < kD / 32; ++c) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(tO + c * 32, r);
          tmem_ld_wait();
          uint8_t* rowp = stg + (c >> 1) * 16384 + rloc * 128;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            uint4 o;
            bf162* o2 = reinterpret_cast<bf162*>(&o);
#pragma unroll
            for (int e = 0; e < 4; ++e)
              o2[e] = __floats2bfloat162_rn(__uint_as_float(r[8 * k + 2 * e]) * inv,
                                            __uint_as_float(r[8 * k + 2 * e + 1]) * inv);
            *reinterpret_cast<uint4*>(rowp + ((uint32_t((c & 1) * 4 + k) ^ swz) << 4)) = o;
          }
        }
        if (row < T)
          p.lse[(size_t(b) * p.QH + h) * T + row] =
              l_run > 0.f ? m_ref * 0.6931471805599453f + logf(l_run) : -INFINITY;
        fence_proxy_async_smem();
        mbar_arrive(&stage_bar[w]);
        if (q == 0 && lane == 0) {
          if (mbar_wait(&stage_bar[w], 0, abort_flag)) {
            tma_store_4d(&tmO, stg, 0, h, mt * 128, b);
            if (kD == 128) tma_store_4d(&tmO, stg + 16384, 64, h, mt * 128, b);
            tma_store_commit();
            tma_store_wait_read<0>();
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, L::kCols);
  }
  if (threadIdx.x == 0 && *abort_flag != 0 && p.status != nullptr) {
    if (atomicCAS(p.status, 0, int(*abort_flag)) == 0) p.status[1] = 302;
  }
}

}  // namespace b200

using namespace b200;

// Same contract as b200_flash_fwd_tc (inputs already rotated) for head_dim 128 or 64; the output must be
// TMA-addressable (16-byte aligned base, strides that are multiples of 8 elements).
B200_API int b200_flash_fwd_tc3(const void* q, const void* k, const void* v, void* o, void* lse, const void* valid_len,
                                const long long* strides, int B, int T, int QH, int KVH, int D, float scale,
                                cudaStream_t st) {
  if (B <= 0 || T <= 0) return 0;
  if ((D != 128 && D != 64) || QH % KVH != 0) return static_cast<int>(cudaErrorInvalidValue);
  for (int i = 0; i < 12; ++i)
    if (strides[i] % 8 != 0) return static_cast<int>(cudaErrorInvalidValue);
  if ((reinterpret_cast<uintptr_t>(o) & 15) != 0) return static_cast<int>(cudaErrorInvalidValue);
  TensorMap tq = get_tensor_map_bthd(q, B, T, QH, D, strides[0], strides[1], strides[2], 128, 64);
  TensorMap tk = get_tensor_map_bthd(k, B, T, KVH, D, strides[3], strides[4], strides[5], 128, 64);
  TensorMap tv = get_tensor_map_bthd(v, B, T, KVH, D, strides[6], strides[7], strides[8], 128, 64);
  TensorMap to = get_tensor_map_bthd(o, B, T, QH, D, strides[9], strides[10], strides[11], 128, 64);
  if (!tq || !tk || !tv || !to) return static_cast<int>(cudaErrorInvalidValue);
  Flash3Params p;
  p.lse = static_cast<float*>(lse);
  p.valid_len = static_cast<const int*>(valid_len);
  p.B = B; p.T = T; p.QH = QH; p.KVH = KVH; p.scale = scale;
  p.status = status_ptr();
  static bool configured = false;
  if (!configured) {
    B200_CHECK(cudaFuncSetAttribute(flash_fwd_tc3_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, F3<128>::kSmem));
    B200_CHECK(cudaFuncSetAttribute(flash_fwd_tc3_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, F3<64>::kSmem));
    configured = true;
  }
  {
    const double per_batch = 2.0 * T * D * 2.0 * KVH;             // K and V; about two thirds of the L2 is budgeted
    const int bc = int(80.0e6 / per_batch);
    p.bchunk = bc < 1 ? 1 : (bc > B ? B : bc);
  }
  const int rows = 128 * (D == 128 ? F3<128>::kW : F3<64>::kW);
  const long long ctas = (long long)((T + rows - 1) / rows) * QH * B;
  if (ctas > 0x7fffffffLL) return static_cast<int>(cudaErrorInvalidValue);
  const dim3 grid(static_cast<unsigned>(ctas));
  if (D == 128)
    return static_cast<int>(launch_pdl(flash_fwd_tc3_kernel<128>, grid, dim3(F3<128>::kThreads), F3<128>::kSmem, st, 0, *tq, *tk,
                                       *tv, *to, p));
  return static_cast<int>(launch_pdl(flash_fwd_tc3_kernel<64>, grid, dim3(F3<64>::kThreads), F3<64>::kSmem, st, 0, *tq, *tk,
                                     *tv, *to, p));
}
