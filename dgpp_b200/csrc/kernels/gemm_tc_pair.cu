// W4A16 GEMM on CTA pairs: out[T, N] = alpha * x[T, K] . W[N, K]^T (+ residual), 4-bit weights (NVFP4 with
// e4m3 scales per 16, or MXFP4 with e8m0 scales per 32) expanded to bf16 on the way into TENSOR MEMORY, bf16
// activations, fp32 accumulation in TMEM.  Same arithmetic as the single-CTA kernel of gemm_tc.cu (bit-identical
// results without split-K: same converted operands, same K order), different tiling:
//
//   two CTAs of a cluster (one TPC) own 256 weight rows x bn tokens (bn <= 256).  Each CTA streams and converts ITS 128
//   weight rows and loads ITS half of the tokens; one `tcgen05.mma.cta_group::2` per K = 16 step, issued by the first
//   CTA, multiplies all 256 rows by all bn tokens (a pair's MMA takes multiples of 32 columns: a tile of another width
//   carries some of the next rows along and drops them).  The converted weights are the A operand and live in TMEM: a
//   converter thread owns one weight row = one TMEM lane, so 64 weights leave its registers as one `tcgen05.st` and
//   never cross shared memory.  (With A in shared memory a K = 64 step of 256 tokens takes 643 cycles, with A in TMEM 544; the
//   arithmetic's own minimum is 512.)  No TMA multicast: every CTA issues plain loads into its own shared memory.
//
// TMEM (all 512 columns): the accumulator (256) and four A stages of 128 K (64 columns each).  Persistent: one pair per TPC
// walks (tile, split) units, tokens fastest, so that the pairs running together share few weight tiles and all token
// tiles of a chunk stay in L2.
//
// What bounds it: at wide tiles the tensor pipe (2048 x 34816 x 5120: 474 us = 1540 TFLOP/s, 0.91 of the measured cuBLAS burst rate;
// the single-CTA kernel 1216 us), at narrow ones the conversion: 345 cycles per K = 64 block up to 128 tokens, 208 of them the integer
// pipe's.  A set of converter warps has a stage of the ring to itself and converts its two blocks behind one wait for raw weights and one
// for the stage's columns (a block at a time, four sets to a raw stage: 480 cycles, half of them waits; 37 x 34816 x 5120 40 us, 36 so).
// The weights have a producer of their own: behind the activations' ring, which ends 512 K ahead of the MMAs,
// their loads were a round trip to HBM on every stage's way (converters waited 780 of 1900 cycles; 37 x 34816 x 5120 50 us).
// 2048 x 5120 x 17408: 266 us, 173 x 5120 x 5120: 20 us.
//
// Handshakes (all waits bounded, expiry -> status code, everything unwinds, TMEM freed):
//   own CTA:          raw_full / raw_empty (TMA -> converters), acc_full (MMA -> epilogue);
//   both -> first:    activation tiles of both CTAs complete on full of the first CTA (`cta_group::2` loads may signal the
//                     pair's other barrier), converter warps of both arrive there too, epilogue warps on acc_empty;
//   first -> both:    `tcgen05.commit` with a CTA mask arrives on done / acc_full of both CTAs when the MMAs of a block (of a
//                     tile) have completed; the producers and the converters both wait for `done`.
// (Arrivals on the other CTA's barriers release at CTA scope: what they order is tensor memory, by the tcgen05 fences; a
// cluster-scope release took 1100 cycles per arrival, three times a block's MMAs.)
// Warp roles (896 threads): warp 0 MMA issuer (first CTA) and TMEM owner, 1 TMA producer of the activations, 2 of the weights, 4..19 converters (four sets, one
// per stage of the ring), 20..27 epilogue.
// (reference counterpart: src/kernels/fp4w_gemm.cu, the W4A16 prefill GEMM.)
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <string.h>

#include "common/common.h"
#include "common/dtypes.cuh"
#include "common/ptx.cuh"
#include "kernels/gemm_common.cuh"

namespace dgpp {

constexpr int kPrBM = 128;          // weight rows per CTA
constexpr int kPrBK = 64;
constexpr int kPrMaxBN = 256;       // tokens per pair tile = MMA N, at most
constexpr int kPrSets = 4;            // converter sets of four warps; set s has stage s of the ring, two K = 64 blocks at a time
constexpr int kPrMma = 0, kPrTma = 1, kPrRaw = 2, kPrConv = 4, kPrEpi = kPrConv + kPrSets * 4;   // first warp of each role
constexpr int kPrEpiWarps = 8;        // two per lane quadrant, taking turns at 16 columns
constexpr int kPrThreads = (kPrEpi + kPrEpiWarps) * 32;
constexpr int kPrStages = 4, kPrSR = 4;   // stages of 128 K (activations and converted weights), raw stages of 256 K
constexpr int kPrHalfB = kPrMaxBN / 2 * 128;    // 16 KB: half of the tile's tokens, 64 K each
constexpr int kPrStageB = 2 * kPrHalfB;
constexpr int kPrStageRaw = kPrBM * 128;        // 16 KB of packed fp4 (256 K per row)
constexpr int kPrStageSf = kPrBM * 16;          // 2 KB of e4m3 scales (NVFP4)
constexpr int kPrStaging = 16 * 64;             // one epilogue warp's 16 tokens x 32 columns of bf16
constexpr uint32_t kPrColA = kPrMaxBN;      // first TMEM column of the A stages
constexpr uint32_t kPrTmemCols = 512;

struct PairParams {
  float alpha;
  bf16* out;
  const bf16* resid;
  const uint8_t* sf_plain;   // MXFP4: e8m0 scales [N, K / 32]
  float* ws;                 // split-K partials [splits, T, N]
  uint32_t* counters;        // two per tile, zero at rest
  DeviceStatus* status;
  int T, N, K, ldc;
  int bn, m_tiles, units, splits, kb_per_split;
  int width;                 // columns of a tile's MMAs: bn, rounded up to a multiple of 32
  int preload;               // weights may be read before the preceding grid has finished
  int vec;                   // rows of `out` (and `resid`) can be accessed as 16-byte vectors
  // Grouped form (experts): the matrices are stacked along N ([experts * N, K], N a multiple of 256); token tile t holds rows
  // t * bn .. of x and `out` and belongs to matrix groups[t] (negative: nothing to do).  The block scales come in the
  // order of the block-scaled kernels (tile_scales: [128 rows][256 K][4 x 512 bytes]), with one factor per matrix.
  const int32_t* groups;
  const float* group_alpha;
  const uint8_t* sf_tiled;
  int n_tiles;
};

constexpr size_t pair_smem_bytes() {
  return 1024 + static_cast<size_t>(kPrStages) * kPrStageB + static_cast<size_t>(kPrSR) * (kPrStageRaw + kPrStageSf) +
         kPrEpiWarps * kPrStaging + (2 * kPrStages + 2 * kPrSR + 2) * 8 + 64;
}

// Arrive on a barrier of the pair's first CTA (`addr`: its shared::cluster address); CTA-scope release.
__device__ __forceinline__ void mbar_arrive_pair(uint32_t addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}

// One K = 64 block of a row: 32 packed bytes -> 32 words of two bf16 each, element 2j in the low half of word j, 2^-14 times
// the weight (the epilogue's factor makes up for it).  A code's three magnitude bits, moved to bits 8..6 of a bf16, read as
// value * 2^-126 (code 1, 0.5, as a subnormal); the bf16 scale carries 2^112.  With the code in the high nibble of a byte, one
// byte permute of (w << 4, w) puts the codes of both halves in place and spreads their signs over the bytes above
// (its sign-replicating selectors); a shift and a mask finish both.  The integer pipe, which has half the rate of the
// multiplier's, gets two instructions for two weights; the f16 conversion of the same codes took five and made it
// the kernel's bound (50 % busy at 840 cycles per block; 384 are the MMAs of a 192-token tile).
__device__ __forceinline__ void expand_e2m1x64(const Pack16& w0, const Pack16& w1, const bf162 (&s)[4], uint32_t (&o)[32]) {
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const uint32_t w = q < 4 ? w0.w[q] : w1.w[q - 4], we = w << 4;
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
      uint32_t x;   // (prmt itself: __byte_perm drops the replicate bit of a selector)
      asm("prmt.b32 %0, %1, %2, %3;" : "=r"(x) : "r"(we), "r"(w), "r"(j | (j + 8) << 4 | (j + 4) << 8 | (j + 12) << 12));
      const uint32_t r = (x << 2) & 0x81C081C0u;
      const bf162 v = __hmul2(*reinterpret_cast<const bf162*>(&r), s[q >> 1]);
      o[q * 4 + j] = *reinterpret_cast<const uint32_t*>(&v);
    }
  }
}

template <int WMODE, bool GROUPED>   // 1 = NVFP4, 3 = MXFP4
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPrThreads, 1)
gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap tmA,   // packed weights as bytes [N, K / 2], box 128 x 128
                    const __grid_constant__ CUtensorMap tmB,   // activations bf16 [T, K], box 64 x width / 2
                    const __grid_constant__ CUtensorMap tmSf,  // NVFP4 scales [N, K / 16], box 16 x 128
                    PairParams p) {
  extern __shared__ __align__(1024) unsigned char smem_dyn[];
  // (the pad to 1024 is the same in both CTAs of a pair: their windows have one layout)
  unsigned char* sp = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  unsigned char* sB = sp;    sp += kPrStages * kPrStageB;
  unsigned char* sRaw = sp;  sp += kPrSR * kPrStageRaw;
  unsigned char* sSf = sp;   sp += kPrSR * kPrStageSf;
  unsigned char* sOut = sp;  sp += kPrEpiWarps * kPrStaging;
  uint64_t* full = reinterpret_cast<uint64_t*>(sp);     // used in the first CTA: activation tiles and converter warps of both
  uint64_t* done = full + kPrStages;                    // the MMAs of the stage have completed
  uint64_t* raw_full = done + kPrStages;
  uint64_t* raw_empty = raw_full + kPrSR;
  uint64_t* acc_full = raw_empty + kPrSR;
  uint64_t* acc_empty = acc_full + 1;                   // used in the first CTA: the epilogue warps of each CTA
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* last_flag = const_cast<int*>(abort_flag) + 1;
  volatile int* epi_failed = last_flag + 1;             // an epilogue warp gave up (split K: read between two barriers of the unit)

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_ctarank());
  const int first_unit = static_cast<int>(blockIdx.x) >> 1, unit_step = static_cast<int>(gridDim.x) >> 1;
  const int num_kb = p.K / kPrBK;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kPrStages; ++i) { mbar_init(&full[i], 1 + 2 * 4); mbar_init(&done[i], 1); }
    for (int i = 0; i < kPrSR; ++i) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], 2 * 4); }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, 2 * kPrEpiWarps);
    *abort_flag = 0;
    *last_flag = 0;
    *epi_failed = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    if (WMODE == 1 && !GROUPED) tma_prefetch_desc(&tmSf);
  }
  if (warp == kPrMma) {
    tmem_alloc_pair(tmem_slot, kPrTmemCols);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_barrier();      // the other CTA's barriers exist before anything arrives on them from here
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // (in a captured pass no kernel writes weights: their first stages are requested in front of the wait)
  const bool preload = !GROUPED && p.preload;
  if (!preload || warp != kPrRaw) pdl_wait();

  // Unit u: k64 blocks [kb0, kb0 + nk), a multiple of four; first weight row (n0 in the tensor map, nc as a column of the output) and
  // first token of the tile.  False: nothing to do.
  auto unit_at = [&](int u, int& n0, int& nc, int& m0, int& split, int& kb0, int& nk, float& alpha) {
    alpha = p.alpha;
    if (GROUPED) {
      const int tile = u / p.n_tiles, e = p.groups[tile];
      nc = (u % p.n_tiles) * 2 * kPrBM + rank * kPrBM;
      n0 = e * p.N + nc;
      m0 = tile * p.bn;
      split = 0; kb0 = 0; nk = num_kb;
      if (e < 0) return false;
      alpha *= p.group_alpha[e];
      return true;
    }
    const int tile = u / p.splits;
    split = u % p.splits;
    n0 = nc = (tile / p.m_tiles) * 2 * kPrBM + rank * kPrBM;
    m0 = (tile % p.m_tiles) * p.bn;
    kb0 = split * p.kb_per_split;
    nk = min(p.kb_per_split, num_kb - kb0);
    return true;
  };

  if (warp == kPrRaw) {
    // ------------------------------------------------------------------ TMA producer of the weights (own rows), up to 1024 K ahead
    if (elect_one()) {
      bool ok = true, waited = !preload;
      int r = 0;
      for (int u = first_unit; u < p.units && ok; u += unit_step) {
        int n0, nc, m0, split, kb0, nk;
        float alpha;
        if (!unit_at(u, n0, nc, m0, split, kb0, nk, alpha)) continue;
        for (int i = 0; i < nk; i += 4, ++r) {
          const int sr = r % kPrSR, kb = kb0 + i;
          if (!waited && r == kPrSR) { pdl_wait(); waited = true; }
          if (!wait_bar(&raw_empty[sr], ((r / kPrSR) & 1) ^ 1)) { report(p.status, kTimeoutStageEmpty, 21); *abort_flag = 1; ok = false; break; }
          if (*abort_flag) { ok = false; break; }
          mbar_expect_tx(&raw_full[sr], kPrStageRaw + (WMODE == 1 ? kPrStageSf : 0));
          tma_load_2d(sRaw + sr * kPrStageRaw, &tmA, kb * 32, n0, &raw_full[sr]);
          if (GROUPED)
            bulk_load_1d(sSf + sr * kPrStageSf, p.sf_tiled + (static_cast<size_t>(n0 / kPrBM) * (p.K / 256) + (kb >> 2)) * kPrStageSf, kPrStageSf, &raw_full[sr]);
          else if (WMODE == 1) tma_load_2d(sSf + sr * kPrStageSf, &tmSf, kb * 4, n0, &raw_full[sr]);
        }
      }
      if (!waited) pdl_wait();
    }
  } else if (warp == kPrTma) {
    // ------------------------------------------------------------------ TMA producer of the activations (own token half)
    if (elect_one()) {
      const uint32_t stage_b = static_cast<uint32_t>(p.width / 2) * 128u;
      int stg = 0;
      bool ok = true;
      for (int u = first_unit; u < p.units && ok; u += unit_step) {
        int n0, nc, m0, split, kb0, nk;
        float alpha;
        if (!unit_at(u, n0, nc, m0, split, kb0, nk, alpha)) continue;
        const int mh = m0 + rank * (p.width / 2);
        for (int i = 0; i < nk; i += 2, ++stg) {
          const int sl = stg % kPrStages, kb = kb0 + i;
          if (!wait_bar(&done[sl], ((stg / kPrStages) & 1) ^ 1)) { report(p.status, kTimeoutStageEmpty, 22); *abort_flag = 1; ok = false; break; }
          if (rank == 0) mbar_expect_tx(&full[sl], 4 * stage_b);
          const uint32_t bar = mapa_shared(smem_u32(&full[sl]), 0u);
          tma_load_2d_pair(sB + sl * kPrStageB, &tmB, kb * kPrBK, mh, bar);
          tma_load_2d_pair(sB + sl * kPrStageB + kPrHalfB, &tmB, (kb + 1) * kPrBK, mh, bar);
        }
      }
    }
  } else if (warp == kPrMma) {
    // ------------------------------------------------------------------ MMA issuer of the pair
    // One thread, one wait per 128 K: this loop is the chain that the tensor pipe waits for.  A wait takes 200 cycles
    // even when its barrier completed long ago, so separate waits for activations and weights per 64 K made a loop
    // of 740 cycles, whatever the tile (MMAs of 64 K x 256 tokens: 544).
    if (rank == 0 && elect_one()) {
      const uint32_t idesc = umma_idesc_f16(2 * kPrBM, static_cast<uint32_t>(p.width), 1u, 1u);
      const uint32_t b_base = smem_u32(sB);
      int sl = 0, tc = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int u = first_unit; u < p.units && ok; u += unit_step) {
        int n0, nc, m0, split, kb0, nk;
        float alpha;
        if (!unit_at(u, n0, nc, m0, split, kb0, nk, alpha)) continue;
        if (!wait_bar(acc_empty, (tc & 1) ^ 1)) { report(p.status, kTimeoutAccum, 23); *abort_flag = 1; break; }
        for (int i = 0; i < nk; i += 2) {
          if (!wait_bar(&full[sl], ph)) { report(p.status, kTimeoutConvert, 24); *abort_flag = 1; ok = false; break; }
          tc_fence_after();
          const uint32_t b_addr = b_base + sl * kPrStageB, a_col = tmem_base + kPrColA + sl * 64;
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            umma_f16_pair_ts(tmem_base, a_col + kk * 8, umma_desc_sw128(b_addr + (kk >> 2) * kPrHalfB + (kk & 3) * 32), idesc,
                             (i > 0 || kk > 0) ? 1u : 0u);
          umma_commit_pair(&done[sl], 3);
          if (++sl == kPrStages) { sl = 0; ph ^= 1; }
        }
        umma_commit_pair(acc_full, 3);
        ++tc;
      }
    }
  } else if (warp >= kPrConv && warp < kPrEpi) {
    // ------------------------------------------------------------------ converters: e2m1 -> bf16 -> TMEM
    const int set = (warp - kPrConv) >> 2, q = warp & 3, row = q * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    const float k112 = 5.192296858534828e33f;
    int stg = 0;               // stages (128 K) of the units so far
    bool ok = true;
    for (int u = first_unit; u < p.units && ok; u += unit_step) {
      int n0, nc, m0, split, kb0, nk;
      float alpha;
      if (!unit_at(u, n0, nc, m0, split, kb0, nk, alpha)) continue;
      const int nstg = nk / 2;
      const int first = (set - stg) & (kPrStages - 1);      // this set's first stage of the unit
      // MXFP4: four scale bytes per stage by plain loads, one stage of this set ahead
      const uint8_t* sf_row = nullptr;
      uint32_t e8 = 0;
      if (WMODE == 3) {
        sf_row = p.sf_plain + static_cast<size_t>(min(n0 + row, p.N - 1)) * (p.K / 32) + kb0 * 2;
        if (first < nstg) e8 = *reinterpret_cast<const uint32_t*>(sf_row + first * 4);
      }
      for (int i = first; i < nstg; i += kPrStages) {
        const int at = stg + i, r = at >> 1, sr = r % kPrSR, half = at & 1;      // (units begin with a raw stage: both counts are even there)
        bool okw = wait_bar(&raw_full[sr], (r / kPrSR) & 1);
        const unsigned char* raw = sRaw + sr * kPrStageRaw + row * 128;
        Pack16 w[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) w[c].u = *reinterpret_cast<const uint4*>(raw + (((half * 4 + c) ^ (row & 7)) << 4));
        uint32_t four[2] = {0u, 0u};
        if (WMODE == 1) {
#pragma unroll
          for (int b = 0; b < 2; ++b)
            four[b] = *reinterpret_cast<const uint32_t*>(
                sSf + sr * kPrStageSf + (GROUPED ? (half * 2 + b) * 512 + lane * 16 + q * 4 : row * 16 + (half * 2 + b) * 4));
        }
        const uint32_t e8_now = e8;
        if (WMODE == 3 && i + kPrStages < nstg) e8 = *reinterpret_cast<const uint32_t*>(sf_row + (i + kPrStages) * 4);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          bf162 s[4];
          if (WMODE == 1) {
            const float2 lo = __half22float2(e4m3x2_to_h2(static_cast<uint16_t>(four[b] & 0xFFFFu)));
            const float2 hi = __half22float2(e4m3x2_to_h2(static_cast<uint16_t>(four[b] >> 16)));
            s[0] = __float2bfloat162_rn(lo.x * k112); s[1] = __float2bfloat162_rn(lo.y * k112);
            s[2] = __float2bfloat162_rn(hi.x * k112); s[3] = __float2bfloat162_rn(hi.y * k112);
          } else {
            const uint32_t e = e8_now >> (16 * b);
            s[0] = s[1] = __float2bfloat162_rn(e8m0_to_f32(static_cast<uint8_t>(e & 255u)) * k112);
            s[2] = s[3] = __float2bfloat162_rn(e8m0_to_f32(static_cast<uint8_t>((e >> 8) & 255u)) * k112);
          }
          uint32_t o[32];
          expand_e2m1x64(w[2 * b], w[2 * b + 1], s, o);
          if (b == 0) {
            __syncwarp();
            if (lane == 0) mbar_arrive(&raw_empty[sr]);   // this warp is done with its half of the raw stage
            if (okw) okw = wait_bar(&done[set], ((at / kPrStages) & 1) ^ 1);   // the stage's columns are free
            if (!okw) { report(p.status, kTimeoutTmaFull, 26); *abort_flag = 1; }
            ok = __all_sync(0xffffffffu, okw && !*abort_flag);
            if (!ok) break;
            tc_fence_after();
          }
          tmem_st_x32_async(tmem_base + kPrColA + set * 64 + b * 32 + lane_addr, o);
        }
        if (!ok) break;
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_pair(mapa_shared(smem_u32(&full[set]), 0u));
      }
      stg += nstg;
    }
  } else if (warp >= kPrEpi) {
    // ------------------------------------------------------------------ epilogue: own 128 rows x bn tokens
    const int q = warp & 3;
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    const int half = (warp - kPrEpi) >> 2;
    bf16* stage = reinterpret_cast<bf16*>(sOut + (warp - kPrEpi) * kPrStaging);
    // Counts this CTA in at its half tile; true, and the counter back at zero, for the last of the splits.
    auto count_in = [&](int u) {
      uint32_t* counter = p.counters + (u / p.splits) * 2 + rank;
      const bool last = atomicAdd(counter, 1u) == static_cast<uint32_t>(p.splits - 1);
      if (last) *counter = 0;
      return last;
    };
    int tc = 0;
    bool dead = false;      // split K: a warp gave up; the remaining units only count themselves in (the counters end at zero)
    for (int u = first_unit; u < p.units; u += unit_step) {
      int n0, nc, m0, split, kb0, nk;
      float alpha;
      if (!unit_at(u, n0, nc, m0, split, kb0, nk, alpha)) continue;
      if (dead) {
        if (warp == kPrEpi && lane == 0) count_in(u);
        continue;
      }
      const uint32_t d = tmem_base + lane_addr;
      bool ok = wait_bar(acc_full, tc & 1);
      if (!ok) { report(p.status, kTimeoutAccum, 27); *abort_flag = 1; }
      ok = __all_sync(0xffffffffu, ok && !*abort_flag);
      tc_fence_after();
      const int nw = nc + q * 32, n = nw + lane;   // this warp's first column, this lane's
      const int cols = min(p.bn, p.T - m0);
      float* wsp = p.splits > 1 ? p.ws + (static_cast<size_t>(split) * p.T + m0) * p.N : nullptr;
      if (ok) {
#pragma unroll 1
        for (int c0 = half * 16; c0 < cols; c0 += 32) {
          uint32_t r[16];
          tmem_ld_x16(d + c0, r);
          const int live = min(16, cols - c0);
          if (p.splits > 1) {
            if (n < p.N) {
#pragma unroll
              for (int j = 0; j < 16; ++j)
                if (j < live) wsp[static_cast<size_t>(c0 + j) * p.N + n] = __uint_as_float(r[j]);
            }
          } else if (p.vec) {
            // turned around through the warp's staging tile: every lane then writes 8 columns of one token
#pragma unroll
            for (int j = 0; j < 16; ++j) stage[j * 32 + lane] = f32_to_bf16(__uint_as_float(r[j]) * alpha);
            __syncwarp();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int m = h * 8 + (lane >> 2), seg = lane & 3;
              if (m < live && nw + seg * 8 < p.N) {
                Pack16 v;
                v.u = *reinterpret_cast<const uint4*>(stage + m * 32 + seg * 8);
                const size_t at = static_cast<size_t>(m0 + c0 + m) * p.ldc + nw + seg * 8;
                if (p.resid) {
                  Pack16 x;
                  x.u = *reinterpret_cast<const uint4*>(p.resid + at);
#pragma unroll
                  for (int j = 0; j < 8; ++j) v.h[j] = f32_to_bf16(bf16_to_f32(x.h[j]) + bf16_to_f32(v.h[j]));
                }
                *reinterpret_cast<uint4*>(p.out + at) = v.u;
              }
            }
            __syncwarp();
          } else if (n < p.N) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              if (j < live) {
                const size_t at = static_cast<size_t>(m0 + c0 + j) * p.ldc + n;
                float y = __uint_as_float(r[j]) * alpha;
                if (p.resid) y = bf16_to_f32(p.resid[at]) + bf16_to_f32(f32_to_bf16(y));
                p.out[at] = f32_to_bf16(y);
              }
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_pair(mapa_shared(smem_u32(acc_empty), 0u));
      if (p.splits > 1) {
        // publish the partials; the last CTA on this half tile adds them in ascending split order.  The eight warps leave the
        // barriers of a unit together: what one of them gave up on is known to all behind the first (nobody writes it
        // again before the second), and all go on without waiting.
        __threadfence();
        if (!ok && lane == 0) *epi_failed = 1;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        dead = *epi_failed != 0;
        if (warp == kPrEpi && lane == 0) *last_flag = count_in(u) ? 1 : 0;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (dead) continue;
        if (*last_flag) {
          __threadfence();
          if (p.vec) {
            // a warp takes whole rows of the half tile, four columns per lane, four rows' partials in flight
            const int n4 = nc + lane * 4, wrow = warp - kPrEpi;
            if (n4 < p.N) {
              for (int mb = wrow; mb < cols; mb += 4 * kPrEpiWarps) {
                float4 acc[4];
#pragma unroll
                for (int mm = 0; mm < 4; ++mm) acc[mm] = make_float4(0.f, 0.f, 0.f, 0.f);
                for (int s0 = 0; s0 < p.splits; ++s0) {
                  float4 t[4];
#pragma unroll
                  for (int mm = 0; mm < 4; ++mm)
                    t[mm] = mb + mm * kPrEpiWarps < cols
                                ? __ldcg(reinterpret_cast<const float4*>(p.ws + (static_cast<size_t>(s0) * p.T + m0 + mb + mm * kPrEpiWarps) * p.N + n4))
                                : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                  for (int mm = 0; mm < 4; ++mm) { acc[mm].x += t[mm].x; acc[mm].y += t[mm].y; acc[mm].z += t[mm].z; acc[mm].w += t[mm].w; }
                }
#pragma unroll
                for (int mm = 0; mm < 4; ++mm) {
                  const int m = mb + mm * kPrEpiWarps;
                  if (m >= cols) break;
                  const size_t at = static_cast<size_t>(m0 + m) * p.ldc + n4;
                  float y[4] = {acc[mm].x * alpha, acc[mm].y * alpha, acc[mm].z * alpha, acc[mm].w * alpha};
                  union { uint2 u; bf16 h[4]; } v, x;
                  if (p.resid) x.u = *reinterpret_cast<const uint2*>(p.resid + at);
#pragma unroll
                  for (int j = 0; j < 4; ++j) {
                    v.h[j] = f32_to_bf16(y[j]);
                    if (p.resid) v.h[j] = f32_to_bf16(bf16_to_f32(x.h[j]) + bf16_to_f32(v.h[j]));
                  }
                  *reinterpret_cast<uint2*>(p.out + at) = v.u;
                }
              }
            }
          } else if (n < p.N) {
            for (int m = half; m < cols; m += 2) {
              float acc = 0.f;
              for (int s0 = 0; s0 < p.splits; ++s0) acc += __ldcg(p.ws + (static_cast<size_t>(s0) * p.T + m0 + m) * p.N + n);
              const size_t at = static_cast<size_t>(m0 + m) * p.ldc + n;
              float y = acc * alpha;
              if (p.resid) y = bf16_to_f32(p.resid[at]) + bf16_to_f32(f32_to_bf16(y));
              p.out[at] = f32_to_bf16(y);
            }
          }
        }
      }
      if (!ok) break;      // (unsplit: the warps share no barrier)
      ++tc;
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_barrier();      // neither CTA leaves (or frees TMEM) while the other may still read its memory or arrive there
  if (warp == kPrMma) tmem_dealloc_pair(tmem_base, kPrTmemCols);
}

// Pairs that fit the device at once (one per TPC; a GPC with an odd number of SMs in use gives one less).
template <int WMODE, bool GROUPED>
static int pair_slots(int* slots) {
  static int cached = 0;
  if (!cached) {
    auto kern = gemm_tc_pair_kernel<WMODE, GROUPED>;
    constexpr size_t smem = pair_smem_bytes();
    static_assert(kPrSets == kPrStages && (kPrStages & (kPrStages - 1)) == 0, "a set has one stage of the ring");
    static_assert(smem <= 227 * 1024, "shared memory budget exceeded");
    DGPP_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2, 1, 1);
    cfg.blockDim = dim3(kPrThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    DGPP_CUDA_OK(cudaOccupancyMaxActiveClusters(&n, kern, &cfg));
    DGPP_REQUIRE(n >= 1, "gemm_tc_pair: no CTA pair fits this device");
    cached = n;
  }
  *slots = cached;
  return 0;
}

// Token tile and K splits of one product.  The product takes as many units one after the other as one pair gets: wide tiles reuse a
// converted weight more often, narrower ones (or splits, where there are fewer tiles than pairs) fill the last round.  A K = 64
// block counts as 345 cycles (the conversion) or 80 + 1.95 bn (the MMAs), whichever is more, a tile's drain and the next one's fill as
// 15 bn + 1500 (the accumulator is not double-buffered: its other half holds the converted weights), s splits as 1000 and 400 s for every
// 32 tokens of a tile (their fold is s round trips to L2).  Fitted to six shapes of 4096 x 2048 to 34816 x 5120 at 129 to 2048 rows with every
// tile: what they choose is within 0.2 % of the best on average, 4 % at most (34816 x 5120 at 953 rows: 276 us at 256 tokens, which 400 + 1.2 bn
// chose, 230 at 192).
// Up to 128 rows the splits are those of 128 rows (seven shapes of 512 x 512 to 34816 x 5120 at 8, 37, 64 and 128 rows against every tile
// and split count: within 4 % of the best, but for 2560 x 8192 at 8 rows, 15.8 us, 14.7 in six splits instead of three, and
// 4096 x 2048 at 128, 12.8, 11.5 without splits), above there are none: on either side of that line a row's bits do not depend
// on how many others share its pass, and prompt products touch no workspace, so that products on several streams share
// nothing.  (A long K over few tiles pays for that: 173 x 5120 x 17408 79 us, 47 in three splits.)
constexpr int kPrSplitRows = 128;

// Cheapest tile and split count for T rows, splits between `fewest` and `most`.
static void pair_search(int T, int N, int K, int slots, int fewest, int most, int* bn_out, int* splits_out) {
  double best = 0;
  const int nt = dgpp_ceil_div(N, 2 * kPrBM), raws = K / 256;
  for (int bn = kPrMaxBN; bn >= 32; bn -= 32) {
    if (bn < kPrMaxBN && bn - 32 >= T) continue;          // a smaller tile holds all rows
    const int tiles = nt * dgpp_ceil_div(T, bn);
    for (int s = fewest; s <= most && s <= raws; ++s) {
      const int per = dgpp_ceil_div(raws, s);
      if (dgpp_ceil_div(raws, per) != s) continue;
      const int rounds = dgpp_ceil_div(tiles * s, slots);
      const double block = 80 + 1.95 * bn;
      const double unit = per * 4 * (block < 345 ? 345 : block) + 15.0 * bn + 1500;
      const double cost = rounds * unit + (s > 1 ? 1000 + 400.0 * s * dgpp_ceil_div(bn < T ? bn : T, 32) : 0.0);
      if (best == 0 || cost < best) { best = cost; *bn_out = bn; *splits_out = s; }
    }
  }
}

static void pair_shape(int T, int N, int K, int slots, int max_splits, int* bn_out, int* splits_out) {
  *bn_out = kPrMaxBN;
  *splits_out = 1;
  if (T <= kPrSplitRows) pair_search(kPrSplitRows, N, K, slots, 1, max_splits, bn_out, splits_out);
  pair_search(T, N, K, slots, *splits_out, *splits_out, bn_out, splits_out);
}

template <int WMODE, bool GROUPED>
static int launch_pair(const CUtensorMap& tA, const CUtensorMap& tB, const CUtensorMap& tSf, PairParams& p, int slots, cudaStream_t st) {
  p.preload = stream_captures(st);
  const int pairs = p.units < slots ? p.units : slots;
  DGPP_CUDA_OK(launch_early(gemm_tc_pair_kernel<WMODE, GROUPED>, 2 * pairs, kPrThreads, pair_smem_bytes(), st, tA, tB, tSf, p));
  DGPP_CUDA_OK(cudaGetLastError());
  return 0;
}

}  // namespace dgpp

using namespace dgpp;

// wmode: 1 nvfp4 (w_scale = e4m3 scales [N, K / 16]), 3 mxfp4 (w_scale = e8m0 scales [N, K / 32]).  K % 256 == 0.
// out bf16 [T, ldc]; resid optional (out = bf16(resid + bf16(alpha * acc))).  bn: token tile, a multiple of 16 up to
// 256, or 0 = chosen here; splits: K splits, or 0 = chosen here (none above 128 rows) among those that the workspace (ws_floats fp32
// values, n_counters counters that are zero at rest) holds for 128 rows.
DGPP_API int dgpp_gemm_tc_pair(int wmode, const void* x, int64_t x_stride, const void* w, const void* w_scale, float alpha,
                               void* out, const void* resid, int ldc, int T, int N, int K, int bn, int splits, void* ws,
                               int64_t ws_floats, void* counters, int n_counters, cudaStream_t st) {
  DGPP_REQUIRE(wmode == 1 || wmode == 3, "gemm_tc_pair: 4-bit weights only (wmode %d)", wmode);
  DGPP_REQUIRE(T >= 1 && N >= 1, "gemm_tc_pair: empty problem");
  DGPP_REQUIRE(K % 256 == 0 && K > 0, "gemm_tc_pair: K %d must be a multiple of 256", K);
  DGPP_REQUIRE(out != nullptr && w_scale != nullptr, "gemm_tc_pair: output and scales required");
  DGPP_REQUIRE(bn >= 0 && bn <= kPrMaxBN && bn % 16 == 0, "gemm_tc_pair: token tile %d (a multiple of 16 up to %d)", bn, kPrMaxBN);
  DGPP_REQUIRE(splits >= 0 && (splits <= 1 || (ws && counters)), "gemm_tc_pair: split-K needs a workspace with counters");
  DGPP_REQUIRE((reinterpret_cast<uintptr_t>(w_scale) & 15) == 0, "gemm_tc_pair: scales must be 16-byte aligned");
  int slots = 0;
  if (wmode == 1 ? pair_slots<1, false>(&slots) : pair_slots<3, false>(&slots)) return -1;
  int most = 1;
  if (ws && counters) {
    const int room = T < kPrSplitRows ? kPrSplitRows : T;      // (rows: the same limit for every T that has splits)
    const int64_t by_ws = ws_floats / (static_cast<int64_t>(room) * N);
    most = static_cast<int>(by_ws < 8 ? (by_ws < 1 ? 1 : by_ws) : 8);
    if (2LL * dgpp_ceil_div(N, 2 * kPrBM) * dgpp_ceil_div(room, 16) > n_counters) most = 1;
  }
  int pick_bn, pick_splits;
  pair_shape(T, N, K, slots, most, &pick_bn, &pick_splits);
  if (bn == 0) bn = pick_bn;
  if (splits == 0) splits = pick_splits;
  DGPP_REQUIRE(splits == 1 || (splits <= 8 && static_cast<int64_t>(splits) * T * N <= ws_floats &&
                               2LL * dgpp_ceil_div(N, 2 * kPrBM) * dgpp_ceil_div(T, bn) <= n_counters),
               "gemm_tc_pair: %d splits do not fit the workspace", splits);
  PairParams p;
  p.alpha = alpha * 16384.f;    // the converted weights carry 2^-14
  p.out = static_cast<bf16*>(out);
  p.resid = static_cast<const bf16*>(resid);
  p.sf_plain = wmode == 3 ? static_cast<const uint8_t*>(w_scale) : nullptr;
  p.ws = static_cast<float*>(ws);
  p.counters = static_cast<uint32_t*>(counters);
  p.status = device_status_ptr();
  p.T = T; p.N = N; p.K = K; p.ldc = ldc;
  p.groups = nullptr; p.group_alpha = nullptr; p.sf_tiled = nullptr; p.n_tiles = 0;
  p.bn = bn;
  p.width = dgpp_ceil_div(bn, 32) * 32;
  p.m_tiles = dgpp_ceil_div(T, bn);
  const int raws = K / 256, per = dgpp_ceil_div(raws, splits);
  p.kb_per_split = per * 4;
  p.splits = dgpp_ceil_div(raws, per);
  p.units = p.m_tiles * dgpp_ceil_div(N, 2 * kPrBM) * p.splits;
  p.vec = N % 8 == 0 && ldc % 8 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0 && (reinterpret_cast<uintptr_t>(resid) & 15) == 0 &&
          (reinterpret_cast<uintptr_t>(ws) & 15) == 0;
  CUtensorMap tA, tB, tSf;
  memset(&tSf, 0, sizeof(tSf));
  if (make_tmap_2d(&tB, x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, K, T, x_stride * 2, 64, p.width / 2, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
  if (make_tmap_2d(&tA, w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, K / 2, N, K / 2, 128, kPrBM, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
  if (wmode == 1 &&
      make_tmap_2d(&tSf, w_scale, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, K / 16, N, K / 16, 16, kPrBM, CU_TENSOR_MAP_SWIZZLE_NONE))
    return -1;
  return wmode == 1 ? launch_pair<1, false>(tA, tB, tSf, p, slots, st) : launch_pair<3, false>(tA, tB, tSf, p, slots, st);
}

// Grouped linear over a stack of NVFP4 matrices w [experts * N, K / 2] with block scales in tile_scales order and one factor per matrix
// (group_alpha [experts]): rows t * bn .. of out = those of x times matrix groups[t]; tiles with a negative entry are
// left alone.  N and K multiples of 256, bn a multiple of 16 up to 256; x and out hold tiles * bn rows.
DGPP_API int dgpp_gemm_tc_pair_grouped(const void* x, int64_t x_stride, const void* w, const void* sf_tiled, const void* group_alpha,
                                       const void* groups, void* out, int ldc, int tiles, int N, int K, int experts, int bn,
                                       cudaStream_t st) {
  DGPP_REQUIRE(N > 0 && N % 256 == 0 && K > 0 && K % 256 == 0, "gemm_tc_pair_grouped: N %d and K %d must be multiples of 256", N, K);
  DGPP_REQUIRE(bn >= 16 && bn <= kPrMaxBN && bn % 16 == 0, "gemm_tc_pair_grouped: token tile %d", bn);
  DGPP_REQUIRE(tiles >= 1 && experts >= 1 && groups && group_alpha && sf_tiled && out, "gemm_tc_pair_grouped: bad group arguments");
  DGPP_REQUIRE((reinterpret_cast<uintptr_t>(sf_tiled) & 15) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0 && ldc % 8 == 0,
               "gemm_tc_pair_grouped: scales and output rows must be 16-byte aligned");
  int slots = 0;
  if (pair_slots<1, true>(&slots)) return -1;
  PairParams p;
  memset(&p, 0, sizeof(p));
  p.alpha = 16384.f;             // the converted weights carry 2^-14
  p.out = static_cast<bf16*>(out);
  p.status = device_status_ptr();
  p.T = tiles * bn; p.N = N; p.K = K; p.ldc = ldc;
  p.bn = bn; p.width = dgpp_ceil_div(bn, 32) * 32; p.m_tiles = tiles; p.splits = 1; p.kb_per_split = K / kPrBK;
  p.n_tiles = N / (2 * kPrBM);
  p.units = tiles * p.n_tiles;
  p.vec = 1;
  p.groups = static_cast<const int32_t*>(groups);
  p.group_alpha = static_cast<const float*>(group_alpha);
  p.sf_tiled = static_cast<const uint8_t*>(sf_tiled);
  CUtensorMap tA, tB, tSf;
  memset(&tSf, 0, sizeof(tSf));
  if (make_tmap_2d(&tB, x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, K, static_cast<uint64_t>(tiles) * bn, x_stride * 2, 64, p.width / 2, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
  if (make_tmap_2d(&tA, w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, K / 2, static_cast<uint64_t>(experts) * N, K / 2, 128, kPrBM, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
  return launch_pair<1, true>(tA, tB, tSf, p, slots, st);
}
