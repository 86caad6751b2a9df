// Causal flash attention for prefill over the paged FP8 KV cache, on tcgen05 (kind::f16).
//
// Work comes in units of one query head x 128 consecutive query positions.  A CTA takes two units of one KV head (the units of a KV
// head are numbered longest span first, heads fastest), or one where that already occupies the device.  K / V tiles of 128 tokens
// come from the cache pages by TMA as stored (e4m3 bytes) and are expanded once per CTA to f16:
//
//   K16[t, d] = f16(K[t, d] * k_scale[t]) / 2^ck       ck, cv: exponents of the largest scales up to this tile; the products are
//   V16[t, d] = f16(V[t, d] * v_scale[t]) / 2^cv       rounded once to 11 bits (the scale's mantissa in two f16 terms)
//   MMA1   S[q, t]  = Q16[q, d] . K16[t, d]^T          Q16 = q / 2^e of its row, exact down to 2^-22 of the row's largest
//   softmax (one thread per query row): s = S * sm * 2^ck, p = 2^(s - m), causal mask, P as f16 over the scores' own columns
//   MMA2   O[q, d] += P[q, t] . V16[t, d]              P is the A operand in tensor memory, V the B operand read MN-major
//
// O stays in tensor memory, in units of 2^cv.  m is a row's reference, not its maximum: it moves only when a tile exceeds it by more
// than 2^8 (f16 and the fp32 sums have the range for that; the lazily moved maximum is a published method of flash attention on this
// chip), so the accumulator is rescaled a few times per row, and when cv grows, instead of once per tile.  Whether m moves depends
// on the row alone, and ck, cv are powers of two; what ties a row's bits to tokens it does not see is f16's range alone: elements of
// K and V below 2^-14 of the largest scale's power of two are held to 2^-25 of it.  Tokens whose row is zero (their scale is a
// placeholder) do not count for the exponents.
//
// Two units: the tensor core works for one while the other's threads exponentiate (S of unit u is rewritten right behind its PV
// product).  One unit: two score buffers, S of tile i + 1 runs under the softmax of tile i.
// Warps: 0..3 / 4..7 softmax of the units (TMEM lane quadrant = warp % 4), 8..11 expand K, 12..15 expand V (thread = token),
// 16 TMA producer, 17 MMA issuer and TMEM owner.
// What bounds it: MUFU and tensor pipe alike (a tile of two units: 2048 cycles each), then the handshakes between them.
// 40 query and 8 KV heads, with two e4m3 terms of q and P, one unit per CTA and the accumulator in registers / so: 173 rows behind 3000
// 92 / 61 us, 2048 rows 172 / 106, 2048 rows behind 6144 944 / 547 (the scales' mantissas, powers of two and zero rows are 5 % of that).
// (reference counterparts: src/kernels/full_attn.cu:442,679,983 tile / TMA / fp8-compute prefill kernels.)
#include <cuda.h>
#include <math.h>
#include <string.h>

#include "common/common.h"
#include "common/dtypes.cuh"
#include "common/ptx.cuh"
#include "kernels/gemm_common.cuh"

namespace dgpp {

constexpr int kApTile = 128;
constexpr int kApConv = 8, kApTma = 16, kApMma = 17;     // first warp of each role behind the softmax warps
constexpr int kApThreads = 18 * 32;
constexpr int kApRing = 4, kApRaw = 2;                   // f16 tiles (K in the even slots, V in the odd ones), tiles as stored
constexpr int kApRawBytes = kApTile * 128;               // 16 KB
constexpr int kApBlk = kApTile * 128;                    // 16 KB: 64 columns of an f16 tile
constexpr int kApF16Bytes = 2 * kApBlk;
constexpr float kApSlack = 8.f;                          // a row's reference may lag its maximum by this power of two

struct AttnPrefillParams {
  const bf16* q;            // [T, q_stride]: head h at column h * 128 (already rotated)
  int64_t q_stride;
  const float* k_scale;     // [blocks, hkv, page]
  const float* v_scale;
  const int32_t* block_table;  // row of this request
  bf16* out;                // [T, hq * 128]
  DeviceStatus* status;
  int T, pos0, hq, hkv, page, max_blocks, window;
  int units, per_cta;       // units of a KV head, units of a CTA (1 or 2)
  float scale;
};

constexpr size_t attn_prefill_smem_bytes() {
  return 1024 + 2 * kApF16Bytes + kApRing * kApF16Bytes + kApRaw * (kApRawBytes + kApTile * 4) + 24 * 4 +
         (2 * kApRing + 2 * kApRaw + 6) * 8 + 16;
}

__device__ __forceinline__ float exp2_of(int e) { return __uint_as_float(static_cast<uint32_t>(e + 127) << 23); }   // -126 <= e <= 127

// (lo, hi) of a pair of packed fp32 values: one instruction for two lanes of arithmetic.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, z, w;\n\t"
      "mov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
      "fma.rn.f32x2 w, x, y, z;\n\tmov.b64 {%0, %1}, w;\n\t}\n"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, w;\n\t"
      "mov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
      "add.rn.f32x2 w, x, y;\n\tmov.b64 {%0, %1}, w;\n\t}\n"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
// 32 scores of a row from tensor memory, tokens t0 .. t0 + 31; those the row does not see become -inf.
template <bool kMask>
__device__ __forceinline__ void scores_x32(uint32_t taddr, int t0, int my_pos, int my_first, uint32_t (&s)[32]) {
  tmem_ld_x32(taddr, s);
  if (kMask) {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (t0 + j > my_pos || t0 + j < my_first) s[j] = 0xff800000u;
  }
}
__device__ __forceinline__ float max_x32(const uint32_t (&s)[32], float m) {
  float m4[4] = {m, -INFINITY, -INFINITY, -INFINITY};      // (four chains)
#pragma unroll
  for (int j = 0; j < 32; j += 8)
#pragma unroll
    for (int c = 0; c < 4; ++c) m4[c] = fmaxf(fmaxf(m4[c], __uint_as_float(s[j + c])), __uint_as_float(s[j + 4 + c]));
  return fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
}
// Probabilities 2^(s * sm + off) of 32 scores as 16 words of the A operand at `paddr`; their sum is added to `sum`.
__device__ __forceinline__ void probs_x32(const uint32_t (&s)[32], float sm, float off, uint32_t paddr, float2 (&sum)[2]) {
  uint32_t o[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    float2 e = fma2(make_float2(__uint_as_float(s[2 * j]), __uint_as_float(s[2 * j + 1])), make_float2(sm, sm), make_float2(off, off));
    e.x = fast_exp2(e.x);
    e.y = fast_exp2(e.y);
    sum[j & 1] = add2(sum[j & 1], e);
    const __half2 h = __floats2half2_rn(e.x, e.y);
    o[j] = *reinterpret_cast<const uint32_t*>(&h);
  }
  tmem_st_x16_async(paddr, o);
}

// Scores of one tile -> probabilities.  Tokens 64..127 stay in registers between the two passes; the P operand takes over their
// columns (64 words at column 64), tokens 0..63 are read again.  `ref` is the row's reference m, `lsum` its probability mass in
// units of 2^m; `rescale(corr)` multiplies the accumulator (called by all lanes of a warp or by none; `regrow`: in any case).
template <bool kMask, class Rescale>
__device__ __forceinline__ void softmax_tile(uint32_t ts, int t0, int my_pos, int my_first, float sm, bool regrow, float& ref,
                                             float& lsum, Rescale rescale) {
  uint32_t a[32], b[32], c[32];
  scores_x32<kMask>(ts, t0, my_pos, my_first, a);
  float mt = max_x32(a, -INFINITY);
  scores_x32<kMask>(ts + 32, t0 + 32, my_pos, my_first, a);
  mt = max_x32(a, mt);
  scores_x32<kMask>(ts + 64, t0 + 64, my_pos, my_first, b);
  mt = max_x32(b, mt);
  scores_x32<kMask>(ts + 96, t0 + 96, my_pos, my_first, c);
  mt = max_x32(c, mt);
  const float top = mt * sm;                   // sm > 0
  const bool move = top > ref + kApSlack;      // (the first tile with a visible token: ref = -inf)
  if (__any_sync(0xffffffffu, move) || regrow) {
    const float next = move ? top : ref;
    const float corr = (move && ref != -INFINITY) ? fast_exp2(ref - next) : 1.f;
    ref = next;
    lsum *= corr;
    rescale(corr);
  }
  const float off = ref == -INFINITY ? 0.f : -ref;
  float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
  probs_x32(b, sm, off, ts + 96, sum);
  probs_x32(c, sm, off, ts + 112, sum);
  scores_x32<kMask>(ts, t0, my_pos, my_first, a);
  probs_x32(a, sm, off, ts + 64, sum);
  scores_x32<kMask>(ts + 32, t0 + 32, my_pos, my_first, a);
  probs_x32(a, sm, off, ts + 80, sum);
  lsum += (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
  tmem_st_wait();
}

__global__ void __launch_bounds__(kApThreads, 1)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                       AttnPrefillParams p) {
  constexpr int D = 128;
  extern __shared__ __align__(1024) unsigned char smem_dyn[];
  unsigned char* sp = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  unsigned char* sQ = sp;    sp += 2 * kApF16Bytes;
  unsigned char* sRing = sp; sp += kApRing * kApF16Bytes;
  unsigned char* sRaw = sp;  sp += kApRaw * kApRawBytes;
  float* sScale = reinterpret_cast<float*>(sp);  sp += kApRaw * kApTile * sizeof(float);
  int* sExp = reinterpret_cast<int*>(sp);        sp += 2 * 4 * sizeof(int);        // [K, V][tile & 3] exponents ck, cv
  int* sMax = reinterpret_cast<int*>(sp);        sp += 2 * 2 * 4 * sizeof(int);    // [K, V][tile & 1][warp] largest exponent of a warp's scales
  uint64_t* raw_full = reinterpret_cast<uint64_t*>(sp);
  uint64_t* raw_empty = raw_full + kApRaw;
  uint64_t* ring_full = raw_empty + kApRaw;
  uint64_t* ring_empty = ring_full + kApRing;
  uint64_t* s_full = ring_empty + kApRing;   // [2] per score buffer
  uint64_t* p_full = s_full + 2;             // [2] per score buffer
  uint64_t* o_full = p_full + 2;             // [2] per unit
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = p.hq / p.hkv, kvh = blockIdx.x % p.hkv;
  const int unit0 = static_cast<int>(blockIdx.x) / p.hkv * p.per_cta;
  const bool dual = p.per_cta == 2;
  const int row_tiles = p.units / group;
  // unit u of this KV head: query head, first row; tiles are counted from the first that any of the CTA's rows sees
  auto unit_row = [&](int u) { return (row_tiles - 1 - u / group) * kApTile; };
  const int low_row = unit_row(min(unit0 + p.per_cta - 1, p.units - 1));
  const int low_pos = p.pos0 + low_row;
  const int first_tok = (p.window > 0 && low_pos + 1 > p.window) ? low_pos + 1 - p.window : 0;
  const int base = first_tok & ~(kApTile - 1);
  auto unit_last = [&](int u) { return p.pos0 + min(unit_row(u) + kApTile, p.T) - 1; };
  auto unit_tiles = [&](int u) { return u < p.units ? (unit_last(u) + kApTile - base) / kApTile : 0; };
  const int n0 = unit_tiles(unit0), n1 = dual ? unit_tiles(unit0 + 1) : 0;       // n0 >= n1, n0 >= 1
  const int last_pos = unit_last(unit0);

  if (threadIdx.x == 0) {
    for (int i = 0; i < kApRaw; ++i) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], 4); }
    for (int i = 0; i < kApRing; ++i) { mbar_init(&ring_full[i], 4); mbar_init(&ring_empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 4); mbar_init(&o_full[i], 1); }
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == kApMma) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();      // the barriers are there, and the columns this CTA's before the next grid is let in
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;      // score buffers at columns 0 and 128, accumulators at 256 and 384
  pdl_wait();
  // ---- the units' query rows as f16 (thread = row): scaled by a power of two to a largest magnitude of 128..256
  const int sub = warp >> 2;
  float q_scale = 1.f;
  if (warp < kApConv && (sub == 0 || n1 > 0)) {
    const int r = (warp & 3) * 32 + lane, row = unit_row(unit0 + sub) + r;
    const int head = kvh * group + (unit0 + sub) % group;
    const uint4* src = reinterpret_cast<const uint4*>(p.q + static_cast<size_t>(row) * p.q_stride + head * D);
    const bool live = row < p.T;
    float amax = 0.f;
    Pack16 x[D / 8];
#pragma unroll
    for (int c = 0; c < D / 8; ++c) x[c].u = live ? src[c] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int c = 0; c < D / 8; ++c)
#pragma unroll
      for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(bf16_to_f32(x[c].h[j])));
    const int e = max(static_cast<int>((__float_as_uint(amax) >> 23) & 255u), 8);      // biased exponent of the largest
    const float mul = __uint_as_float(static_cast<uint32_t>(261 - e) << 23);
    q_scale = __uint_as_float(static_cast<uint32_t>(e - 7) << 23);
#pragma unroll
    for (int c = 0; c < D / 8; ++c) {
      Pack16 y;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const __half2 h = __floats2half2_rn(bf16_to_f32(x[c].h[2 * j]) * mul, bf16_to_f32(x[c].h[2 * j + 1]) * mul);
        y.w[j] = *reinterpret_cast<const uint32_t*>(&h);
      }
      *reinterpret_cast<uint4*>(sQ + sub * kApF16Bytes + (c >> 3) * kApBlk + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = y.u;
    }
    fence_proxy_async_smem();
  }
  // (K and V are on their way and being expanded meanwhile: only the softmax warps and the MMA issuer meet here)
  if (warp < kApConv || warp == kApMma) asm volatile("bar.sync 3, 288;" ::: "memory");

  if (warp == kApTma) {
    // ------------------------------------------------------------------ TMA producer: K0, V0, K1, V1, ...
    if (elect_one()) {
      const int ppt = kApTile / p.page, last_page = min(last_pos / p.page, p.max_blocks - 1);
      bool ok = true;
      for (int i = 0; i < n0 && ok; ++i) {
        const int page0 = (base + i * kApTile) / p.page;
        for (int v = 0; v < 2; ++v) {      // item 2 i + v, raw slot v
          if (!wait_bar(&raw_empty[v], (i & 1) ^ 1)) { report(p.status, kTimeoutStageEmpty, 31); *abort_flag = 1; ok = false; break; }
          mbar_expect_tx(&raw_full[v], kApRawBytes + kApTile * sizeof(float));
          for (int pg = 0; pg < ppt; ++pg) {
            const int r0 = (p.block_table[min(page0 + pg, last_page)] * p.hkv + kvh) * p.page;
            tma_load_2d(sRaw + v * kApRawBytes + pg * p.page * D, v ? &tmV : &tmK, 0, r0, &raw_full[v]);
            bulk_load_1d(sScale + v * kApTile + pg * p.page, (v ? p.v_scale : p.k_scale) + r0, p.page * sizeof(float), &raw_full[v]);
          }
        }
        if (*abort_flag) break;
      }
    }
  } else if (warp == kApMma) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      constexpr uint32_t idesc1 = umma_idesc_f16(128, 128, 0u, 0u);                 // Q (K-major) x K (K-major)
      constexpr uint32_t idesc2 = umma_idesc_f16(128, 128, 0u, 0u) | (1u << 16);    // P (tensor memory) x V (MN-major B)
      const uint32_t q_addr = smem_u32(sQ), ring = smem_u32(sRing);
      bool ok = true;
      auto wait = [&](uint64_t* bar, uint32_t parity, int code, int detail) {
        if (!ok) return;
        if (!wait_bar(bar, parity) || *abort_flag) { report(p.status, code, detail); *abort_flag = 1; ok = false; }
        tc_fence_after();
      };
      // item j of the ring: slot j % 4, phase j / 4; tile i's K is item 2 i, its V item 2 i + 1
      auto wait_item = [&](int j) { wait(&ring_full[j & 3], (j >> 2) & 1, kTimeoutTmaFull, 32); };
      auto scores = [&](int u, int buf, int i) {
        const uint32_t k_addr = ring + ((2 * i) & 3) * kApF16Bytes, a_addr = q_addr + u * kApF16Bytes;
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_f16(tmem_base + buf * 128, umma_desc_sw128(a_addr + (k >> 2) * kApBlk + (k & 3) * 32),
                   umma_desc_sw128(k_addr + (k >> 2) * kApBlk + (k & 3) * 32), idesc1, k > 0 ? 1u : 0u);
        umma_commit(&s_full[buf]);
      };
      auto values = [&](int u, int buf, int i) {
        const uint32_t v_addr = ring + ((2 * i + 1) & 3) * kApF16Bytes;
#pragma unroll
        for (int k = 0; k < 8; ++k)      // 16 tokens per step: 8 columns of P, two 8-row groups of V
          umma_f16_ts(tmem_base + 256 + u * 128, tmem_base + buf * 128 + 64 + k * 8, umma_desc_sw128_mn(v_addr + k * 2048, kApBlk), idesc2,
                      (i > 0 || k > 0) ? 1u : 0u);
        umma_commit(&o_full[u]);
      };
      wait_item(0);
      if (ok) {
        scores(0, 0, 0);
        if (n1 > 0) scores(1, 1, 0);
        umma_commit(&ring_empty[0]);
      }
      for (int i = 0; i < n0 && ok; ++i) {
        if (dual) {
          wait(&p_full[0], i & 1, kTimeoutConvert, 33);
          wait_item(2 * i + 1);
          if (ok) values(0, 0, i);
          if (i + 1 < n0) {
            wait_item(2 * i + 2);
            if (ok) scores(0, 0, i + 1);
          }
          if (i < n1) {
            wait(&p_full[1], i & 1, kTimeoutConvert, 34);
            if (ok) values(1, 1, i);
          }
          if (ok) umma_commit(&ring_empty[(2 * i + 1) & 3]);
          if (i + 1 < n1 && ok) scores(1, 1, i + 1);
          if (i + 1 < n0 && ok) umma_commit(&ring_empty[(2 * i + 2) & 3]);
        } else {
          if (i + 1 < n0) {
            wait_item(2 * i + 2);
            if (ok) {
              scores(0, (i + 1) & 1, i + 1);
              umma_commit(&ring_empty[(2 * i + 2) & 3]);
            }
          }
          wait(&p_full[i & 1], (i >> 1) & 1, kTimeoutConvert, 33);
          wait_item(2 * i + 1);
          if (ok) {
            values(0, i & 1, i);
            umma_commit(&ring_empty[(2 * i + 1) & 3]);
          }
        }
      }
    }
  } else if (warp >= kApConv) {
    // ------------------------------------------------------------------ expansion to f16: four warps for K, four for V, thread = token
    const int v = (warp - kApConv) >> 2, t = (warp & 3) * 32 + lane;
    bool ok = true;
    int unit = -100;      // exponent of the largest scale so far, at least this
    constexpr int kGaveUp = 1 << 20;
    for (int i = 0; i < n0; ++i) {
      const int j = 2 * i + v, slot = j & 3;
      bool okw = wait_bar(&raw_full[v], i & 1);
      if (!okw) report(p.status, kTimeoutTmaFull, 35);
      Pack16 x[8];
      const unsigned char* raw = sRaw + v * kApRawBytes + t * 128;
#pragma unroll
      for (int c = 0; c < 8; ++c) x[c].u = *reinterpret_cast<const uint4*>(raw + ((c ^ (t & 7)) << 4));
      // tokens that no row of this CTA sees hold whatever the page held and become zeros
      const int tok = base + i * kApTile + t;
      uint32_t any = 0;
#pragma unroll
      for (int c = 0; c < 8; ++c) any |= x[c].w[0] | x[c].w[1] | x[c].w[2] | x[c].w[3];
      const bool live = tok >= first_tok && tok <= last_pos && (any & 0x7f7f7f7fu) != 0;
      const float sc = live ? sScale[v * kApTile + t] : 0.f;
      const int e = static_cast<int>((__float_as_uint(sc) >> 23) & 255u) - 127;
      // a failed wait must not leave the other warps alone at the barrier: all four read the verdicts and leave together
      const int top = __reduce_max_sync(0xffffffffu, !okw || *abort_flag ? kGaveUp : (live ? e : -127));
      int* tops = sMax + (v * 2 + (i & 1)) * 4;
      if (lane == 0) tops[warp & 3] = top;
      if (v) asm volatile("bar.sync 2, 128;" ::: "memory");
      else asm volatile("bar.sync 1, 128;" ::: "memory");
      const int4 m4 = *reinterpret_cast<const int4*>(tops);
      const int most = max(max(m4.x, m4.y), max(m4.z, m4.w));
      if (most == kGaveUp) { *abort_flag = 1; break; }
      unit = max(unit, min(most, 127));
      // mantissa (in two terms) and power of two of the scale; f16 has no power of two below 2^-24, what is below that loses bits anyway
      const float m = e == 128 ? sc : __uint_as_float((__float_as_uint(sc) & 0x007fffffu) | 0x3f800000u);
      const int d = e - unit, b = min(d + 24, 0);
      const float mb = m * exp2_of(max(b, -126));
      const __half2 hi = __float2half2_rn(mb);
      const __half2 lo = __float2half2_rn(mb - __low2float(hi));
      const __half2 pow = __float2half2_rn(exp2_of(min(max(d - b, -24), 0)));
      if (okw && !wait_bar(&ring_empty[slot], ((j >> 2) & 1) ^ 1)) { report(p.status, kTimeoutStageEmpty, 36); okw = false; }
      if (!okw) *abort_flag = 1;
      ok = __all_sync(0xffffffffu, okw && !*abort_flag);
      if (!ok) continue;      // (to the verdict of the next tile)
      if (!__all_sync(0xffffffffu, live)) {
#pragma unroll
        for (int c = 0; c < 8; ++c)
          if (!live) x[c].u = make_uint4(0u, 0u, 0u, 0u);
      }
      unsigned char* dst = sRing + slot * kApF16Bytes + t * 128;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        Pack16 y[2];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const __half2 h = e4m3x2_to_h2(x[c].s[k]);
          const __half2 r = __hmul2(__hfma2(h, hi, __hmul2(h, lo)), pow);
          y[k >> 2].w[k & 3] = *reinterpret_cast<const uint32_t*>(&r);
        }
        unsigned char* blk = dst + (c >> 2) * kApBlk;
        *reinterpret_cast<uint4*>(blk + (((c * 2) & 7) ^ (t & 7)) * 16) = y[0].u;
        *reinterpret_cast<uint4*>(blk + (((c * 2 + 1) & 7) ^ (t & 7)) * 16) = y[1].u;
      }
      if (warp == kApConv + 4 * v && lane == 0) sExp[v * 4 + (i & 3)] = unit;
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) { mbar_arrive(&raw_empty[v]); mbar_arrive(&ring_full[slot]); }
    }
  } else if (sub == 0 || n1 > 0) {
    // ------------------------------------------------------------------ softmax (thread = query row of unit `sub`)
    const int r = (warp & 3) * 32 + lane, n = sub == 0 ? n0 : n1;
    const uint32_t lanes = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const uint32_t acc = lanes + 256 + sub * 128;
    const int row = unit_row(unit0 + sub) + r;
    const int my_pos = p.pos0 + row;
    const int my_first = (p.window > 0 && my_pos + 1 > p.window) ? my_pos + 1 - p.window : 0;
    const float sm = p.scale * 1.4426950408889634f * q_scale;
    float ref = -INFINITY, lsum = 0.f;
    int cv = 0;
    bool ok = true;
    for (int i = 0; i < n; ++i) {
      const int buf = dual ? sub : (i & 1), phase = dual ? (i & 1) : ((i >> 1) & 1), jv = 2 * i + 1;
      // (V's exponent is wanted here; its tile is expanded long before this product needs it)
      bool okw = wait_bar(&ring_full[jv & 3], (jv >> 2) & 1) && wait_bar(&s_full[buf], phase);
      if (!okw) { report(p.status, kTimeoutAccum, 37); *abort_flag = 1; }
      ok = __all_sync(0xffffffffu, okw && !*abort_flag);
      if (!ok) break;
      tc_fence_after();
      const int t0 = base + i * kApTile;
      const int cv_before = cv;
      cv = sExp[4 + (i & 3)];
      const bool regrow = i > 0 && cv != cv_before;
      const float sm_t = sm * exp2_of(sExp[i & 3]);
      const uint32_t ts = lanes + buf * 128;
      // the accumulator of the tiles before, times the rows' corrections and in its new unit: all of their products must have landed
      auto rescale = [&](float corr) {
        if (i == 0) return;
        corr *= exp2_of(max(cv_before - cv, -126));
        // (two units: S of this tile was issued behind that product, its barrier is complete)
        if (!__all_sync(0xffffffffu, wait_bar(&o_full[sub], (i - 1) & 1))) { report(p.status, kTimeoutAccum, 38); *abort_flag = 1; return; }
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < D; c += 16) {
          uint32_t o[16];
          tmem_ld_x16(acc + c, o);
#pragma unroll
          for (int j = 0; j < 16; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * corr);
          tmem_st_x16_async(acc + c, o);
        }
      };
      // warp-uniform choice: tcgen05.ld is .sync.aligned, every lane of the warp must take the same path
      const bool full = __all_sync(0xffffffffu, (t0 + kApTile - 1 <= my_pos) && (t0 >= my_first)) != 0;
      if (full) softmax_tile<false>(ts, t0, my_pos, my_first, sm_t, regrow, ref, lsum, rescale);
      else softmax_tile<true>(ts, t0, my_pos, my_first, sm_t, regrow, ref, lsum, rescale);
      // one unit: S of this tile says nothing of the product before it, whose phase must be behind us before the last one is waited for
      if (!dual && i > 0 && i == n - 1 && !__all_sync(0xffffffffu, wait_bar(&o_full[sub], (i - 1) & 1))) {
        report(p.status, kTimeoutAccum, 38);
        *abort_flag = 1;
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[buf]);
    }
    if (ok && !__all_sync(0xffffffffu, wait_bar(&o_full[sub], (n - 1) & 1))) { report(p.status, kTimeoutAccum, 39); *abort_flag = 1; ok = false; }
    if (ok) {
      tc_fence_after();
      const int head = kvh * group + (unit0 + sub) % group;
      const float inv_l = lsum > 0.f ? 1.f / lsum : 0.f, unit = exp2_of(cv);
      uint4* dst = reinterpret_cast<uint4*>(p.out + (static_cast<size_t>(row) * p.hq + head) * D);
#pragma unroll 1
      for (int c = 0; c < D; c += 32) {
        uint32_t o[32];
        tmem_ld_x32(acc + c, o);
        if (row < p.T) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            Pack16 x;
#pragma unroll
            for (int j = 0; j < 8; ++j) x.h[j] = f32_to_bf16(__uint_as_float(o[k * 8 + j]) * inv_l * unit);
            dst[c / 8 + k] = x.u;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kApMma) tmem_dealloc(tmem_base, 512);
}

// Two units per CTA share an expanded tile and fill each other's waits: 3.4 us per tile against 2.3 for one alone, behind 8 us for a
// CTA's first and last steps.  One each is the shorter span where units are fewer than SMs, and up to twice as many where the second
// wave's, the short ones, fit behind the first one's last: unit sms + i follows unit sms - 1 - i.  (us, one / two per CTA: 40 heads
// over 512 rows 28.3 / 31.1, behind 5000 more 191 / 151; 32 heads over 768 rows 33.6 / 38.4; 64 over 512 35.0 / 31.2; 8 over 4096 83 / 114.)
static int units_per_cta(const AttnPrefillParams& p, int sms) {
  const int64_t all = static_cast<int64_t>(p.units) * p.hkv;
  if (all <= sms) return 1;
  if (all > 2 * sms) return 2;
  const int row_tiles = dgpp_ceil_div(p.T, kApTile);
  auto tiles = [&](int u) {      // of the u-th longest unit
    const int row = (row_tiles - 1 - u / p.hq) * kApTile, low = p.pos0 + row;
    const int first = p.window > 0 && low + 1 > p.window ? low + 1 - p.window : 0;
    return (p.pos0 + (row + kApTile < p.T ? row + kApTile : p.T) - 1) / kApTile - first / kApTile + 1;
  };
  double one = 8 + 2.3 * tiles(0);
  for (int i = 0; i < all - sms; ++i) {
    const double two_waves = 16 + 2.3 * (tiles(sms - 1 - i) + tiles(sms + i));
    if (two_waves > one) one = two_waves;
  }
  return one <= 8.5 + 3.4 * tiles(0) ? 1 : 2;
}

}  // namespace dgpp

using namespace dgpp;

// Causal attention of T chunk rows (positions pos0 .. pos0 + T - 1 of the request whose block-table row is
// `block_table_row`) against the FP8 paged cache, which must already hold those positions.  head_dim 128.
DGPP_API int dgpp_attn_prefill_tc(const void* q, int64_t q_stride, const void* k_cache, const void* v_cache,
                                  const void* k_scale, const void* v_scale, const void* block_table_row, void* out,
                                  int T, int pos0, int hq, int hkv, int d, int page, int max_blocks, int num_blocks,
                                  float scale, int window, cudaStream_t st) {
  DGPP_REQUIRE(d == 128, "attn_prefill_tc: head_dim %d != 128", d);
  DGPP_REQUIRE(hkv > 0 && hq % hkv == 0, "attn_prefill_tc: bad head grouping %d/%d", hq, hkv);
  DGPP_REQUIRE(page == 16 || page == 32 || page == 64 || page == 128, "attn_prefill_tc: page %d unsupported", page);
  if (T == 0) return 0;
  AttnPrefillParams p;
  p.q = static_cast<const bf16*>(q);
  p.q_stride = q_stride;
  p.k_scale = static_cast<const float*>(k_scale);
  p.v_scale = static_cast<const float*>(v_scale);
  p.block_table = static_cast<const int32_t*>(block_table_row);
  p.out = static_cast<bf16*>(out);
  p.status = device_status_ptr();
  p.T = T; p.pos0 = pos0; p.hq = hq; p.hkv = hkv; p.page = page; p.max_blocks = max_blocks; p.window = window;
  p.scale = scale;
  const uint64_t total_rows = static_cast<uint64_t>(num_blocks) * hkv * page;
  CUtensorMap tK, tV;
  if (make_tmap_2d(&tK, k_cache, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, 128, total_rows, 128, 128, page, CU_TENSOR_MAP_SWIZZLE_128B))
    return -1;
  if (make_tmap_2d(&tV, v_cache, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, 128, total_rows, 128, 128, page, CU_TENSOR_MAP_SWIZZLE_128B))
    return -1;
  constexpr size_t smem = attn_prefill_smem_bytes();
  static_assert(smem <= 227 * 1024, "shared memory budget exceeded");
  static bool attr = false;
  static int sms = 0;
  if (!attr) {
    int dev = 0;
    DGPP_CUDA_OK(cudaGetDevice(&dev));
    DGPP_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    DGPP_CUDA_OK(cudaFuncSetAttribute(attn_prefill_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(smem)));
    attr = true;
  }
  p.units = hq / hkv * dgpp_ceil_div(T, kApTile);
  p.per_cta = units_per_cta(p, sms);
  DGPP_CUDA_OK(launch_early(attn_prefill_tc_kernel, hkv * dgpp_ceil_div(p.units, p.per_cta), kApThreads, smem, st, tK, tV, p));
  DGPP_CUDA_OK(cudaGetLastError());
  return 0;
}
