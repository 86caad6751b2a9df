// Activation producer + NVFP4 residual-term quantiser, one thread-block CLUSTER per row.
//
// A decode batch has only a handful of rows, so one CTA per row leaves the GPU idle; here the K columns of a row
// are split over the CTAs of a cluster (up to 8).  A thread owns 8 columns (half a block of 16) from the load to the
// packed codes, so a CTA has no barrier of its own; the two row-wide reductions (sum of squares for RMSNorm, max |x|
// for the activation scale) are one exchange: every warp sends its pair of partials to every CTA of the cluster
// (`st.async`, counted by the receiver's mbarrier), and every warp folds the CTA's copy in one fixed order, so
// all CTAs compute bit-identical row statistics.  The cluster barrier that makes the mbarriers known to the peers, and
// the loads of the norm weights, stand before the wait on the preceding grid.
// What bounds it: one chain of latencies: loads, exchange, three terms one after the other.  A pass of 16 layers of 5120 / 17408 took
// 1544 us at one row and 1741 at eight with a thread per block of 16, two barriers per reduction and cluster-wide barriers, 1440 and
// 1624 so; 16 layers of 2048 at eight rows 1046, 968 so.  A quantiser then adds 4 to 7 us to its layer's chain (5 to 10 before).  Alone, with
// nothing in front whose tail hides the barrier, it is 0.2 to 0.6 us slower than that form (8 normed rows of 5120 4.1 us, 4.7 so).
//
// Modes, output layout and arithmetic are those of fused_act_quant_kernel in gemm_fp4.cu:
//   0 plain rows, 1 swiglu([gate | up]), 2 rmsnorm(resid + delta) * w
//   q rows [token tile][term][token], scale factors in tcgen05.cp atom order per token tile.
#include <string.h>

#include "common/common.h"
#include "common/dtypes.cuh"
#include "common/ptx.cuh"
#include "kernels/comm.cuh"
#include "kernels/gemm_common.cuh"

namespace dgpp {

constexpr int kAqMaxThreads = 512;
constexpr int kAqNormThreads = 128;   // of the norm's rows: who adds which squares is part of the per-layer kernel's contract
constexpr int kAqNormWarps = kAqNormThreads / 32;
constexpr int kAqMaxWarps = kAqMaxThreads / 32;
constexpr int kAqMaxCluster = 8;
constexpr int kAqSplitBlock = 4;      // attention splits whose partials are in flight at once
constexpr int kAqAtom = 512;
constexpr int kAqMaxSegment = 48 * 1024;      // bytes of a row in one CTA

struct ClusterQuantArgs {
  const bf16* in;
  int64_t in_stride;
  const bf16* delta;
  const bf16* w;
  bf16* resid_out;
  bf16* x_out;
  uint8_t* q;
  uint8_t* sf;
  float* g;
  int T, T_pad, K, R, bn, cl;
  DeviceStatus* status;
  float eps, limit, alpha;     // alpha > 0: gate * sigmoid(alpha * gate) * (up + 1) in the swiglu mode
  int one_plus_w;
  // MODE 2 with fold = 1: `delta` is not read from memory but folded from the W partial tiles that the
  // tensor-parallel GEMMs pushed into this rank's symmetric region (ascending rank order, fp32, one bf16
  // rounding: the bits an all-reduce would have produced).  The kernel waits for the tile flags it needs and its
  // last CTA advances the collective epoch.
  int fold;
  CommState comm;
  // Grouped rows (mixture-of-experts): row t belongs to slot t / bn; rows of inactive slots (group_list[slot] < 0)
  // and rows t % bn >= group_rows are skipped.
  const int32_t* group_list;
  int group_rows;
  // MODE 3: the row is the decode-attention output, folded here from the split-KV partials (max / sum pairs and
  // unnormalised accumulators per (row, head, split)) in the arithmetic of the stand-alone combine kernel, so the
  // combine launch and one round trip of the attention output disappear.
  const float* part_ml;
  const float* part_acc;
  int splits, hq, D;
};

// Stores a pair of floats in a CTA of the cluster; the 8 bytes are counted by the mbarrier at `bar` there.
__device__ __forceinline__ void st_async_f32x2(uint32_t addr, float x, float y, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(addr), "f"(x), "f"(y), "r"(bar)
               : "memory");
}

// Eight columns of the folded decode attention row: split partials weighted by e^(their max - the row's), ascending.
__device__ __forceinline__ void fold_splits(const ClusterQuantArgs& a, int t, int col, float (&acc)[8], float& ll) {
  const int h = col / a.D, d0 = col % a.D;
  const size_t rh = static_cast<size_t>(t) * a.hq + h;
  const float* ml = a.part_ml + rh * a.splits * 2;
  const float* pa = a.part_acc + rh * a.splits * a.D + d0;
  float mm = -INFINITY;
#pragma unroll 8
  for (int sp = 0; sp < a.splits; ++sp) mm = fmaxf(mm, ml[sp * 2]);
  ll = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  for (int s0 = 0; s0 < a.splits; s0 += kAqSplitBlock) {
    float2 m[kAqSplitBlock];
    float4 v[kAqSplitBlock][2];
#pragma unroll
    for (int i = 0; i < kAqSplitBlock; ++i) {
      if (s0 + i >= a.splits) break;
      m[i] = make_float2(ml[(s0 + i) * 2], ml[(s0 + i) * 2 + 1]);
      const float4* src = reinterpret_cast<const float4*>(pa + static_cast<size_t>(s0 + i) * a.D);
      v[i][0] = src[0];
      v[i][1] = src[1];
    }
#pragma unroll
    for (int i = 0; i < kAqSplitBlock; ++i) {
      if (s0 + i >= a.splits) break;
      const float cw = m[i].x == -INFINITY ? 0.f : __expf(m[i].x - mm);
      ll += m[i].y * cw;
      acc[0] += v[i][0].x * cw; acc[1] += v[i][0].y * cw; acc[2] += v[i][0].z * cw; acc[3] += v[i][0].w * cw;
      acc[4] += v[i][1].x * cw; acc[5] += v[i][1].y * cw; acc[6] += v[i][1].z * cw; acc[7] += v[i][1].w * cw;
    }
  }
}

// Eight columns of swiglu: x the gate's, u the up projection's.
__device__ __forceinline__ void swiglu8(const ClusterQuantArgs& a, Pack16& x, const Pack16& u) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    float gv = bf16_to_f32(x.h[j]), uv = bf16_to_f32(u.h[j]);
    if (a.limit > 0.f) { gv = fminf(gv, a.limit); uv = fminf(fmaxf(uv, -a.limit), a.limit); }
    float sl;
    if (a.alpha > 0.f) {
      sl = bf16_to_f32(f32_to_bf16(gv / (1.f + __expf(-a.alpha * gv))));
      uv += 1.f;
    } else {
      sl = bf16_to_f32(f32_to_bf16(gv / (1.f + __expf(-gv))));
    }
    x.h[j] = f32_to_bf16(sl * uv);
  }
}

// Eight columns of a row to be normed: their squares, and the largest |x w|.
__device__ __forceinline__ void norm_statistics(const ClusterQuantArgs& a, const Pack16& x, const Pack16& w, float& ss, float& amax) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float f = bf16_to_f32(x.h[j]);
    ss += f * f;
    float gw = bf16_to_f32(w.h[j]);
    if (a.one_plus_w) gw += 1.f;
    amax = fmaxf(amax, fabsf(f * gw));
  }
}
__device__ __forceinline__ void norm_scale(const ClusterQuantArgs& a, Pack16& x, const Pack16& w, float rstd) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float nrm = bf16_to_f32(f32_to_bf16(bf16_to_f32(x.h[j]) * rstd));
    float gw = bf16_to_f32(w.h[j]);
    if (a.one_plus_w) gw += 1.f;
    x.h[j] = f32_to_bf16(nrm * gw);
  }
}

template <int MODE>
__global__ void __launch_bounds__(kAqMaxThreads) act_quant_cluster_kernel(ClusterQuantArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint4* seg = reinterpret_cast<uint4*>(smem_raw);  // this CTA's K / cl columns; a thread reads back what it wrote
  // (sum of squares, max |x|) of every warp of every CTA of the cluster
  __shared__ __align__(16) float2 part[kAqMaxCluster * kAqMaxWarps];
  __shared__ __align__(8) uint64_t arrived;
  const int c = blockIdx.x, t = blockIdx.y, tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, wid = tid >> 5;
  const int cl = a.cl, K = a.K, kseg = K / cl, k0 = c * kseg, nvec = kseg / 8;
  for (int i = tid; i < kAqMaxCluster * kAqMaxWarps; i += nthr) part[i] = make_float2(0.f, 0.f);
  if (tid == 0) {
    mbar_init(&arrived, 1);
    mbar_expect_tx(&arrived, cl * (nthr / 32) * 8);
    fence_mbar_init();
  }
  const uint4* wv = reinterpret_cast<const uint4*>(a.w + k0);
  Pack16 w0;      // the norm weights of this thread's first columns
  w0.u = make_uint4(0u, 0u, 0u, 0u);
  if (MODE == 2 && tid < nvec) w0.u = wv[tid];
  cluster_barrier();
  pdl_wait();
  if (a.group_list && (a.group_list[t / a.bn] < 0 || t % a.bn >= a.group_rows)) return;   // whole cluster leaves together
  float ss = 0.f, amax = 0.f;
  uint32_t fold_epoch = 0;
  int fold_parity = 0;
  if (MODE == 2 && a.fold) {
    fold_epoch = *a.comm.epoch + 1;
    fold_parity = fold_epoch & 1;
    const int tile0 = k0 / 128, ntile = (k0 + kseg - 1) / 128 - tile0 + 1;
    for (int i = tid; i < ntile * a.comm.world; i += nthr) {
      const int src = i / ntile, tl = tile0 + i % ntile;
      if (!wait_flag(flag(a.comm, a.comm.rank, fold_parity, src, tl), fold_epoch)) report(a.status, kTimeoutPeerFlag, src);
    }
    __syncthreads();
  }
  for (int i = tid; i < nvec; i += nthr) {
    Pack16 x;
    if (MODE == 2) {
      x.u = reinterpret_cast<const uint4*>(a.in + static_cast<size_t>(t) * a.in_stride + k0)[i];
      uint4* sum_out = reinterpret_cast<uint4*>(a.resid_out + static_cast<size_t>(t) * K + k0) + i;
      if (a.fold) {
        float acc[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = 0.f;
        for (int r = 0; r < a.comm.world; ++r) {
          Pack16 d;
          d.u = ld_v4_global_volatile(payload(a.comm, a.comm.rank, fold_parity, r) +
                                      (static_cast<size_t>(t) * K + k0) * 2 + static_cast<size_t>(i) * 16);
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[j] += bf16_to_f32(d.h[j]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) x.h[j] = f32_to_bf16(bf16_to_f32(x.h[j]) + bf16_to_f32(f32_to_bf16(acc[j])));
        *sum_out = x.u;
      } else if (a.delta) {
        Pack16 d;
        d.u = reinterpret_cast<const uint4*>(a.delta + static_cast<size_t>(t) * K + k0)[i];
#pragma unroll
        for (int j = 0; j < 8; ++j) x.h[j] = f32_to_bf16(bf16_to_f32(x.h[j]) + bf16_to_f32(d.h[j]));
        *sum_out = x.u;
      }
      Pack16 w;
      w.u = i == tid ? w0.u : wv[i];
      norm_statistics(a, x, w, ss, amax);
    } else {
      if (MODE == 3) {
        float acc[8], ll;
        fold_splits(a, t, k0 + i * 8, acc, ll);
#pragma unroll
        for (int j = 0; j < 8; ++j) x.h[j] = f32_to_bf16(ll > 0.f ? acc[j] / ll : 0.f);
      } else {
        const uint4* rr = reinterpret_cast<const uint4*>(a.in + static_cast<size_t>(t) * a.in_stride + k0);
        x.u = rr[i];
        if (MODE == 1) {
          Pack16 u;
          u.u = rr[K / 8 + i];
          swiglu8(a, x, u);
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(bf16_to_f32(x.h[j])));
      if (a.x_out) reinterpret_cast<uint4*>(a.x_out + static_cast<size_t>(t) * K + k0)[i] = x.u;
    }
    seg[i] = x.u;
  }
  // the row's statistics: this warp's partials to every CTA, then all of them from the own copy
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    if (MODE == 2) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  }
  if (lane < cl)
    st_async_f32x2(mapa_shared(smem_u32(&part[c * kAqMaxWarps + wid]), lane), ss, amax, mapa_shared(smem_u32(&arrived), lane));
  if (!wait_bar(&arrived, 0) && lane == 0) report(a.status, kTimeoutConvert, 61);
  {
    const float4* pp = reinterpret_cast<const float4*>(part) + lane * 2;      // four pairs per lane, in order of CTA and warp
    const float4 x = pp[0], y = pp[1];
    amax = fmaxf(fmaxf(x.y, x.w), fmaxf(y.y, y.w));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (MODE == 2) {
      // the norm's rows have at most four warps per CTA: lane 4 c holds those of CTA c; warps, then CTAs in ascending order (the sum
      // that the per-layer kernel forms)
      const float r = x.x + x.z + y.x + y.z;
      ss = 0.f;
#pragma unroll
      for (int i = 0; i < kAqMaxCluster; ++i) ss += __shfl_sync(0xffffffffu, r, i * (kAqMaxWarps / 4));
    }
  }
  float rstd = 0.f;
  if (MODE == 2) {
    rstd = rsqrtf(ss / static_cast<float>(K) + a.eps);
    // Row scale from a bound instead of the exact maximum of the normalised row: |bf16(bf16(x rstd) w)| <=
    // |x w| rstd (1 + 2^-8)^2, so max |x w| * rstd * 1.0079 covers every element (at most 0.8 % above the true
    // maximum) and is known from this single pass: no second row-wide reduction.
    amax = amax * rstd * 1.0079f;
  }
  const float gs = amax > 0.f ? amax / (6.f * 256.f) : 1.f;
  if (c == 0 && tid == 0) a.g[t] = gs;
  const float inv_g = 1.f / gs;
  const int stages = K / 256;
  const int atoms = a.R * a.bn > 128 ? 2 : 1;
  const int tile = t / a.bn, m = t % a.bn;
  for (int i0 = 0; i0 < nvec; i0 += nthr) {      // (whole warps: the two threads of a block exchange its maxima)
    const int i = i0 + tid;
    const bool on = i < nvec;
    Pack16 x;
    x.u = on ? seg[i] : make_uint4(0u, 0u, 0u, 0u);
    if (MODE == 2 && on) {
      Pack16 w;
      w.u = i0 == 0 ? w0.u : wv[i];
      norm_scale(a, x, w, rstd);
      if (a.x_out) reinterpret_cast<uint4*>(a.x_out + static_cast<size_t>(t) * K + k0)[i] = x.u;
    }
    float res[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) res[j] = bf16_to_f32(x.h[j]) * inv_g;
    const int gi = k0 / 16 + (i >> 1);
    const int st = gi >> 4, step = (gi >> 2) & 3, fi = gi & 3;
    for (int r = 0; r < a.R; ++r) {
      float bm = fmaxf(fmaxf(fmaxf(fabsf(res[0]), fabsf(res[1])), fmaxf(fabsf(res[2]), fabsf(res[3]))),
                       fmaxf(fmaxf(fabsf(res[4]), fabsf(res[5])), fmaxf(fabsf(res[6]), fabsf(res[7]))));
      bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, 1));
      const uint8_t sb = f32_to_e4m3(bm * (1.f / 6.f));
      const float s = e4m3_value_f32(bm * (1.f / 6.f));   // value of the code sb, without an fp8 decode of it
      const float inv_s = s > 0.f ? 1.f / s : 0.f;
      float sc[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) sc[j] = res[j] * inv_s;
      const uint32_t codes = f32x8_to_e2m1x8(sc);
      e2m1x8_residual(codes, s, res);
      if (!on) continue;
      const size_t ro = static_cast<size_t>(tile) * a.R * a.bn + static_cast<size_t>(r) * a.bn + m;
      *reinterpret_cast<uint32_t*>(a.q + ro * (K / 2) + k0 / 2 + i * 4) = codes;
      if ((i & 1) == 0) {
        const int brow = r * a.bn + m, h = brow >> 7, mm = brow & 127;
        const size_t atom_idx = ((static_cast<size_t>(tile) * stages + st) * 4 + step) * atoms + h;
        a.sf[atom_idx * kAqAtom + (mm & 31) * 16 + (mm >> 5) * 4 + fi] = sb;
      }
    }
  }
  if (MODE == 2 && a.fold) {
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      if (atomicAdd(a.comm.done_ctas, 1u) == gridDim.x * gridDim.y - 1) {
        *a.comm.done_ctas = 0;
        *a.comm.epoch = fold_epoch;
        __threadfence();
      }
    }
  }
}

// Bulk rows (rows fill the SMs by themselves): one CTA of 128 threads per row, a thread per block of 16.  The results are the cluster
// form's bit for bit: a maximum does not depend on its order, and the norm's squares are added as the warps of a cluster of `cl` CTAs
// would add them, whose places this CTA's warps take in turns.  Bound by issue slots rather than latency there: no exchange, no
// mbarrier, no shuffles per term and 8-byte stores of codes.  2048 x 5120, three terms, plain / swiglu: cluster form of one CTA 41.0 /
// 49.2 us, so 16.3 / 25.1; 128 rows 5.7 / 6.7 and 4.6 / 7.0.  2048 normed rows of 5120 against
// eight CTAs each: 75.6 us, 28.7 so.
constexpr int kAqBulkThreads = 128;
// Normed rows beyond this many (us, this form / a cluster of eight: 2048 columns 128 rows 3.9 / 4.7; 5120 columns 128 rows 7.7 / 6.8, 173
// rows 8.6 / 10.0; 17408 columns 173 rows 20.7 / 17.9, 256 rows 20.9 / 23.0).
static int bulk_norm_rows(int K) { return K <= 2048 ? 64 : K <= 6144 ? 160 : 255; }

template <int MODE>
__global__ void __launch_bounds__(kAqBulkThreads) act_quant_bulk_kernel(ClusterQuantArgs a) {
  static_assert(MODE >= 0 && MODE <= 2, "plain, swiglu or normed rows");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint4* row = reinterpret_cast<uint4*>(smem_raw);
  __shared__ float wmax[kAqBulkThreads / 32];
  pdl_wait();
  const int t = blockIdx.x, tid = threadIdx.x, K = a.K;
  if (a.group_list && (a.group_list[t / a.bn] < 0 || t % a.bn >= a.group_rows)) return;
  const uint4* rr = reinterpret_cast<const uint4*>(a.in + static_cast<size_t>(t) * a.in_stride);
  const uint4* wv = reinterpret_cast<const uint4*>(a.w);
  float amax = 0.f, rstd = 0.f;
  if (MODE == 2) {
    __shared__ __align__(16) float squares[kAqMaxCluster * kAqNormWarps];
    const int lane = tid & 31, nvec = K / a.cl / 8, warps = nvec < kAqNormThreads ? (nvec + 31) / 32 : kAqNormWarps;
    for (int vw = tid >> 5; vw < a.cl * warps; vw += kAqBulkThreads / 32) {      // warp vw % warps of CTA vw / warps
      const int c = vw / warps;
      float ss = 0.f;
      for (int i = (vw - c * warps) * 32 + lane; i < nvec; i += warps * 32) {
        const int at = c * nvec + i;
        Pack16 x, w;
        x.u = rr[at];
        w.u = wv[at];
        if (a.delta) {
          Pack16 d;
          d.u = reinterpret_cast<const uint4*>(a.delta + static_cast<size_t>(t) * K)[at];
#pragma unroll
          for (int j = 0; j < 8; ++j) x.h[j] = f32_to_bf16(bf16_to_f32(x.h[j]) + bf16_to_f32(d.h[j]));
          reinterpret_cast<uint4*>(a.resid_out + static_cast<size_t>(t) * K)[at] = x.u;
        }
        norm_statistics(a, x, w, ss, amax);
        row[at] = x.u;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (lane == 0) squares[c * kAqNormWarps + (vw - c * warps)] = ss;
    }
    if (tid < kAqMaxCluster * kAqNormWarps && (tid / kAqNormWarps >= a.cl || tid % kAqNormWarps >= warps)) squares[tid] = 0.f;
    __syncthreads();
    float ss = 0.f;
#pragma unroll
    for (int c = 0; c < kAqMaxCluster; ++c) {
      const float4 s4 = reinterpret_cast<const float4*>(squares)[c];
      ss += s4.x + s4.y + s4.z + s4.w;
    }
    rstd = rsqrtf(ss / static_cast<float>(K) + a.eps);
  }
  for (int i = tid; MODE != 2 && i < K / 8; i += kAqBulkThreads) {
    Pack16 x;
    x.u = rr[i];
    if (MODE == 1) {
      Pack16 u;
      u.u = rr[K / 8 + i];
      swiglu8(a, x, u);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(bf16_to_f32(x.h[j])));
    row[i] = x.u;
    if (a.x_out) reinterpret_cast<uint4*>(a.x_out + static_cast<size_t>(t) * K)[i] = x.u;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((tid & 31) == 0) wmax[tid >> 5] = amax;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kAqBulkThreads / 32; ++i) amax = fmaxf(amax, wmax[i]);
  if (MODE == 2) amax = amax * rstd * 1.0079f;      // (a bound, as in the cluster form)
  const float gs = amax > 0.f ? amax / (6.f * 256.f) : 1.f;
  if (tid == 0) a.g[t] = gs;
  const float inv_g = 1.f / gs;
  const int stages = K / 256, atoms = a.R * a.bn > 128 ? 2 : 1, tile = t / a.bn, m = t % a.bn;
  for (int gi = tid; gi < K / 16; gi += kAqBulkThreads) {
    Pack16 lo, hi;
    lo.u = row[gi * 2];
    hi.u = row[gi * 2 + 1];
    if (MODE == 2) {
      Pack16 w[2];
      w[0].u = wv[gi * 2];
      w[1].u = wv[gi * 2 + 1];
      norm_scale(a, lo, w[0], rstd);
      norm_scale(a, hi, w[1], rstd);
      if (a.x_out) {
        uint4* xo = reinterpret_cast<uint4*>(a.x_out + static_cast<size_t>(t) * K);
        xo[gi * 2] = lo.u;
        xo[gi * 2 + 1] = hi.u;
      }
    }
    float res[16];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      res[j] = bf16_to_f32(lo.h[j]) * inv_g;
      res[8 + j] = bf16_to_f32(hi.h[j]) * inv_g;
    }
    const int st = gi >> 4, step = (gi >> 2) & 3, fi = gi & 3;
    for (int r = 0; r < a.R; ++r) {
      float bm = 0.f;
#pragma unroll
      for (int j = 0; j < 16; ++j) bm = fmaxf(bm, fabsf(res[j]));
      const uint8_t sb = f32_to_e4m3(bm * (1.f / 6.f));
      const float s = e4m3_value_f32(bm * (1.f / 6.f));   // value of the code sb, without an fp8 decode of it
      const float inv_s = s > 0.f ? 1.f / s : 0.f;
      float sc[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) sc[j] = res[j] * inv_s;
      const uint32_t c0 = f32x8_to_e2m1x8(sc), c1 = f32x8_to_e2m1x8(sc + 8);
      e2m1x8_residual(c0, s, res);
      e2m1x8_residual(c1, s, res + 8);
      const size_t ro = static_cast<size_t>(tile) * a.R * a.bn + static_cast<size_t>(r) * a.bn + m;
      *reinterpret_cast<uint2*>(a.q + ro * (K / 2) + gi * 8) = make_uint2(c0, c1);
      const int brow = r * a.bn + m, h = brow >> 7, mm = brow & 127;
      const size_t atom_idx = ((static_cast<size_t>(tile) * stages + st) * 4 + step) * atoms + h;
      a.sf[atom_idx * kAqAtom + (mm & 31) * 16 + (mm >> 5) * 4 + fi] = sb;
    }
  }
}

// A row segment of up to 48 KB is admitted; with the kernels' own static shared memory that is more than a launch gets unasked.
template <class Kernel>
static int allow_segment(Kernel kern, size_t bytes) {
  constexpr size_t kUnasked = 46 * 1024;
  if (bytes > kUnasked) DGPP_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kAqMaxSegment));
  return 0;
}

template <int MODE>
static int launch_cluster(const ClusterQuantArgs& a, cudaStream_t st) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(a.cl, a.T, 1);
  const int vecs = a.K / a.cl / 8, most = MODE == 2 ? kAqNormThreads : kAqMaxThreads;      // one thread each, as far as a CTA goes
  cfg.blockDim = dim3(vecs < most ? (vecs + 31) / 32 * 32 : most, 1, 1);
  cfg.dynamicSmemBytes = static_cast<size_t>(a.K / a.cl) * 2;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = a.cl;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (allow_segment(act_quant_cluster_kernel<MODE>, cfg.dynamicSmemBytes)) return -1;
  DGPP_CUDA_OK(cudaLaunchKernelEx(&cfg, act_quant_cluster_kernel<MODE>, a));
  return 0;
}

}  // namespace dgpp

using namespace dgpp;

// Same contract as dgpp_act_quant_nvfp4, row split over a cluster of `cl` CTAs (1, 2, 4 or 8; K / cl % 16 == 0).
DGPP_API int dgpp_act_quant_nvfp4_cluster(int mode, const void* in, int64_t in_stride, const void* delta,
                                          const void* w, void* resid_out, void* x_out, void* q, void* sf, void* g,
                                          int T, int T_pad, int K, int R, int bn, int cl, float eps, float limit,
                                          float alpha, int one_plus_w, void* comm_fold, const void* group_list, int group_rows,
                                          cudaStream_t st) {
  DGPP_REQUIRE(K % 256 == 0, "act_quant: K %d must be a multiple of 256", K);
  DGPP_REQUIRE(cl == 1 || cl == 2 || cl == 4 || cl == 8, "act_quant: cluster size %d not in {1,2,4,8}", cl);
  DGPP_REQUIRE((K / cl) % 16 == 0 && K % cl == 0, "act_quant: K %d does not split over %d CTAs", K, cl);
  DGPP_REQUIRE(R >= 1 && R <= 4 && R * bn <= 256, "act_quant: bad terms %d / tile %d", R, bn);
  DGPP_REQUIRE(T_pad % bn == 0 && T_pad >= T, "act_quant: T_pad %d must be a multiple of bn %d and >= T", T_pad, bn);
  DGPP_REQUIRE(static_cast<size_t>(K / cl) * 2 <= kAqMaxSegment, "act_quant: segment too large");
  if (T == 0) return 0;
  ClusterQuantArgs a;
  a.in = static_cast<const bf16*>(in);
  a.in_stride = in_stride;
  a.delta = static_cast<const bf16*>(delta);
  a.w = static_cast<const bf16*>(w);
  a.resid_out = static_cast<bf16*>(resid_out);
  a.x_out = static_cast<bf16*>(x_out);
  a.q = static_cast<uint8_t*>(q);
  a.sf = static_cast<uint8_t*>(sf);
  a.g = static_cast<float*>(g);
  a.T = T; a.T_pad = T_pad; a.K = K; a.R = R; a.bn = bn; a.cl = cl; a.eps = eps; a.limit = limit; a.alpha = alpha;
  a.one_plus_w = one_plus_w;
  a.status = device_status_ptr();
  a.group_list = static_cast<const int32_t*>(group_list);
  a.group_rows = group_rows;
  a.fold = 0;
  memset(&a.comm, 0, sizeof(a.comm));
  if (comm_fold) {
    const DgppComm* c = static_cast<const DgppComm*>(comm_fold);
    DGPP_REQUIRE(mode == 2, "act_quant: the all-reduce fold exists for the add + RMSNorm mode only");
    DGPP_REQUIRE(resid_out != nullptr, "act_quant fold: resid_out required");
    DGPP_REQUIRE(K % 128 == 0 && K / 128 <= kCommMaxCtas && static_cast<size_t>(T) * K * 2 <= c->st.slot_bytes,
                 "act_quant fold: %d x %d does not fit the symmetric slot / flag table", T, K);
    a.fold = 1;
    a.comm = c->st;
  }
  const size_t smem = static_cast<size_t>(K) * 2;
  if ((cl == 1 && (mode == 0 || mode == 1)) || (mode == 2 && !a.fold && T > bulk_norm_rows(K) && smem <= kAqMaxSegment)) {
    auto kern = mode == 0 ? act_quant_bulk_kernel<0> : mode == 1 ? act_quant_bulk_kernel<1> : act_quant_bulk_kernel<2>;
    if (allow_segment(kern, smem)) return -1;
    kern<<<T, kAqBulkThreads, smem, st>>>(a);
    DGPP_CUDA_OK(cudaGetLastError());
    return 0;
  }
  if (mode == 0) return launch_cluster<0>(a, st);
  if (mode == 1) return launch_cluster<1>(a, st);
  if (mode == 2) return launch_cluster<2>(a, st);
  dgpp_set_error("act_quant: unknown mode %d", mode);
  return -1;
}

// Decode attention epilogue: fold the split-KV partials of dgpp_attn_decode_tc / dgpp_attn_decode (called with a null
// output) and quantise the rows for the o projection in one launch.  K = hq * d; x_out (optional) receives the bf16
// attention output [T, K].
DGPP_API int dgpp_attn_combine_quant(const void* part_ml, const void* part_acc, int splits, int hq, int d, void* x_out,
                                     void* q, void* sf, void* g, int T, int T_pad, int R, int bn, int cl,
                                     cudaStream_t st) {
  const int K = hq * d;
  DGPP_REQUIRE(part_ml && part_acc && splits >= 1, "attn_combine_quant: partials required");
  DGPP_REQUIRE(K % 256 == 0 && d % 8 == 0, "attn_combine_quant: hq %d x d %d must give K %% 256 == 0", hq, d);
  DGPP_REQUIRE(cl == 1 || cl == 2 || cl == 4 || cl == 8, "attn_combine_quant: cluster size %d not in {1,2,4,8}", cl);
  DGPP_REQUIRE((K / cl) % 16 == 0 && K % cl == 0, "attn_combine_quant: K %d does not split over %d CTAs", K, cl);
  DGPP_REQUIRE(R >= 1 && R <= 4 && R * bn <= 256, "attn_combine_quant: bad terms %d / tile %d", R, bn);
  DGPP_REQUIRE(T_pad % bn == 0 && T_pad >= T, "attn_combine_quant: T_pad %d must be a multiple of bn %d and >= T", T_pad, bn);
  DGPP_REQUIRE(static_cast<size_t>(K / cl) * 2 <= kAqMaxSegment, "attn_combine_quant: segment too large");
  if (T == 0) return 0;
  ClusterQuantArgs a;
  memset(&a, 0, sizeof(a));
  a.x_out = static_cast<bf16*>(x_out);
  a.q = static_cast<uint8_t*>(q);
  a.sf = static_cast<uint8_t*>(sf);
  a.g = static_cast<float*>(g);
  a.T = T; a.T_pad = T_pad; a.K = K; a.R = R; a.bn = bn; a.cl = cl; a.eps = 0.f; a.limit = 0.f; a.alpha = 0.f;
  a.status = device_status_ptr();
  a.part_ml = static_cast<const float*>(part_ml);
  a.part_acc = static_cast<const float*>(part_acc);
  a.splits = splits; a.hq = hq; a.D = d;
  return launch_cluster<3>(a, st);
}
