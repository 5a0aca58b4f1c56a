// Rows of 256 bytes on the tcgen05 kernels: bf16 heads of 128 (kWide128) and fp32 heads of up to 64 under
// "tf32", every value held as a bf16 pair hi + lo (kSplit; Rows in tc_common.cuh).  Both have the same
// tiles — two [rows][64 bf16] sub-tiles — and the same accumulators: 128 columns, which are the 128
// features of a head, or X_hi and X_lo products of 64 features that the epilogue adds.  At the end of the file, the
// relu, relu2 and softplus bids of bf16 heads of 64 (kPairs64).
// The shares, pdp, P~ and do' that these kernels form are multiplied as pairs hi + lo, 16 bits of each: the tile
// kernels that they replace keep 11 (tf32), one bf16 value would keep 8.
//
// The forward is row pass + column-sum scan + query-stationary main pass, the wide instantiations of the
// kernels in tc_kernels.cuh and tc_rowpass_kernels.cuh; the reverse main pass has a kernel of its own, since the
// narrow one's accumulators would need 656 of the 512 TMEM columns.
//
// Forward + backward at B4 H8 T4096 on one B200, before (tile kernels with tf32 products) and after, the same tensors call
// after call (other tensors every call: 2.02 and 1.97 ms):
//   bf16 d = 128  14.8 ms -> 1.93 ms  (reverse pass 7.24 -> 0.94, main pass 3.82 -> 0.31)
//   fp32 d = 64    7.1 ms -> 1.84 ms  (reverse pass 3.51 -> 0.81, main pass 1.61 -> 0.31)
// (with single bf16 values bf16 d = 128 takes 1.64 ms, its outputs 1.0e-3 off; with exponentials that lose a NaN and
// masks that end at the last key only both are 0.9% faster).  Against 64 bits, 2-norm: bf16 outputs
// 1.3e-4 -> 1.6e-6, gradients 1.7e-3 before and after (their own rounding to bf16); fp32 outputs 2.8e-4 -> about 1e-5.
#pragma once

#include "tc_kernels.cuh"
#include "tc_rowpass_kernels.cuh"

namespace dil {
namespace tc {

// fp32 (rows, d) -> bf16 (rows, 128): [hi 64 | lo 64], zeros behind d.  One thread per 4 features of a row; grid.y
// picks the tensor.  Bound by memory: 16 bytes read and 16 written per 4 values of d = 64.
struct SplitArgs {
  const float* src[3];
  __nv_bfloat16* dst[3];
};
__global__ void split_operands_kernel(SplitArgs a, int64_t rows, int d) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= rows * 16) return;
  const int64_t r = idx >> 4;
  const int c = (int)(idx & 15) * 4;
  float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
  if (c < d) x = *reinterpret_cast<const float4*>(a.src[blockIdx.y] + r * d + c);
  uint2 hi, lo;
  split_pair(x.x, x.y, hi.x, lo.x);
  split_pair(x.z, x.w, hi.y, lo.y);
  uint2* dst = reinterpret_cast<uint2*>(a.dst[blockIdx.y] + r * 128 + c);
  dst[0] = hi;
  dst[16] = lo;
}

__device__ __forceinline__ void load_vec(const float* p, float (&x)[2]) {
  const float2 v = *reinterpret_cast<const float2*>(p);
  x[0] = v.x; x[1] = v.y;
}
__device__ __forceinline__ void load_vec(const float* p, float (&x)[4]) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
}
template <int E> __device__ __forceinline__ void load_vec(const __nv_bfloat16* p, float (&x)[E]) {
#pragma unroll
  for (int e = 0; e < E; e += 2) {
    const uint32_t v = *reinterpret_cast<const uint32_t*>(p + e);
    x[e] = __uint_as_float(v << 16);
    x[e + 1] = __uint_as_float(v & 0xffff0000u);
  }
}

// backward_prep_kernel for wide rows: dbar' and do' = sinv * dout as [hi | lo], 128 | 128 (kWide128) or 64 | 64 features.
template <typename TD, int W>
__global__ void wide_backward_prep_kernel(const TD* __restrict__ dout, const float* __restrict__ out,
                                          const float* __restrict__ ssum, float eps, int64_t rows, int d,
                                          float* __restrict__ dbarp, __nv_bfloat16* __restrict__ dop,
                                          float* __restrict__ ghat, float* __restrict__ dq_main) {
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  constexpr int E = Rows<W>::kHead / 32;                 // features per lane: 4 or 2
  const int c = lane * E;
  float a[E], b[E];
#pragma unroll
  for (int e = 0; e < E; ++e) a[e] = b[e] = 0.f;
  if (c < d) {
    load_vec(dout + row * d + c, a);
    load_vec(out + row * d + c, b);
  }
  const float sinv = 1.f / (ssum[row] + eps);
  float dot = 0.f;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    dot = fmaf(a[e], b[e], dot);
    a[e] *= sinv;
  }
  dot = warp_sum(dot);
  if (W == kWide128) {
    uint2 hi, lo;
    split_pair(a[0], a[1], hi.x, lo.x);
    split_pair(a[E - 2], a[E - 1], hi.y, lo.y);
    reinterpret_cast<uint2*>(dop + row * 256)[lane] = hi;
    reinterpret_cast<uint2*>(dop + row * 256 + 128)[lane] = lo;
    reinterpret_cast<float4*>(dq_main + row * 128)[lane] = make_float4(0.f, 0.f, 0.f, 0.f);
  } else {
    uint32_t hi, lo;
    split_pair(a[0], a[1], hi, lo);
    reinterpret_cast<uint32_t*>(dop + row * 128)[lane] = hi;
    reinterpret_cast<uint32_t*>(dop + row * 128 + 64)[lane] = lo;
    reinterpret_cast<float2*>(dq_main + row * 64)[lane] = make_float2(0.f, 0.f);
  }
  if (lane == 0) {
    dbarp[row] = dot * sinv;
    ghat[row] = 0.f;
  }
}

// dq = dq_main - ghat * pk in fp32, rows of d out of padded rows of 64.
__global__ void split_dq_from_pk_kernel(const float* __restrict__ dq_main, const float* __restrict__ pk,
                                        const float* __restrict__ ghat, float* __restrict__ dq, int64_t rows, int d) {
  const int per = d / 4;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows * per) return;
  const int64_t r = i / per;
  const float4 a = reinterpret_cast<const float4*>(dq_main + r * 64)[i - r * per];
  const float4 b = reinterpret_cast<const float4*>(pk)[i];
  const float gh = ghat[r];
  reinterpret_cast<float4*>(dq)[i] =
      make_float4(fmaf(-gh, b.x, a.x), fmaf(-gh, b.y, a.y), fmaf(-gh, b.z, a.z), fmaf(-gh, b.w, a.w));
}

// Main reverse pass over wide rows: the arithmetic of backward_main_kernel (two compute warpgroups, lane =
// key, two threads per key and half-step of 64 queries, reverse_sweeps), 384 threads, one CTA per SM.
//   TMEM: S^T 64 | dOV^T 64 | dV 128 | dK 128 | dQ^T 64.
// What differs from the narrow kernel, and why:
//  * one stage of scores instead of two (dV and dK take 256 columns): the scores of half-step h + 1 are issued right
//    behind the dV and dK products of h, which read the share and pdp values stored over the scores of h;
//  * dQ comes out transposed, dQ^T [128 features x 64 queries] = K^T pdp, M = the 128 columns of a K row: pdp is
//    then the B operand [keys][64 queries], 16 KB per half-step instead of 32 KB per 128 queries, and a
//    thread of the read-out (lane = feature) writes one fp32 column of the [query][32 features] staging
//    tile of its warp, 128 consecutive bytes per warp and store;
//  * V stays in shared memory (as a TMEM operand it would take 64 columns);
//  * ghat, the sum of pdp over keys, is formed by shuffles in fp32 once the half-step's tiles are handed over, while
//    the compute warps would wait for the next scores (as a product of its own against a tile of ones it was 16 of
//    the 76 MMAs of a kWide128 half-step: 1.11 -> 0.94 ms, kSplit 0.92 -> 0.81 ms, n = 32, T = 4096, when one thread
//    issued them at about 50 cycles each).
//  * share and pdp are multiplied as hi and lo planes (two A operands side by side in TMEM, two pdp tiles); for kSplit
//    dQ^T rows 64..127 (K_lo) are reduced into the same columns of dq_main as rows 0..63;
//  * kWide128 stages 32 queries of dQ at a time (16 KB instead of 32): its do' takes 64 KB.
// kPairs64 serves pass 2 of the f(a) / rowsum(f) bids: ghat (of backward_main_kernel's pass 1) is subtracted before the
// factor multiplies, dk is final (written as TOut to dk_main), and rows 64..127 of dQ^T, whose A operand is the V tile
// behind K, are not used.
template <int W> constexpr int kDqRows = W == kWide128 ? 32 : 64;
// Its accumulators leave TMEM for two stages of scores, so the products of a half-step and the scores of the next but one
// run under the arithmetic of the next (with one stage the softplus pass at n = 32, T = 8192 took 3.12 ms, now 2.99).
template <int W> constexpr int kScoreStages = W == kPairs64 ? 2 : 1;
template <int W> constexpr int kRowStages = 2 * kScoreStages<W>;          // half-steps of q and do' in shared memory
template <int W> constexpr int kBwdWideSmem =
    2 * (int)Rows<W>::kBytes + kRowStages<W> * (Rows<W>::kSub + Rows<W>::kDoSub) * (int)kTileBytes / 2 +
    Rows<W>::kPlanes * (int)kTileBytes + kDqRows<W> * 512 + 2048 + 2048 + 1024 + 256 + 1024;

template <int W, typename TOut, int BID = kBidSoftmax, int SHARE = kShareInclusive, int PASS = 0>
__global__ void __launch_bounds__(kBwdThreads, 1) wide_backward_main_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
    const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
    const __grid_constant__ CUtensorMap map_dq, Geom g, const float* __restrict__ rmax,
    const float* __restrict__ rden, const float* __restrict__ dbarp, const float* __restrict__ carry,
    const float* __restrict__ total, std::conditional_t<PASS == 2, TOut, float>* __restrict__ dk_main,
    TOut* __restrict__ dv, float* __restrict__ ghat) {
  static_assert(PASS == 0 || PASS == 2, "pass 1 is backward_main_kernel's");
  constexpr uint32_t TB = Rows<W>::kBytes;                 // [128] rows of k or v: 32 KB
  constexpr uint32_t HB = TB / 2, HSub = kTileBytes / 2;   // [64] rows of q, and one of their sub-tiles
  constexpr uint32_t HBd = Rows<W>::kDoSub * HSub;         // [64] rows of do'
  constexpr int kDqFeat = W == kPairs64 ? 64 : 128;        // rows of dQ^T that count
  constexpr int P = Rows<W>::kPlanes;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  const uint32_t sK = smem_u32(smem), sV = sK + TB;
  constexpr int NS = kScoreStages<W>, NR = kRowStages<W>;
  const uint32_t sQ0 = sK + 2 * TB, sD0 = sQ0 + NR * HB;       // [NR] stages each
  const uint32_t sPd = sD0 + NR * HBd;                         // [P][128 keys][64 queries] bf16
  const uint32_t sDq = sPd + P * kTileBytes;                   // [4 warps][kDqRows queries][32 features] fp32
  float* sLse = reinterpret_cast<float*>(smem + (sDq - sK) + kDqRows<W> * 512);   // [4][64]
  float* sDbar = sLse + 256;                                   // [4][64]
  float* sG = sDbar + 256;                                     // [2][2][128] sums of dk_share
  float* sGh = sG + 512;                                       // PASS 2: [4][64] ghat of the queries
  uint64_t* bars = reinterpret_cast<uint64_t*>(sGh + 256);
  Ctl* ctl = reinterpret_cast<Ctl*>(bars + 12);
  const uint32_t kfull = smem_u32(bars), qfull = smem_u32(bars + 1);           // qfull[4]
  const uint32_t sdone = smem_u32(bars + 5), tiles = smem_u32(bars + 7), dqdone = smem_u32(bars + 9);   // [2], [2]

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, wg = tid >> 7, row = tid & 127;
  const int warp_u = uniform_warp();
  const uint32_t lead = elect_one();
  const int nqb = (g.tq + kTileRows - 1) / kTileRows;
  const int ncb = (g.tq + kCarryRows - 1) / kCarryRows;
  const int n = (int)(blockIdx.x % g.n);
  const int jb = (int)(blockIdx.x / g.n);
  const int k0 = jb * kTileRows;
  const int nhalf = 2 * (nqb - jb);                // 64-query blocks 2 nqb - 1 .. 2 jb, visited in this order
  const int64_t row_base = (int64_t)n * g.tq;
  const int ja = k0 + row;
  const bool dead = ja >= g.tk;

  auto load_stats = [&](int hb, float* lse, float* dbar, float* gh) {      // of query 64 hb + row % 64
    const int i = hb * 64 + (row & 63);
    *lse = load_lse<BID>(rmax, rden, row_base, i, g.tq, g.lshift);
    *dbar = i < g.tq ? dbarp[row_base + i] : 0.f;
    *gh = PASS == 2 && i < g.tq ? ghat[row_base + i] : 0.f;
  };

  if (tid == 0) {
    ctl->abort = 0;
    for (int i = 0; i < 7; ++i) mbar_init(kfull + 8 * i, 1);      // kfull, qfull[4], sdone[2]
    mbar_init(tiles, 8);
    mbar_init(tiles + 8, 8);
    mbar_init(dqdone, 1);
    fence_barrier_init();
  }
  __syncwarp();
  if (warp == 0) tmem_alloc(smem_u32(&ctl->tmem), 512);
  if (wg == 0) {                                     // of the first two half-steps (nhalf >= 2)
    float l, db, gh;
    load_stats(2 * nqb - 1 - (row >> 6), &l, &db, &gh);
    sLse[row] = l;
    sDbar[row] = db;
    if (PASS == 2) sGh[row] = gh;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = uniform(ctl->tmem);
  // score stage s at tS + 128 s and tDOV + 128 s
  const uint32_t tS = tmem, tDOV = tmem + 64, tDV = tmem + 128 * NS, tDK = tDV + Rows<W>::kCols, tDQ = tDK + Rows<W>::kCols;
  const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
  if (wg < 2) {
    // dV and dK start from zero, so that every MMA into them accumulates
    uint32_t z[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) z[c] = 0u;
#pragma unroll
    for (int c = 0; c < Rows<W>::kCols / 16; ++c) tmem_st16((wg == 0 ? tDV : tDK) + lane_base + 16 * c, z);
    tmem_st_wait();
  }
  auto load_stage = [&](int h) {                     // one lane: q and do' of half-step h
    const int st = h % NR, r0 = (2 * nqb - 1 - h) * 64;
    mbar_expect_tx(qfull + 8 * st, HB + HBd);
    tma_load_rows<W>(sQ0 + HB * st, &map_q, r0, n, qfull + 8 * st, HSub);
    tma_load_rows<W, Rows<W>::kDoSub>(sD0 + HBd * st, &map_do, r0, n, qfull + 8 * st, HSub);
  };
  if (tid == 256) {
    mbar_expect_tx(kfull, 2 * TB);
    tma_load_rows<W>(sK, &map_k, k0, n, kfull);
    tma_load_rows<W>(sV, &map_v, k0, n, kfull);
    for (int h = 0; h < NR && h < nhalf; ++h) load_stage(h);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  if (wg == 2) {
    // ------------------------------------------------------------ issue, and the dQ read-out
    asm volatile("setmaxnreg.dec.sync.aligned.u32 104;");
    constexpr uint32_t id_s = instr_desc(128, 64, 0, 0);     // scores: both operands K-major
    constexpr uint32_t id_kd = instr_desc(128, Rows<W>::kCols, 0, 1);   // dV, dK: A from TMEM (M = keys), B MN-major
    constexpr uint32_t id_qd = instr_desc(128, 64, 1, 1);    // dQ^T: A and B MN-major
    const Desc dKk = make_desc(sK, 16, 1024), dVk = make_desc(sV, 16, 1024);
    const Desc dKm = make_desc(sK, kTileBytes, 1024);
    const Desc dPm = make_desc(sPd, kTileBytes, 1024);
    auto issue_scores = [&](int h) {
      const int st = h % NR;
      const uint32_t col = NS == 2 ? 128 * (h & 1) : 0;
      mbar_wait_warp(qfull + 8 * st, (h / NR) & 1, ctl, &g_status, kErrWaitTma);
      tc_fence_after();
      mma_scores_wide<W>(lead, tS + col, dKk, kTileBytes, make_desc(sQ0 + HB * st, 16, 1024), HSub, id_s);
      mma_dov_wide<W>(lead, tDOV + col, dVk, kTileBytes, make_desc(sD0 + HBd * st, 16, 1024), HSub, id_s);
    };
    if (warp_u == 8) {
      mbar_wait_warp(kfull, 0, ctl, &g_status, kErrWaitTma);
      for (int h = 0; h < NS; ++h) {
        issue_scores(h);
        mma_commit(lead, sdone + 8 * h);
      }
    }
    __syncwarp();
    for (int h = 0; h < nhalf; ++h) {
      const int st = h % NR, sc = NS == 2 ? h & 1 : 0;      // stage of q and do', stage of the scores
      if (warp_u == 8) {
        mbar_wait_warp(tiles + 8 * sc, (h / NS) & 1, ctl, &g_status, kErrWaitTile);
        tc_fence_after();
        const Desc dQm = make_desc(sQ0 + HB * st, HSub, 1024), dDm = make_desc(sD0 + HBd * st, HSub, 1024);
#pragma unroll
        for (int pl = 0; pl < P; ++pl)
#pragma unroll
          for (int kq = 0; kq < 4; ++kq) {                    // contraction over the 64 queries, 16 each
            const uint32_t col = 128 * sc + 32 * (kq >> 1) + 16 * pl + 8 * (kq & 1);
            mma_ts(lead, tDV, tS + col, dDm, 128 * kq, id_kd, 1);
            if (Rows<W>::kDoParts == 2 && pl == 0)            // share_hi do'_lo; share_lo do'_lo is left out (2^-18)
              mma_ts(lead, tDV, tS + col, dDm, (HSub >> 4) * Rows<W>::kSub + 128 * kq, id_kd, 1);
            mma_ts(lead, tDK, tDOV + col, dQm, 128 * kq, id_kd, 1);
          }
        if (h + NS < nhalf) issue_scores(h + NS);
        mma_commit(lead, sdone + 8 * sc);
#pragma unroll
        for (int pl = 0; pl < P; ++pl)
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)                      // contraction over the 128 keys
            mma_ss(lead, tDQ, dKm, 128 * kk, dPm, 1024 * pl + 128 * kk, id_qd, (pl > 0 || kk > 0));
        mma_commit(lead, dqdone);
        if (NS == 1) {
          if (h + 2 < nhalf) {
            // the products that read this stage come before the scores of h + 1, whose commit covers them
            mbar_wait_warp(sdone, (h + 1) & 1, ctl, &g_status, kErrWaitMma);
            if (lead) load_stage(h + 2);
          }
        } else if (h >= 1 && h + 3 < nhalf) {
          // the products of h - 1 have completed once the commit behind them has: their stage takes h + 3
          mbar_wait_warp(sdone + 8 * ((h - 1) & 1), ((h - 1) / 2 + 1) & 1, ctl, &g_status, kErrWaitMma);
          if (lead) load_stage(h + 3);
        }
      }
      __syncwarp();
      // dQ^T of the half-step's 64 queries: lane = feature.  Each warp stages its 32 features and
      // adds them to dq_main with one tensor reduction.
      if (lane == 0) mbar_wait(dqdone, h & 1, ctl, &g_status, kErrWaitMma);
      __syncwarp();
      tc_fence_after();
      const int q0 = (2 * nqb - 1 - h) * 64, w4 = warp & 3;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        constexpr bool kEach = kDqRows<W> == 32;        // staged and reduced 32 queries at a time
        if (32 * w4 >= kDqFeat) break;
        if (kEach || c == 0) {
          if (lane == 0) tma_wait_read_all();           // the previous reduction has read this warp's staging
          __syncwarp();
        }
        const uint32_t stage = sDq + w4 * (kDqRows<W> * 128), off = kEach ? 0 : 32 * c;
        float x[32];
        tmem_ld32(tDQ + lane_base + 32 * c, x);
        tmem_ld_wait(x);
#pragma unroll
        for (int e = 0; e < 32; ++e)
          asm volatile("st.shared.f32 [%0], %1;" ::"r"(stage + lane * 4 + (off + e) * 128), "f"(x[e] * g.scale) : "memory");
        if (kEach || c == 1) {
          fence_async_smem();
          __syncwarp();
          const int qr = q0 + (kEach ? 32 * c : 0);
          if (lane == 0 && qr < g.tq)                   // a reduction never starts behind the last row
            tma_reduce_add_tile(&map_dq, stage, W == kSplit ? 32 * (w4 & 1) : 32 * w4, qr, n);
        }
      }
      tc_fence_before();
      __syncwarp();
      asm volatile("bar.sync 2, 128;" ::: "memory");    // every warp has read the tile: the next one may be issued
      tc_fence_after();
    }
    if (lane == 0) tma_wait_read_all();
    __syncwarp();
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 200;");
    // ------------------------------------------------------------ the compute warps
    const int cw = 32 * (1 - wg);                    // this warpgroup's queries of a half-step
    auto load_edge = [&](int h) {                    // demand in front of this thread's 32 queries of half-step h
      if (dead || SHARE == kShareNone) return 0.f;   // no share step: no demand is read
      const int rb = 2 * (2 * nqb - 1 - h) + (wg == 0 ? 1 : 0);
      return rb < ncb ? carry[((int64_t)n * ncb + rb) * g.tk + ja] : total[(int64_t)n * g.tk + ja];
    };
    float sigma = 0.f;                               // suffix of dk_share behind the half-step
    float incl = load_edge(0);
    float incl_next = load_edge(1);                  // nhalf >= 2
    const uint32_t tcol = lane_base + cw;
    for (int h = 0; h < nhalf; ++h) {
      const int b = h & 1, hb = 2 * nqb - 1 - h;
      const uint32_t sc = NS == 2 ? 128 * b : 0;       // columns of the score stage
      float incl_next2 = 0.f, nx_lse = INFINITY, nx_dbar = 0.f, nx_gh = 0.f;
      if (h + 2 < nhalf) incl_next2 = load_edge(h + 2);
      // statistics go two half-steps ahead: one barrier of the compute warps lies between their store and their use
      const bool fetch = wg == 0 && row < 64 && h + 2 < nhalf;
      if (fetch) load_stats(hb - 2, &nx_lse, &nx_dbar, &nx_gh);
      mbar_wait_warp(sdone + (NS == 2 ? 8 * b : 0), (h / NS) & 1, ctl, &g_status, kErrWaitMma);
      tc_fence_after();
      float vs[32], vd[32];
      tmem_ld32(tS + sc + tcol, vs);
      tmem_ld32(tDOV + sc + tcol, vd);
      tmem_ld_wait(vs);
      tmem_ld_wait(vd);
      const int iq0 = hb * 64 + cw;                   // position of this thread's first query
      const bool masked = dead || hb * 64 < k0 + kTileRows - 1 || iq0 + 32 > g.tq;
      const float4* Lse4 = reinterpret_cast<const float4*>(sLse + (h & 3) * 64 + cw);
      const float4* Dbar4 = reinterpret_cast<const float4*>(sDbar + (h & 3) * 64 + cw);
      uint32_t shp[16 * P];
      // warpgroup 0 (queries 32..63) knows the suffix of dk_share behind its queries; warpgroup 1 starts
      // from zero and adds p * (the suffix warpgroup 0 ends with) afterwards: dp is linear in it
      float R = wg == 0 ? sigma : 0.f;
      auto chunk = [&](auto mask_tag) {
        reverse_sweeps<BID, SHARE, decltype(mask_tag)::value, true, true, PASS>(
            vs, vd, shp, R, incl + g.eps, Lse4, Dbar4, g, dead, ja - iq0, g.tq - iq0,
            reinterpret_cast<const float4*>(sGh + (h & 3) * 64 + cw));
      };
      if (masked) chunk(std::true_type{}); else chunk(std::false_type{});
      sG[(b * 2 + wg) * 128 + row] = R;
      tmem_st16(tS + sc + tcol, shp);                  // the shares, over score columns this thread has consumed
      tmem_st16(tS + sc + tcol + 16, shp + 16);
      asm volatile("bar.sync 1, 256;" ::: "memory");   // the compute warps
      const float rother = sG[(b * 2 + (1 - wg)) * 128 + row];
      const float fix = wg == 1 ? rother : 0.f;
      sigma = R + rother;                              // the suffix behind the next half-step
      // the dQ products of the previous half-step read the pdp buffer that is written next
      if (h >= 1) mbar_wait_warp(dqdone, (h - 1) & 1, ctl, &g_status, kErrWaitMma);
      {
        uint32_t pdt[16 * P];
#pragma unroll
        for (int e8 = 0; e8 < 4; ++e8) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int e = e8 * 8 + 2 * u;
            const float2 f2 = fma2(make_float2(vs[e], vs[e + 1]), make_float2(fix, fix), make_float2(vd[e], vd[e + 1]));
            vd[e] = f2.x;
            vd[e + 1] = f2.y;
            pdt[e8 * 4 + u] = pack_bf16(f2.x, f2.y);
            pdt[16 + e8 * 4 + u] = pack_bf16_rest(f2.x, f2.y, pdt[e8 * 4 + u]);
          }
#pragma unroll
          for (int pl = 0; pl < P; ++pl) {              // [key][query]: the MN-major B operand of dQ^T
            const uint32_t* w = pdt + 16 * pl + 4 * e8;
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sPd + kTileBytes * pl + share_chunk_offset(row, cw + e8 * 8)),
                         "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3])
                         : "memory");
          }
        }
        tmem_st16(tDOV + sc + tcol, pdt);                  // the A operand of dK (M = keys)
        tmem_st16(tDOV + sc + tcol + 16, pdt + 16);
      }
      if (fetch) {
        sLse[((h + 2) & 3) * 64 + row] = nx_lse;
        sDbar[((h + 2) & 3) * 64 + row] = nx_dbar;
        if (PASS == 2) sGh[((h + 2) & 3) * 64 + row] = nx_gh;
      }
      incl = incl_next;
      incl_next = incl_next2;
      tmem_st_wait();
      fence_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tiles + (NS == 2 ? 8 * b : 0));
      if (PASS == 0) {
        const float sum = sum_over_lanes(vd, lane);
        if (iq0 + lane < g.tq) atomicAdd(ghat + row_base + iq0 + lane, sum);
      }
    }
  }
  mbar_wait_warp(sdone + 8 * (NS - 1), (nhalf / NS) & 1, ctl, &g_status, kErrWaitMma);   // the last commit: every product
  tc_fence_after();
  if (warp < 8) {
    // lane = key: each warpgroup stores half of the columns of dk_main and dv, 32 at a time
    constexpr int kHead = Rows<W>::kHead, kHalf = kHead / 2;
    const int d = W == kSplit ? g.d : kHead;
    auto fetch32 = [&](uint32_t t, float* a) {
      tmem_ld32(t + lane_base, a);
      tmem_ld_wait(a);
      if (W == kSplit) {                              // A X_hi + A X_lo
        float lo[32];
        tmem_ld32(t + lane_base + 64, lo);
        tmem_ld_wait(lo);
#pragma unroll
        for (int e = 0; e < 32; ++e) a[e] += lo[e];
      }
    };
#pragma unroll
    for (int c0 = 0; c0 < kHalf; c0 += 32) {
      const int col = kHalf * wg + c0;
      float a[32];
      fetch32(tDK + col, a);
#pragma unroll
      for (int e = 0; e < 32; ++e) a[e] *= g.scale;
      if (!dead) store_row32<kNarrow>(dk_main + ((int64_t)n * g.tk + ja) * kHead + col, a, 32);
      fetch32(tDV + col, a);
      if (!dead) store_row32<W>(dv + ((int64_t)n * g.tk + ja) * d + col, a, d - col);
    }
  }
  drain_if_aborted(ctl);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_free(tmem, 512);
}

// ---------------------------------------------------------------- host launchers
inline int split_operands(const SplitArgs& a, int count, int64_t rows, int d, cudaStream_t st, char* err, size_t errlen) {
  split_operands_kernel<<<dim3((unsigned)((rows * 16 + 255) / 256), (unsigned)count), 256, 0, st>>>(a, rows, d);
  return launch_status("split_operands", err, errlen);
}

struct WideMaps {
  CUtensorMap q, k, v;
};
inline int wide_maps(WideMaps* m, const void* q, const void* k, const void* v, const Geom& g, char* err, size_t errlen) {
  if (int rc = make_map(&m->q, q, g.n, g.tq, err, errlen, 128)) return rc;
  if (int rc = make_map(&m->k, k, g.n, g.tk, err, errlen, 128)) return rc;
  return make_map(&m->v, v, g.n, g.tk, err, errlen, 128);
}

// Passes 1-3 on wide rows; pk (n, t, d) fp32 is written when it is not null.
template <int W>
inline int wide_forward(const void* q, const void* k, const void* v, const Geom& g, float* rmax, float* rden,
                        float* carry, float* total, float* out, float* ssum, float* pk, cudaStream_t st, char* err,
                        size_t errlen, void (*mark)(const char*, cudaStream_t, int)) {
  WideMaps m;
  if (int rc = wide_maps(&m, q, k, v, g, err, errlen)) return rc;
  const unsigned grid = (unsigned)(g.n * ((g.tq + kTileRows - 1) / kTileRows));
  if (pk != nullptr) {
    CUtensorMap mk64;
    if (int rc = make_map(&mk64, k, g.n, g.tk, err, errlen, 128, 64)) return rc;
    auto kern = rowpass_issuer_kernel<1, float, W>;
    constexpr int smem = RowIssuer<1, W>::kBytes;
    static_assert(smem <= 232448 && 2 * smem > 233472, "one CTA (512 TMEM columns) per SM");
    if (int rc = set_smem_attr((const void*)kern, smem, err, errlen)) return rc;
    mark("tc_wide_rowstats_pk", st, 0);
    kern<<<grid, RowIssuer<1, W>::kThreads, smem, st>>>(m.q, mk64, mk64, g, rmax, rden, pk);
    mark("tc_wide_rowstats_pk", st, 1);
  } else {
    constexpr int smem = kRowstatsSmem<W>;
    if (int rc = set_smem_attr((const void*)rowstats_kernel<W>, smem, err, errlen)) return rc;
    mark("tc_wide_rowstats", st, 0);
    rowstats_kernel<W><<<grid, 256, smem, st>>>(m.q, m.k, g, rmax, rden);
    mark("tc_wide_rowstats", st, 1);
  }
  if (int rc = launch_status("tc wide rowstats", err, errlen)) return rc;
  {
    constexpr int smem = kColsumSmem<W>;
    auto kern = colsum_scan_kernel<32, kBidSoftmax, W>;
    if (int rc = set_smem_attr((const void*)kern, smem, err, errlen)) return rc;
    mark("tc_wide_colsum_scan", st, 0);
    kern<<<grid, 256, smem, st>>>(m.q, m.k, g, rmax, rden, nullptr, carry, total);
    mark("tc_wide_colsum_scan", st, 1);
  }
  if (int rc = launch_status("tc wide colsum_scan", err, errlen)) return rc;
  {
    constexpr int smem = kMainSmem<W>;
    static_assert(smem <= 232448 && 2 * smem > 233472, "one CTA (512 TMEM columns) per SM");
    auto kern = pair_demands(g) ? forward_main_async_kernel<kBidSoftmax, kShareInclusive, W, true>
                                : forward_main_async_kernel<kBidSoftmax, kShareInclusive, W, false>;
    if (int rc = set_smem_attr((const void*)kern, smem, err, errlen)) return rc;
    mark("tc_wide_forward_main", st, 0);
    kern<<<grid, kMainThreads<W>, smem, st>>>(m.q, m.k, m.v, g, rmax, rden, carry, nullptr, (const __nv_bfloat16*)v, out,
                                           ssum);
    mark("tc_wide_forward_main", st, 1);
  }
  return launch_status("tc wide forward_main", err, errlen);
}

// dq_main and dk_main: (n, t, 128), kSplit (n, t, 64); dop: (n, t, 64 kDoSub) bf16; ghat, dbarp: (n, t).
template <int W>
inline int wide_backward(const void* q, const void* k, const void* v, const Geom& g, const void* dout, int dout_dtype,
                         const float* out, const float* rmax, const float* rden, const float* carry,
                         const float* total, const float* ssum, const float* pk, float* dq_main, float* dk_main,
                         void* dop, float* ghat, float* dbarp, void* dq, void* dk, void* dv, cudaStream_t st,
                         char* err, size_t errlen, void (*mark)(const char*, cudaStream_t, int)) {
  using TOut = std::conditional_t<W == kSplit, float, __nv_bfloat16>;
  constexpr int kHead = Rows<W>::kHead;
  WideMaps m;
  if (int rc = wide_maps(&m, q, k, v, g, err, errlen)) return rc;
  CUtensorMap mq64, md64, mdq;
  if (int rc = make_map(&mq64, q, g.n, g.tq, err, errlen, 128, 64)) return rc;
  if (int rc = make_map(&md64, dop, g.n, g.tq, err, errlen, 64 * Rows<W>::kDoSub, 64)) return rc;
  if (int rc = make_map_f32(&mdq, dq_main, g.n, g.tq, err, errlen, kHead, kDqRows<W>, false)) return rc;
  const int64_t rows = g.n * g.tq;
  const unsigned grid = (unsigned)(g.n * ((g.tk + kTileRows - 1) / kTileRows));
  mark("tc_wide_backward_prep", st, 0);
  if (dout_dtype == 0)
    wide_backward_prep_kernel<float, W><<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(
        (const float*)dout, out, ssum, g.eps, rows, g.d, dbarp, (__nv_bfloat16*)dop, ghat, dq_main);
  else
    wide_backward_prep_kernel<__nv_bfloat16, W><<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(
        (const __nv_bfloat16*)dout, out, ssum, g.eps, rows, g.d, dbarp, (__nv_bfloat16*)dop, ghat, dq_main);
  mark("tc_wide_backward_prep", st, 1);
  if (int rc = launch_status("tc wide backward_prep", err, errlen)) return rc;
  {
    constexpr int smem = kBwdWideSmem<W>;
    static_assert(smem <= 232448 && 2 * smem > 233472, "the wide reverse pass runs one CTA per SM");
    auto kern = wide_backward_main_kernel<W, TOut>;
    if (int rc = set_smem_attr((const void*)kern, smem, err, errlen, kBwdRegs)) return rc;
    mark("tc_wide_backward_main", st, 0);
    kern<<<grid, kBwdThreads, smem, st>>>(mq64, m.k, m.v, md64, mdq, g, rmax, rden, dbarp, carry, total, dk_main,
                                          (TOut*)dv, ghat);
    mark("tc_wide_backward_main", st, 1);
  }
  if (int rc = launch_status("tc wide backward_main", err, errlen)) return rc;
  {
    constexpr int smem = kCorrKey64Smem<W>;
    auto kern = backward_key_correction64_kernel<W, TOut>;
    if (int rc = set_smem_attr((const void*)kern, smem, err, errlen)) return rc;
    mark("tc_wide_backward_key_correction", st, 0);
    kern<<<grid, 256, smem, st>>>(m.q, m.k, g, rmax, rden, ghat, dk_main, (TOut*)dk);
    mark("tc_wide_backward_key_correction", st, 1);
  }
  if (int rc = launch_status("tc wide backward_key_correction", err, errlen)) return rc;
  mark("tc_wide_dq_from_pk", st, 0);
  if (W == kSplit) {
    const int64_t n4 = rows * (g.d / 4);
    split_dq_from_pk_kernel<<<(unsigned)((n4 + 255) / 256), 256, 0, st>>>(dq_main, pk, ghat, (float*)dq, rows, g.d);
  } else {
    const int64_t n4 = rows * (kHead / 4);
    dq_from_pk_kernel<kHead><<<(unsigned)((n4 + 255) / 256), 256, 0, st>>>(dq_main, pk, ghat, (__nv_bfloat16*)dq, n4);
  }
  mark("tc_wide_dq_from_pk", st, 1);
  return launch_status("tc wide dq_from_pk", err, errlen);
}

// ---------------------------------------------------------------- f(a) / rowsum(f) bids of bf16 heads of 64
// relu, relu2, softplus.  The row mass and the column sums only need scores and run on the narrow kernels.
// softplus / inclusive at B4 H8 T8192, forward + backward on one B200: 39.2 ms on the tile kernels -> 7.1 ms (row mass
// 0.54, column sums 0.67, main pass 1.25, ghat 1.6, reverse pass 3.0); outputs 1.3e-4 -> 1.5e-6 off 64 bits (2-norm),
// gradients 1.7e-3 before and after.  Bound by the special-function unit (four operations per score in the reverse
// passes, three in the main pass) and, with one CTA per SM in the two product passes, by the hand-over between scores,
// arithmetic and products.
inline int mass_forward_main(const void* q, const void* k, const void* v, const Geom& g, const float* rmax,
                             const float* rden, const float* carry, float* out, float* ssum, cudaStream_t st, char* err,
                             size_t errlen) {
  CUtensorMap mq, mk, mv;
  if (int rc = make_map(&mq, q, g.n, g.tq, err, errlen)) return rc;
  if (int rc = make_map(&mk, k, g.n, g.tk, err, errlen)) return rc;
  if (int rc = make_map(&mv, v, g.n, g.tk, err, errlen)) return rc;
  constexpr int smem = kMainSmem<kPairs64>;
  static_assert(smem <= 232448 && 2 * smem > 233472, "one CTA (512 TMEM columns) per SM");
  const unsigned grid = (unsigned)(g.n * ((g.tq + kTileRows - 1) / kTileRows));
  DIL_TC_MASS_BID(g, DIL_TC_SHARE(g, DIL_TC_PAIR(g, SHARE, {
    auto kern = forward_main_async_kernel<BID, SHARE, kPairs64, PAIR>;
    if (int rc = set_smem_attr((const void*)kern, smem, err, errlen)) return rc;
    kern<<<grid, kMainThreads<kPairs64>, smem, st>>>(mq, mk, mv, g, rmax, rden, carry, nullptr, (const __nv_bfloat16*)v, out, ssum);
  })))
  return launch_status("tc forward_main", err, errlen);
}

// dq_main: (n, t, 64) fp32; dop: (n, t, 128) bf16; ghat, dbarp: (n, t).
inline int mass_backward(const void* q, const void* k, const void* v, const Geom& g, const float* dout, const float* out,
                         const float* rmax, const float* rden, const float* carry, const float* total,
                         const float* ssum, float* dq_main, void* dop, float* ghat, float* dbarp, void* dq, void* dk,
                         void* dv, cudaStream_t st, char* err, size_t errlen, void (*mark)(const char*, cudaStream_t, int)) {
  CUtensorMap mq, mk, mv, md, mq64, md64, mdq;
  if (int rc = make_map(&mq, q, g.n, g.tq, err, errlen)) return rc;
  if (int rc = make_map(&mk, k, g.n, g.tk, err, errlen)) return rc;
  if (int rc = make_map(&mv, v, g.n, g.tk, err, errlen)) return rc;
  if (int rc = make_map(&md, dop, g.n, g.tq, err, errlen, 128)) return rc;
  if (int rc = make_map(&mq64, q, g.n, g.tq, err, errlen, 64, 64)) return rc;
  if (int rc = make_map(&md64, dop, g.n, g.tq, err, errlen, 128, 64)) return rc;
  if (int rc = make_map_f32(&mdq, dq_main, g.n, g.tq, err, errlen, 64, kDqRows<kPairs64>, false)) return rc;
  using bf = __nv_bfloat16;
  const int64_t rows = g.n * g.tq;
  const unsigned grid = (unsigned)(g.n * ((g.tk + kTileRows - 1) / kTileRows));
  mark("tc_backward_prep", st, 0);
  wide_backward_prep_kernel<float, kPairs64><<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(
      dout, out, ssum, g.eps, rows, 64, dbarp, (bf*)dop, ghat, dq_main);
  mark("tc_backward_prep", st, 1);
  if (int rc = launch_status("tc backward_prep", err, errlen)) return rc;
  // ghat first, also without a share step, where it is zero in exact arithmetic: do' and the shares are rounded, and a
  // factor of 1 / (row mass) would multiply what that leaves of it
  DIL_TC_MASS_BID(g, DIL_TC_SHARE(g, {
    auto kern = backward_main_kernel<BID, SHARE, 1>;
    if (int rc = set_smem_attr((const void*)kern, kBwdSmem, err, errlen, kBwdRegs)) return rc;
    mark("tc_backward_ghat", st, 0);
    kern<<<grid, kBwdThreads, kBwdSmem, st>>>(mq, mk, md, mdq, g, (const bf*)v, rmax, rden, dbarp, carry, total, nullptr,
                                              nullptr, nullptr, ghat);
    mark("tc_backward_ghat", st, 1);
    if (int rc = launch_status("tc backward_ghat", err, errlen)) return rc;
    auto main = wide_backward_main_kernel<kPairs64, bf, BID, SHARE, 2>;
    constexpr int smem = kBwdWideSmem<kPairs64>;
    static_assert(smem <= 232448 && 2 * smem > 233472, "the wide reverse pass runs one CTA per SM");
    if (int rc = set_smem_attr((const void*)main, smem, err, errlen, kBwdRegs)) return rc;
    mark("tc_backward_main", st, 0);
    main<<<grid, kBwdThreads, smem, st>>>(mq64, mk, mv, md64, mdq, g, rmax, rden, dbarp, carry, total, (bf*)dk, (bf*)dv,
                                          ghat);
    mark("tc_backward_main", st, 1);
  }))
  if (int rc = launch_status("tc backward_main", err, errlen)) return rc;
  const int64_t n4 = rows * kHeadDim / 4;
  mark("tc_cast_dq", st, 0);
  cast_dq_kernel<<<(unsigned)((n4 + 255) / 256), 256, 0, st>>>(dq_main, (bf*)dq, n4);
  mark("tc_cast_dq", st, 1);
  return launch_status("tc cast_dq", err, errlen);
}

}  // namespace tc
}  // namespace dil
