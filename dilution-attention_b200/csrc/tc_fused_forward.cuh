// Key-stationary forward of whole rows on the tensor cores: passes 2 and 3 in one sweep
// (the reference's training forward, _dilution_key_forward + _dilution_normalize,
// kernels.py:200-248, does the same on its side of the fence).
//
// A CTA owns 512 keys, 128 per compute warpgroup (lane = key), and walks the queries that can see them in causal
// order, 64 at a time.  The demand of a key stays in its thread for the whole sweep, so no checkpoint is read; the checkpoints that
// the backward needs (every 32 query rows, or 64) and the demand totals are stored on the way.  Per half tile of 64 queries and
// warpgroup:
//   S^T  = K Q^T            A = the keys' rows in TMEM, written there once: 4 MMAs of N = 64
//   p, demand, share        64 queries per thread, the arithmetic of forward_main_kernel but for the demand, which is an output
//                           here: bids of 32 queries are summed from zero and folded into a compensated total
//   O^T | rs                = [V | 1 0 .. 0]^T share, M = 64 features, the row sums and 63 rows of zeros (as 64 copies of the sums
//                           they cost power, which long rows are short of: 5.08 -> 5.00 ms), K = 128 keys, N = 64: 8 MMAs into a
//                           FRESH tile per half tile that all four warpgroups add to
// and the tile is added to `out` / `ssum` in global memory: two warps of a fifth warpgroup (lane = feature) move it from TMEM
// to a staging tile and issue a TMA tensor reduction each, the row sums go by atomics from the third.  `out` and `ssum`
// therefore start at zero and a small kernel divides at the end.  One exponential and one QK^T sweep per score less than
// column-sum pass + query-stationary main pass.
//
// Four warpgroups are four warps per scheduler.  They fit because the keys are a TMEM operand and O comes out transposed
// (64 columns): S^T 4 x 64, K 4 x 32, O^T 2 x 64 = 512 columns, V + ones + shares + q + staging = 192 KB.  Two warpgroups of 128
// keys with S^T double-buffered took 6.5 ms at n = 64, T = 16384 and left the special-function unit idle
// whenever both waited; output tiles are added half as often.  640 threads, one CTA per SM.  Every wait is bounded.
//
// The fifth warpgroup's last warp does nothing but issue every TMA copy and MMA: as one of the four that move O out (two took the
// row sums then) it was in the middle of that whenever a warpgroup wanted its next scores.  Moved out of the read-out, at
// n = 64, T = 16384 5.9 -> 4.7 ms, n = 16, T = 131072 86 -> 75 ms, n = 384, T = 1024 279 -> 251 us, n = 16, T = 1777 (128 keys
// per CTA) 70 -> 55 us.  What is left: half of the special-function unit's rate; long rows run at the card's power limit.
#pragma once

#include "tc_kernels.cuh"

namespace dil {
namespace tc {

constexpr int kFusedRing = 4;                              // half tiles of q
constexpr int kFusedRegs = 96;                             // per thread at launch of four compute warpgroups, by the launch bounds
static_assert(4 * 104 + 64 <= 5 * kFusedRegs, "setmaxnreg hands out what the block was launched with");
// V[G] ones shares[G] | Q[4] (8 KB each) | staging (16 KB) | lse [4][64] | barriers
template <int G> constexpr int kFusedSmem = (2 * G + 1) * kTileBytes + kFusedRing * kTileBytes / 2 + kTileBytes + 1024 + 256 + 1024;

// G: compute warpgroups of 128 keys.  CR: query rows per checkpoint.  BID, with the inclusive share step: softmax, the sigmoid's form, or
// expshift, which has no row statistics (every log-sum-exp is the shift's logarithm) and whose bids have no upper end: an exponential may
// overflow, and so may a demand, which then stays infinite while the rows behind it are finite.
template <int G, int CR, bool PAIR, int BID = kBidSoftmax>
__global__ void __launch_bounds__(128 * (G + 1), G == 1 ? 2 : 1) forward_fused_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_v,
    const __grid_constant__ CUtensorMap map_out, Geom g, const __nv_bfloat16* __restrict__ k,
    const float* __restrict__ rmax, const float* __restrict__ rden, float* __restrict__ carry,
    float* __restrict__ total, float* __restrict__ ssum) {
  constexpr int R = kFusedRing, kTmem = G == 1 ? 256 : 512;
  constexpr uint32_t HB = kTileBytes / 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  const uint32_t sV = smem_u32(smem), sOnes = sV + G * kTileBytes;           // A of O^T: [V | 1 0 .. 0], MN-major
  uint8_t* ones_ptr = smem + G * kTileBytes;
  const uint32_t sSh = sOnes + kTileBytes;                                   // [G][128 keys][64 queries]
  const uint32_t sQ = sSh + G * kTileBytes, sStage = sQ + R * HB;            // staging: [2 warps][64 queries][32 features] fp32
  float* sL = reinterpret_cast<float*>(smem + (sStage - sV) + kTileBytes);   // [4][64] -lse of a half tile's queries
  uint64_t* bars = reinterpret_cast<uint64_t*>(sL + 256);
  const uint32_t vfull = smem_u32(bars), qfull = vfull + 8, ofull = qfull + 8 * R;            // 1, [R], [2]
  const uint32_t sdone = ofull + 16, odone = sdone + 8 * G, sfree = odone + 8 * G, shready = sfree + 8 * G,   // [G] each
                 ofree = shready + 8 * G;                                                                  // [2]
  Ctl* ctl = reinterpret_cast<Ctl*>(bars + 5 + R + 4 * G);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, wg = tid >> 7, row = tid & 127;
  const int warp_u = uniform_warp();
  const uint32_t lead = elect_one();
  const int ncb = (g.tq + CR - 1) / CR;
  const int n = (int)(blockIdx.x % g.n);
  const int k0 = (int)(blockIdx.x / g.n) * (G * kTileRows);
  const int h0 = k0 / 64, nh = (g.tq + 63) / 64;          // half tiles of queries; warpgroup w sees those from h0 + 2 w on
  const int groups = min(G, (g.tk - k0 + kTileRows - 1) / kTileRows);
  const int64_t row_base = (int64_t)n * g.tq;
  // what a query's scores are added to: minus its log-sum-exp, or plus (the sigmoid's exponent is lse - z)
  auto offset = [&](float lse) { return BID == kBidSigmoid ? lse : -lse; };

  if (tid == 0) {
    ctl->abort = 0;
    for (int i = 0; i < 3 + R + 2 * G; ++i) mbar_init(vfull + 8 * i, 1);
    for (int i = 0; i < 2 * G; ++i) mbar_init(sfree + 8 * i, 4);
    for (int i = 0; i < 2; ++i) mbar_init(ofree + 8 * i, 3);
    fence_barrier_init();
  }
  __syncwarp();
  if (warp == 0) tmem_alloc(smem_u32(&ctl->tmem), kTmem);
  if (wg == G) {
    sL[row] = offset(load_lse<BID>(rmax, rden, row_base, h0 * 64 + row, g.tq, g.lshift));    // of the first three half tiles
  } else if (wg == 0) {
    if (row < 64) sL[128 + row] = offset(load_lse<BID>(rmax, rden, row_base, h0 * 64 + 128 + row, g.tq, g.lshift));
#pragma unroll
    for (int c = 0; c < 8; ++c)
      reinterpret_cast<uint4*>(ones_ptr)[row * 8 + c] = make_uint4(c == (row & 7) ? 0x3f80u : 0u, 0u, 0u, 0u);
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = uniform(ctl->tmem);
  const uint32_t tS = tmem, tK = tmem + 64 * G, tO = tmem + 96 * G;        // O^T tile b at tO + 64 b
  const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
  const int ja = k0 + wg * kTileRows + row;
  const bool dead = ja >= g.tk;
  if (wg < G) {
    // this key's row as an A operand: two head-dim elements per 32-bit column
    uint32_t w[32];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      uint4 x = make_uint4(0u, 0u, 0u, 0u);
      if (!dead) x = reinterpret_cast<const uint4*>(k + ((int64_t)n * g.tk + ja) * kHeadDim)[c];
      w[4 * c] = x.x; w[4 * c + 1] = x.y; w[4 * c + 2] = x.z; w[4 * c + 3] = x.w;
    }
    __syncwarp();
    tmem_st16(tK + 32 * wg + lane_base, w);
    tmem_st16(tK + 32 * wg + lane_base + 16, w + 16);
    tmem_st_wait();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  if (wg == G) {
    // ------------------------------------------------------------ issue (its last warp), and the O read-out
    if (G == 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    if (warp_u == 4 * G + 3) {
      constexpr uint32_t id_s = instr_desc(128, 64, 0, 0);     // scores: A from TMEM, B K-major
      constexpr uint32_t id_o = instr_desc(128, 64, 1, 1);     // O^T: A and B MN-major
      const Desc dQ = make_desc(sQ, 16, 1024), dSh = make_desc(sSh, kTileBytes, 1024);
      auto load_q = [&](int h) {
        const int st = (h - h0) % R;
        if (!lead) return;
        mbar_expect_tx(qfull + 8 * st, HB);
        tma_load_tile(sQ + HB * st, &map_q, h * 64, n, qfull + 8 * st);
      };
      auto issue_scores = [&](int w, int h) {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          mma_ts(lead, tS + 64 * w, tK + 32 * w + 8 * kk, dQ, (HB >> 4) * ((h - h0) % R) + 2 * kk, id_s, kk > 0);
        mma_commit(lead, sdone + 8 * w);
      };
      if (lead) {
        mbar_expect_tx(vfull, groups * kTileBytes);
        for (int w = 0; w < groups; ++w) tma_load_tile(sV + kTileBytes * w, &map_v, k0 + w * kTileRows, n, vfull);
      }
      for (int h = h0; h < h0 + R && h < nh; ++h) load_q(h);
      mbar_wait_warp(qfull, 0, ctl, &g_status, kErrWaitTma);
      tc_fence_after();
      issue_scores(0, h0);
      mbar_wait_warp(vfull, 0, ctl, &g_status, kErrWaitTma);
      for (int h = h0; h < nh; ++h) {
        const int u = h - h0;
        // O^T of h - 2 is out of its buffer, and the lse of h + 1 are in place
        if (u >= 2) mbar_wait_warp(ofree + 8 * (u & 1), ((u >> 1) + 1) & 1, ctl, &g_status, kErrWaitDrain);
        if (h + 1 < nh) {
          // scores of h + 1, as soon as a warpgroup has taken those of h out of TMEM
          mbar_wait_warp(qfull + 8 * ((u + 1) % R), ((u + 1) / R) & 1, ctl, &g_status, kErrWaitTma);
          for (int w = 0; w < groups; ++w) {
            const int t = u - 2 * w;                           // the warpgroup's own count of half tiles
            if (t + 1 < 0) break;
            if (t >= 0) mbar_wait_warp(sfree + 8 * w, t & 1, ctl, &g_status, kErrWaitTile);
            tc_fence_after();
            issue_scores(w, h + 1);
          }
        }
        for (int w = 0; w < groups; ++w) {
          const int t = u - 2 * w;
          if (t < 0) break;
          mbar_wait_warp(shready + 8 * w, t & 1, ctl, &g_status, kErrWaitTile);
          tc_fence_after();
          const Desc dVw = make_desc(sV + kTileBytes * w, sOnes - sV - kTileBytes * w, 1024);
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            mma_ss(lead, tO + 64 * (u & 1), dVw, 128 * kk, dSh, 1024 * w + 128 * kk, id_o, w > 0 || kk > 0);
          mma_commit(lead, odone + 8 * w);
        }
        mma_commit(lead, ofull + 8 * (u & 1));
        if (h + R < nh) load_q(h + R);                         // every share of h exists, so its scores are complete
      }
      __syncwarp();
    } else {
      // O^T of half tile h, lane = feature (and the row sums on the lanes behind them), to global memory.  On the way, the
      // lse of h + 3: the issuing warp waits for this tile's release before it issues the scores of h + 3, and the hand-over of
      // h, which ofull waits for, lies behind the last use of the slot (h - 1).
      for (int h = h0; h < nh; ++h) {
        float nx_max = INFINITY, nx_den = 1.f;
        const int i3 = (h + 3) * 64 + row;
        const bool fetch = row < 64 && h + 3 < nh;
        if (fetch && i3 < g.tq) {
          if (BID != kBidSoftmax) {
            nx_max = g.lshift;
          } else {
            nx_max = rmax[row_base + i3];
            nx_den = rden[row_base + i3];
          }
        }
        const int u = h - h0, w4 = warp & 3;
        if (lane == 0) mbar_wait(ofull + 8 * (u & 1), (u >> 1) & 1, ctl, &g_status, kErrWaitMma);
        __syncwarp();
        tc_fence_after();
        if (fetch) sL[64 * ((u + 3) & 3) + row] = offset(nx_max + log2f(nx_den));
        __syncwarp();
        const uint32_t tOb = tO + 64 * (u & 1) + lane_base;
        const uint32_t stage = sStage + HB * w4;
        float rs[2] = {0.f, 0.f};
        if (w4 < 2) {
          if (lane == 0) tma_wait_read_all();                  // the previous reduction has read this warp's staging
          __syncwarp();
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            float o[16];
            tmem_ld16(tOb + 16 * c, o);
            tmem_ld_wait16(o);
#pragma unroll
            for (int e = 0; e < 16; ++e)
              asm volatile("st.shared.f32 [%0], %1;" ::"r"(stage + lane * 4 + (16 * c + e) * 128), "f"(o[e]) : "memory");
          }
          fence_async_smem();
        } else {
          // the first of these lanes holds the row sums of all queries: lane l takes those of queries l and 32 + l from it
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            float o[16];
            tmem_ld16(tOb + 16 * c, o);
            tmem_ld_wait16(o);
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              const float x = __shfl_sync(0xffffffffu, o[e], 0);
              rs[c >> 1] = lane == 16 * (c & 1) + e ? x : rs[c >> 1];
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(ofree + 8 * (u & 1));       // this warp has read the tile
        if (w4 < 2) {
          if (lane == 0) tma_reduce_add_tile(&map_out, stage, 32 * w4, h * 64, n);
        } else {
          const int i = h * 64 + lane;
          if (i < g.tq) atomicAdd(ssum + row_base + i, rs[0]);
          if (i + 32 < g.tq) atomicAdd(ssum + row_base + i + 32, rs[1]);
        }
        __syncwarp();
      }
      if (lane == 0) tma_wait_read_all();
      __syncwarp();
    }
  } else {
    if (G == 4) asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    // ------------------------------------------------------------ the compute warps: lane = key
    const uint32_t tSw = tS + 64 * wg + lane_base;
    const uint32_t sShw = sSh + kTileBytes * wg;
    const int kw = k0 + wg * kTileRows;
    // committed + eps in front of a chunk of 32 queries, and what its sum has rounded off: the bids of a chunk are added up from
    // zero and folded in once, so that neither thousands of roundings nor bids under half an ulp of a large demand add up
    float base = g.eps, low = 0.f;
    const float zscale = BID == kBidSigmoid ? -g.zscale : g.zscale;
    for (int h = h0 + 2 * wg; h < nh && wg < groups; ++h) {
      const int t = h - h0 - 2 * wg;
      float v0[32], v1[32];
      uint32_t pk[16];
      auto arith = [&](const float* v, int c) {
        const int q0 = h * 64 + 32 * c;
        if (CR == 32 || c == 0) {                            // checkpoint in front of the chunk's first query
          const int rb = q0 / CR;
          if (!dead && rb < ncb) carry[((int64_t)n * ncb + rb) * g.tk + ja] = base - g.eps;
        }
        float chunk_sum = 0.f;
        const float4* L4 = reinterpret_cast<const float4*>(sL + 64 * ((h - h0) & 3) + 32 * c);
        const bool masked = dead || kw + kTileRows - 1 > q0;
        auto chunk = [&](auto mask_tag) {
          constexpr bool MASK = decltype(mask_tag)::value;
#pragma unroll
          for (int e8 = 0; e8 < 4; ++e8) {
            const float4 la = L4[2 * e8], lb = L4[2 * e8 + 1];
            const float ls[8] = {la.x, la.y, la.z, la.w, lb.x, lb.y, lb.z, lb.w};
            float z[8], sh[8], dn[8];
#pragma unroll
            for (int u = 0; u < 8; u += 2) {
              const float2 z2 = fma2(make_float2(v[e8 * 8 + u], v[e8 * 8 + u + 1]), make_float2(zscale, zscale),
                                     make_float2(ls[u], ls[u + 1]));
              z[u] = z2.x;
              z[u + 1] = z2.y;
            }
            // every fourth exponential is a polynomial on the FMA pipe (7.30 -> 7.08 ms when two warps shared a scheduler), of
            // degree 5: with degree 4 the demand, an output in fp32, is off by up to 4.6e-6 instead of 2.5e-6
            // (the sigmoid's exponents are of either sign: capped, where the bid is 1e-38 and less.  Expshift's go past 128, where the
            // polynomial's scale would run into the sign: twice 2^(z - 1) up to the infinity at z = 129.  657 -> 665 us at n = 32,
            // T = 8192, 686 with every exponential from the special-function unit)
            float2 fourth;
            if (BID == kBidExpshift) {
              fourth = poly_exp2_two<5>(make_float2(min_nan(z[3] - 1.f, 128.f), min_nan(z[7] - 1.f, 128.f)));
              fourth = add2(fourth, fourth);
            } else if (BID == kBidSigmoid) fourth = poly_exp2_two<5>(make_float2(min_nan(z[3], 126.f), min_nan(z[7], 126.f)));
            else fourth = poly_exp2_two<5>(make_float2(z[3], z[7]));
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              float p = (u & 3) != 3 ? fast_exp2(z[u]) : u == 3 ? fourth.x : fourth.y;
              if (BID == kBidSigmoid) p = fast_rcp(1.f + p);
              if (MASK && (dead || ja > q0 + e8 * 8 + u)) p = 0.f;
              chunk_sum += p;
              sh[u] = p;
              dn[u] = chunk_sum;
            }
#pragma unroll
            for (int u = 0; u < 8; u += 2) {
              const float2 den = add2(make_float2(base, base), make_float2(dn[u], dn[u + 1]));
              const float2 s2 = mul2(make_float2(sh[u], sh[u + 1]), rcp_two<PAIR>(den.x, den.y));
              pk[e8 * 4 + u / 2] = pack_bf16(s2.x, s2.y);
            }
          }
        };
        if (masked) chunk(std::true_type{}); else chunk(std::false_type{});
        const float add = chunk_sum - low, sum = base + add;
        low = BID == kBidExpshift && !(sum < INFINITY) ? 0.f : (sum - base) - add;      // (inf - inf)
        base = sum;
        __syncwarp();
      };
      auto store = [&](int c) {
#pragma unroll
        for (int e8 = 0; e8 < 4; ++e8)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sShw + share_chunk_offset(row, 32 * c + 8 * e8)),
                       "r"(pk[4 * e8]), "r"(pk[4 * e8 + 1]), "r"(pk[4 * e8 + 2]), "r"(pk[4 * e8 + 3])
                       : "memory");
      };
      mbar_wait_warp(sdone + 8 * wg, t & 1, ctl, &g_status, kErrWaitMma);
      tc_fence_after();
      tmem_ld32(tSw, v0);
      tmem_ld_wait(v0);
      tmem_ld32(tSw + 32, v1);
      arith(v0, 0);
      tmem_ld_wait(v1);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(sfree + 8 * wg);            // these scores are out of TMEM
      // the products of the previous half tile have read this warpgroup's share tile
      if (t >= 1) mbar_wait(odone + 8 * wg, (t - 1) & 1, ctl, &g_status, kErrWaitMma);
      store(0);
      arith(v1, 1);
      store(1);
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(shready + 8 * wg);
    }
    if (!dead) total[(int64_t)n * g.tk + ja] = base - g.eps;
  }
  drain_if_aborted(ctl);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_free(tmem, kTmem);
}

// Zeroes what the sweep adds up (one launch where two memsets cost the host twice).
__global__ void zero_sums_kernel(float* __restrict__ out, float* __restrict__ ssum, int64_t rows) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows * (kHeadDim / 4)) return;
  reinterpret_cast<float4*>(out)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (i < rows) ssum[i] = 0.f;
}

// out = O / (rs + eps) in place, four columns per thread (grid over n*t*16 float4).
__global__ void normalize_out_kernel(float* __restrict__ out, const float* __restrict__ ssum, float eps,
                                     int64_t n4) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n4) return;
  const float inv = 1.f / (ssum[i >> 4] + eps);
  float4 x = reinterpret_cast<float4*>(out)[i];
  x.x *= inv; x.y *= inv; x.z *= inv; x.w *= inv;
  reinterpret_cast<float4*>(out)[i] = x;
}

// Compute warpgroups per CTA.  Four need blocks of 512 keys for the SMs; with fewer than 200 of them a CTA of 128 keys, two to
// an SM, is faster.  Passes 2 and 3, one / four warpgroups, in us: 384 blocks (n = 64, T = 3000) 262 / 231; 248 (n = 31, T = 4096)
// 220 / 189; 200 (n = 100, T = 768) 60.0 / 56.6; 192 (n = 24, T = 4096) 180 / 180; 144 (n = 48, T = 1536) 74 / 83; 128 (n = 16,
// T = 4096) 120 / 173.
inline int fused_groups(int64_t n, int64_t t) { return n * ((t + 511) / 512) >= 200 ? 4 : 1; }

// Passes 2 and 3 of a call over whole rows (q_off = 0, tq = tk) in one
// key-stationary sweep.  carry: (n, ceil(t/32 or t/64), t); total: (n, t); out: (n, t, 64) fp32; ssum: (n, t).
inline int forward_fused(const void* q, const void* k, const void* v, const Geom& g, const float* rmax,
                         const float* rden, float* carry, float* total, float* out, float* ssum,
                         cudaStream_t st, char* err, size_t errlen) {
  CUtensorMap mq, mv, mo;
  if (int rc = make_map(&mq, q, g.n, g.tq, err, errlen, kHeadDim, 64)) return rc;
  if (int rc = make_map(&mv, v, g.n, g.tk, err, errlen)) return rc;
  if (int rc = make_map_f32(&mo, out, g.n, g.tq, err, errlen, kHeadDim, 64, false)) return rc;
  if ((uintptr_t)k & 15) {
    snprintf(err, errlen, "bf16 tensor-core path needs 16-byte aligned q/k/v");
    return 1;
  }
  const int64_t rows = g.n * g.tq;
  zero_sums_kernel<<<(unsigned)((rows * (kHeadDim / 4) + 255) / 256), 256, 0, st>>>(out, ssum, rows);
  auto launch = [&](auto groups_c, auto cr_c, auto pair_c, auto bid_c) -> int {
    constexpr int G = decltype(groups_c)::value, smem = kFusedSmem<G>;
    static_assert(smem <= 232448 && (G > 1 || 2 * (smem + 1024) <= 233472), "one or two CTAs fit one SM's shared memory");
    auto kern = forward_fused_kernel<G, decltype(cr_c)::value, decltype(pair_c)::value, decltype(bid_c)::value>;
    if (int rc = set_smem_attr((const void*)kern, smem, err, errlen, G == 4 ? kFusedRegs : 0)) return rc;
    const int nsb = (g.tk + G * kTileRows - 1) / (G * kTileRows);
    kern<<<(unsigned)(g.n * nsb), 128 * (G + 1), smem, st>>>(mq, mv, mo, g, (const __nv_bfloat16*)k, rmax, rden, carry, total,
                                                            ssum);
    return 0;
  };
  using std::integral_constant;
  using Softmax = integral_constant<int, kBidSoftmax>;
  using Sigmoid = integral_constant<int, kBidSigmoid>;
  using Expshift = integral_constant<int, kBidExpshift>;
  auto by_pair = [&](auto groups_c, auto cr_c) {
    return pair_demands(g) ? launch(groups_c, cr_c, std::true_type{}, Softmax{}) : launch(groups_c, cr_c, std::false_type{}, Softmax{});
  };
  auto by_rows = [&](auto groups_c) {
    if (g.bid == kBidSigmoid) {                             // (variants have checkpoints every 32 rows)
      return pair_demands(g) ? launch(groups_c, integral_constant<int, 32>{}, std::true_type{}, Sigmoid{})
                             : launch(groups_c, integral_constant<int, 32>{}, std::false_type{}, Sigmoid{});
    }
    if (!g.normalised) return launch(groups_c, integral_constant<int, 32>{}, std::false_type{}, Expshift{});
    return g.carry_rows == 64 ? by_pair(groups_c, integral_constant<int, 64>{}) : by_pair(groups_c, integral_constant<int, 32>{});
  };
  if (int rc = fused_groups(g.n, g.tk) == 4 ? by_rows(integral_constant<int, 4>{}) : by_rows(integral_constant<int, 1>{})) return rc;
  return launch_status("tc forward_fused", err, errlen);
}

// The division that ends the fused forward: out = O / (rs + eps), in place.
inline int normalize_out(const Geom& g, float* out, const float* ssum, cudaStream_t st, char* err, size_t errlen) {
  const int64_t n4 = g.n * g.tq * kHeadDim / 4;
  normalize_out_kernel<<<(unsigned)((n4 + 255) / 256), 256, 0, st>>>(out, ssum, g.eps, n4);
  return launch_status("tc normalize_out", err, errlen);
}

}  // namespace tc
}  // namespace dil
