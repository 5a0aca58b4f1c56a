// Row pass with a product: causal-softmax row statistics AND  O = P B  in one sweep,
// bf16 inputs, head_dim 64, on the same tcgen05 / TMEM / TMA building blocks as the other
// tensor-core kernels.
//
//   B = K : O / den * scale = pk = scale * softmax(q k^T) k, the query half of the
//           softmax-Jacobian correction that the reference's K1 saves for the backward
//           (kernels.py:161-188); with pk saved, the backward's correction pass only has the
//           key half left (kernels.py:777-826).
//   B = V : O / den = causal softmax attention, the reference's CausalSelfAttention layers
//           (model.py:96-117: F.scaled_dot_product_attention(q, k, v, is_causal=True)).
//
// grid = n * ceil(tq/128), longest rows first.  S = Q K^T, lane = query, 256 threads: the
// two warpgroups split a tile's 128 key columns and are independent of each other: each keeps,
// per query row, its own reference maximum, its own sum of 2^(z - reference) and its own
// accumulator O_wg [128 queries x 64] in TMEM, fed by P~ = 2^(z - reference) written as bf16
// pairs over the score columns the thread has just consumed (the A operand of O_wg += P~ B, with
// B the MN-major view of the K or V tile).  The two halves are merged once, at the end.
// The reference exponent follows the scores lazily: it is set from the first tile's maximum and
// moves again only when a tile's P~ sum to more than 2^40, and only then is the accumulator
// rescaled (one TMEM round trip per warp).  The common tile therefore takes no maximum and no
// rescaling; bf16 has fp32's exponent range, so P~ of any magnitude below that limit keeps its
// 8 bits, and sums run in fp32.  rmax therefore holds the reference, not the exact row maximum:
// the pair (rmax, rden) is exact only as the log-sum-exp rmax + log2(rden), which is all the
// other passes use.
// TMEM: S 128 columns + 2 x 64 accumulator columns = 256; two CTAs per SM.
#pragma once

#include "tc_kernels.cuh"

namespace dil {
namespace tc {

constexpr float kRefLimit = 1099511627776.f;         // 2^40: a tile whose P~ sum to more moves the reference
template <int MODE> struct RowpassSmem {
  // Q | K[stages] | (V[stages]) | stats [2][128] float4 | barriers + control.  Three stages when
  // K is the only streamed operand; two of K and two of V otherwise, so that two CTAs fit an SM.
  static constexpr int kStages = MODE == 2 ? 2 : 3;
  static constexpr int kTiles = 1 + kStages * (MODE == 2 ? 2 : 1);
  static constexpr int kBytes = kTiles * (int)kTileBytes + 4096 + 256 + 1024;
};

// One step of a warpgroup of a row pass (lane = query): the 64 scores of keys first_key and on at tS, of which it forms P~ over the
// scores it has read (keys 2c, 2c+1 in column c, two planes: the lo plane over the other 32), and the sums.  tO: its accumulator;
// ia: the lane's query; edge: some of the keys are masked for some of the tile's queries.
template <int W>
__device__ __forceinline__ void row_half_tile(uint32_t tS, uint32_t tO, const Geom& g, int first_key, int ia, bool edge, float& m_ref,
                                              float& s) {
  constexpr int kAcc = Rows<W>::kCols;
  float v[64];
  tmem_ld32(tS, v);
  tmem_ld32(tS + 32, v + 32);
  tmem_ld_wait(v);
  tmem_ld_wait(v + 32);
  uint32_t pw[32], pr[Rows<W>::kPlanes == 2 ? 32 : 1];
  float ps = 0.f;
  // P~ = 2^(z - reference) for the thread's 64 scores, two per instruction; their sum in ps
  auto exponentials = [&]() {
    const float mr = m_ref == -INFINITY ? 0.f : m_ref;
    const float2 zs = make_float2(g.zscale, g.zscale), off = make_float2(-mr, -mr);
    float2 acc0 = make_float2(0.f, 0.f), acc1 = make_float2(0.f, 0.f);
#pragma unroll
    for (int e = 0; e < 64; e += 4) {
      const float2 z0 = fma2(make_float2(v[e], v[e + 1]), zs, off);
      const float2 z1 = fma2(make_float2(v[e + 2], v[e + 3]), zs, off);
      const float2 p0 = make_float2(fast_exp2(z0.x), fast_exp2(z0.y));
      const float2 p1 = make_float2(fast_exp2(z1.x), fast_exp2(z1.y));
      acc0 = add2(acc0, p0);
      acc1 = add2(acc1, p1);
      pw[e >> 1] = pack_bf16(p0.x, p0.y);
      pw[(e >> 1) + 1] = pack_bf16(p1.x, p1.y);
      if (Rows<W>::kPlanes == 2) {
        pr[e >> 1] = pack_bf16_rest(p0.x, p0.y, pw[e >> 1]);
        pr[(e >> 1) + 1] = pack_bf16_rest(p1.x, p1.y, pw[(e >> 1) + 1]);
      }
    }
    const float2 acc = add2(acc0, acc1);
    ps = acc.x + acc.y;
  };
  // The common tile takes no maximum at all: the reference stays where it is as long as the
  // tile's sum of P~ stays below 2^40 (then every P~ does, and nothing overflowed).
  // Edge tiles (masking), rows that have not seen a score yet and tiles that outgrow the
  // reference take the slow path: mask, take the tile's maximum, move the reference there,
  // rescale what was accumulated under the old one, and form P~ again.
  bool slow = edge || __any_sync(0xffffffffu, m_ref == -INFINITY);
  if (!slow) {
    exponentials();
    slow = __any_sync(0xffffffffu, !(ps < kRefLimit));
    if (slow) {                      // rare: the scores are still in TMEM, fetch them again
      tmem_ld32(tS, v);
      tmem_ld32(tS + 32, v + 32);
      tmem_ld_wait(v);
      tmem_ld_wait(v + 32);
    }
  }
  if (slow) {
    float cmax = -INFINITY;
    if (edge) {
#pragma unroll
      for (int e = 0; e < 64; ++e) {
        const int ja = first_key + e;
        if (ja > ia || ja >= g.tk) v[e] = -INFINITY;
        cmax = fmaxf(cmax, v[e]);
      }
    } else {
#pragma unroll
      for (int e = 0; e < 64; ++e) cmax = fmaxf(cmax, v[e]);
    }
    const float m_new = fmaxf(m_ref, cmax * g.zscale);
    if (__any_sync(0xffffffffu, m_new != m_ref)) {
      const bool fresh = __all_sync(0xffffffffu, m_ref == -INFINITY);   // nothing accumulated yet
      // (no branch: the TMEM loads below are warp-wide; a row without a reference has nothing but zeros or NaN yet)
      const float f = fast_exp2(m_ref - (m_new == -INFINITY ? 0.f : m_new));
      if (!fresh) {
#pragma unroll
        for (int c = 0; c < kAcc / 16; ++c) {
          float o[16];
          tmem_ld16(tO + 16 * c, o);
          tmem_ld_wait16(o);
          uint32_t w[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) w[e] = __float_as_uint(o[e] * f);
          tmem_st16(tO + 16 * c, w);
        }
      }
      s *= f;
      m_ref = m_new;
    }
    exponentials();
  }
  s += ps;
  tmem_st16(tS, pw);
  tmem_st16(tS + 16, pw + 16);
  if (Rows<W>::kPlanes == 2) {
    tmem_st16(tS + 32, pr);
    tmem_st16(tS + 48, pr + 16);
  }
  tmem_st_wait();
}

// The end of a row pass: the two warpgroups' halves of every row are merged.  Each finishes half of the output columns: it hands the
// other half of its accumulator, with its statistics, to the other one through sX [2][128][half a row].  n, i: the lane's row and query;
// sync: a barrier of the two.
template <int MODE, int WG, int W, typename TOut, typename Sync>
__device__ __forceinline__ void row_merge(uint32_t tO, const Geom& g, int n, int i, int row, float m_ref, float s, float4* sStat, float* sX,
                                          float* __restrict__ rmax, float* __restrict__ rden, TOut* __restrict__ out, Sync sync) {
  constexpr int kHalf = Rows<W>::kHead / 2;
  // columns [base, base + 32) of this warpgroup's accumulator (kSplit: P K_hi + P K_lo)
  auto fetch = [&](int base, float* o) {
    __syncwarp();                                         // (rows behind the last query leave the loops below)
    tmem_ld32(tO + base, o);
    tmem_ld_wait(o);
    if (W == kSplit) {
      float lo[32];
      tmem_ld32(tO + 64 + base, lo);
      tmem_ld_wait(lo);
#pragma unroll
      for (int e = 0; e < 32; ++e) o[e] += lo[e];
    }
  };
  sStat[WG * 128 + row] = make_float4(m_ref, s, 0.f, 0.f);
  float* give = sX + ((1 - WG) * 128 + row) * kHalf;      // read by the other warpgroup
#pragma unroll
  for (int c0 = 0; c0 < kHalf; c0 += 32) {
    float o[32];
    fetch(kHalf * (1 - WG) + c0, o);
#pragma unroll
    for (int c = 0; c < 8; ++c)
      reinterpret_cast<float4*>(give + c0)[c ^ (row & 7)] = make_float4(o[4 * c], o[4 * c + 1], o[4 * c + 2], o[4 * c + 3]);
  }
  sync();
  const float4 other = sStat[(1 - WG) * 128 + row];
  const float m = fmaxf(m_ref, other.x);                  // finite: warpgroup 0 always sees key 0
  const float ref = m == -INFINITY ? 0.f : m;
  const float f_own = fast_exp2(m_ref - ref), f_oth = fast_exp2(other.x - ref);
  const float den = s * f_own + other.y * f_oth;
  const float inv = (MODE == 1 ? g.scale : 1.f) / den;
  __syncwarp();                                           // (a division has paths of its own for NaN and the like)
  const float a_own = f_own * inv, a_oth = f_oth * inv;
  const float* take = sX + (WG * 128 + row) * kHalf;
  const int d = W == kSplit ? g.d : Rows<W>::kHead;
#pragma unroll
  for (int c0 = 0; c0 < kHalf; c0 += 32) {
    float r[32];
    fetch(kHalf * WG + c0, r);
    if (i >= g.tq) continue;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const float4 x = reinterpret_cast<const float4*>(take + c0)[c ^ (row & 7)];
      r[4 * c] = r[4 * c] * a_own + x.x * a_oth;
      r[4 * c + 1] = r[4 * c + 1] * a_own + x.y * a_oth;
      r[4 * c + 2] = r[4 * c + 2] * a_own + x.z * a_oth;
      r[4 * c + 3] = r[4 * c + 3] * a_own + x.w * a_oth;
    }
    TOut* dst = out + ((int64_t)n * g.tq + i) * d + kHalf * WG + c0;
    if (std::is_same<TOut, float>::value) {
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (W != kSplit || kHalf * WG + c0 + 4 * c < d)
          reinterpret_cast<float4*>(dst)[c] = make_float4(r[4 * c], r[4 * c + 1], r[4 * c + 2], r[4 * c + 3]);
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c)
        reinterpret_cast<uint4*>(dst)[c] =
            make_uint4(pack_bf16(r[8 * c], r[8 * c + 1]), pack_bf16(r[8 * c + 2], r[8 * c + 3]),
                       pack_bf16(r[8 * c + 4], r[8 * c + 5]), pack_bf16(r[8 * c + 6], r[8 * c + 7]));
    }
  }
  if (WG == 0 && i < g.tq && rmax != nullptr) {
    // the merged reference, not necessarily the row maximum (it lags behind it by design);
    // every consumer uses the pair only as the log-sum-exp rmax + log2(rden)
    rmax[(int64_t)n * g.tq + i] = m;
    rden[(int64_t)n * g.tq + i] = den;
  }
}

// ONE_POLLS: one lane of the issuing warp waits for the next tiles, the others behind it (kOnePollsAbove).
template <int MODE, typename TOut, bool ONE_POLLS = false>
__global__ void __launch_bounds__(256, 2) rowpass_product_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
    const __grid_constant__ CUtensorMap map_v, Geom g, float* __restrict__ rmax, float* __restrict__ rden,
    TOut* __restrict__ out) {
  static_assert(MODE == 1 || MODE == 2, "1: B = K (pk); 2: B = V (softmax attention)");
  constexpr uint32_t TB = kTileBytes;
  constexpr int kAcc = kHeadDim;                     // accumulator columns of one warpgroup
  constexpr int kTmem = 256;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  const uint32_t sQ = smem_u32(smem), sK0 = sQ + TB;
  constexpr int kRowpassStages = RowpassSmem<MODE>::kStages;
  const uint32_t sB0 = MODE == 2 ? sK0 + kRowpassStages * TB : sK0;
  constexpr int kTiles = RowpassSmem<MODE>::kTiles;
  float4* sStat = reinterpret_cast<float4*>(smem + kTiles * TB);            // [2][128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kTiles * TB + 4096);
  Ctl* ctl = reinterpret_cast<Ctl*>(bars + 8);
  const uint32_t kfull = smem_u32(bars), sdone = smem_u32(bars + 4);
  float* sX = reinterpret_cast<float*>(smem + TB);    // merge area over the K stages: [2][128][half a row]

  const int tid = threadIdx.x, warp = tid >> 5, wg = tid >> 7, row = tid & 127;
  const int warp_u = uniform_warp();
  const uint32_t lead = elect_one();
  const int nqb = (g.tq + kTileRows - 1) / kTileRows;
  const int n = (int)(blockIdx.x % g.n);
  const int ib = nqb - 1 - (int)(blockIdx.x / g.n);
  const int q0 = g.q_off + ib * kTileRows;
  const int njb = min(g.tk - 1, q0 + kTileRows - 1) / kTileRows + 1;
  constexpr uint32_t kStageTx = (MODE == 2 ? 2u : 1u) * TB;

  if (tid == 0) {
    ctl->abort = 0;
    for (int i = 0; i < kRowpassStages; ++i) mbar_init(kfull + 8 * i, 1);
    mbar_init(sdone, 1);
    fence_barrier_init();
  }
  __syncwarp();
  if (warp == 0) tmem_alloc(smem_u32(&ctl->tmem), kTmem);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = uniform(ctl->tmem);
  const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
  const uint32_t tS = tmem, tO = tmem + 128 + kAcc * wg;      // this warpgroup's accumulator
  {
    uint32_t z[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) z[c] = 0u;
#pragma unroll
    for (int c = 0; c < kAcc / 16; ++c) tmem_st16(tO + lane_base + 16 * c, z);
    tmem_st_wait();
  }
  auto load_stage = [&](int jb) {          // thread 0: K (and V) tile jb into its ring slot
    const int st = jb % kRowpassStages;
    mbar_expect_tx(kfull + 8 * st, kStageTx);
    tma_load_tile(sK0 + TB * st, &map_k, jb * kTileRows, n, kfull + 8 * st);
    if (MODE == 2) tma_load_tile(sB0 + TB * st, &map_v, jb * kTileRows, n, kfull + 8 * st);
  };
  if (tid == 0) {
    mbar_expect_tx(kfull, kStageTx + TB);
    tma_load_tile(sQ, &map_q, ib * kTileRows, n, kfull);
    tma_load_tile(sK0, &map_k, 0, n, kfull);
    if (MODE == 2) tma_load_tile(sB0, &map_v, 0, n, kfull);
    for (int jb = 1; jb < kRowpassStages && jb < njb; ++jb) load_stage(jb);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp_u == 0) {
    mbar_wait(kfull, 0, ctl, &g_status, kErrWaitTma);
    tc_fence_after();
    mma_scores_w<kNarrow>(lead, tS, sQ, sK0, 128);
    mma_commit(lead, sdone);
  }
  __syncwarp();

  float m_ref = -INFINITY, s = 0.f;
  const int ia = q0 + row;
  for (int jb = 0; jb < njb; ++jb) {
    const int st = jb % kRowpassStages;
    // scores of tile jb are ready, and the product of tile jb-1 has completed
    mbar_wait(sdone, jb & 1, ctl, &g_status, kErrWaitMma);
    tc_fence_after();
    if (tid == 0 && jb >= 1 && jb - 1 + kRowpassStages < njb)
      load_stage(jb - 1 + kRowpassStages);                          // the slot of tile jb-1 is free
    __syncwarp();
    const bool edge = (jb * kTileRows + kTileRows - 1 > q0) || ((jb + 1) * kTileRows > g.tk);
    row_half_tile<kNarrow>(tS + lane_base + 64 * wg, tO + lane_base, g, jb * kTileRows + wg * 64, ia, edge, m_ref, s);
    tc_fence_before();
    __syncthreads();
    if (warp_u == 0) {
      tc_fence_after();
      constexpr uint32_t id_pv = instr_desc(128, kAcc, 0, 1);   // A from TMEM (M = queries), B MN-major
      const Desc dB = make_desc(sB0 + TB * st, kTileBytes, 1024);
#pragma unroll
      for (int w = 0; w < 2; ++w)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)        // 16 keys per instruction: 16 rows of 128 B = 128 units
          mma_ts(lead, tmem + 128 + kAcc * w, tS + 64 * w + 8 * kk, dB, 128 * (4 * w + kk), id_pv, 1);
      if (jb + 1 < njb) {
        const int sn = (jb + 1) % kRowpassStages;
        if (!ONE_POLLS || (tid & 31) == 0) mbar_wait(kfull + 8 * sn, ((jb + 1) / kRowpassStages) & 1, ctl, &g_status, kErrWaitTma);
        if (ONE_POLLS) __syncwarp();
        tc_fence_after();
        mma_scores_w<kNarrow>(lead, tS, sQ, sK0 + TB * sn, 128);
      }
      mma_commit(lead, sdone);
    }
    __syncwarp();
  }
  mbar_wait(sdone, njb & 1, ctl, &g_status, kErrWaitMma);
  tc_fence_after();
  auto sync = [] { __syncthreads(); };
  const int i = ib * kTileRows + row;
  if (wg == 0) row_merge<MODE, 0, kNarrow>(tO + lane_base, g, n, i, row, m_ref, s, sStat, sX, rmax, rden, out, sync);
  else row_merge<MODE, 1, kNarrow>(tO + lane_base, g, n, i, row, m_ref, s, sStat, sX, rmax, rden, out, sync);
  drain_if_aborted(ctl);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_free(tmem, kTmem);
}

// The same with a warp that issues every TMA copy and MMA.  Of each query tile's two warpgroups one takes the half tiles of 64 keys
// 0, 2, 4, .., the other 1, 3, 5, ..: the keys that they have in rowpass_product_kernel, with scores of their own.  The issuing warp
// serves a warpgroup's P~ B and, behind it in the pipe, its next scores as soon as its P~ is written, and nothing in the loop waits for
// the whole CTA.  Keys, their order and every operation on them are those of rowpass_product_kernel, and so are the results, bit for bit.
//
// Wide rows: one query tile per CTA.  With one CTA per SM nothing else hides the round trip of a tile's scores.  Row pass with pk,
// as rowpass_product_kernel / this, in us: d = 128 n = 32, T = 4096 263 / 209, n = 4, T = 4096 68 / 53, n = 100, T = 1024 91 / 81, n = 300,
// T = 128 27.7 / 27.6, n = 20, T = 300 14.9 / 14.9; fp32 heads of 64 n = 32, T = 4096 281 / 223, n = 148, T = 256 21.2 / 21.2.  Two query
// tiles per CTA, one per warpgroup, take 196 and 220 us at n = 32, T = 4096 and more than this with few blocks (n = 5, T = 8192 174,
// here 123), but a row's accumulator then takes twice as many additions: the error of pk against 64 bits went from 1.71e-6 to 2.43e-6
// (d = 128, n = 32, T = 2048), and that of dq of fp32 heads from 6.56e-6 to 6.57e-6.
//
// Narrow rows: two query tiles per CTA (kRowPairsFrom), so that each half tile of keys is copied once for 256 queries.  Long calls run at
// the card's power limit, where one tile per CTA and two CTAs per SM gain nothing: softmax, n = 64, T = 8192, calls without a pause
// 851 us as rowpass_product_kernel, 857 so, 800 with two tiles.
// TMEM: [S 64 | O] per warpgroup.  grid = n * ceil(tq / queries of a CTA), longest rows first; one CTA per SM.
template <int MODE, int W> struct RowIssuer {
  static constexpr int kTiles = W == kNarrow ? 2 : 1;                    // query tiles
  static constexpr int kThreads = 256 * kTiles + 32;
  static constexpr int kRing = 8;                                        // half tiles of K (and V)
  // Q[tiles] | K[ring] (V[ring]) | stats [tiles][2][128] float4 | barriers + control
  static constexpr int kOperands = (2 * kTiles + kRing * MODE) * (int)Rows<W>::kBytes / 2;
  static constexpr int kBytes = kOperands + 4096 * kTiles + 256 + 1024;
};

template <int MODE, typename TOut, int W>
__global__ void __launch_bounds__(RowIssuer<MODE, W>::kThreads, 1) rowpass_issuer_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
    const __grid_constant__ CUtensorMap map_v, Geom g, float* __restrict__ rmax, float* __restrict__ rden,
    TOut* __restrict__ out) {
  static_assert(MODE == 1 || MODE == 2, "1: B = K (pk); 2: B = V (softmax attention)");
  using Form = RowIssuer<MODE, W>;
  constexpr int R = Form::kRing, NT = Form::kTiles, kTmem = 512;
  constexpr uint32_t TB = Rows<W>::kBytes, HB = TB / 2, HSub = kTileBytes / 2;    // a tile, half a tile, a sub-tile of that
  constexpr int kAcc = Rows<W>::kCols, kWg = 64 + kAcc;                            // TMEM columns of O, and of a warpgroup
  static_assert(2 * NT * kWg <= kTmem, "the warpgroups' columns fit the allocation");
  static_assert(NT * 128 * Rows<W>::kHead * 4 <= R * MODE * (int)HB, "the merge area fits the K stages");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  const uint32_t sQ = smem_u32(smem), sK = sQ + NT * TB, sB = MODE == 2 ? sK + R * HB : sK;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Form::kOperands + 4096 * NT);
  const uint32_t qfull = smem_u32(bars), kfull = qfull + 8, kfree = kfull + 8 * R, sdone = kfree + 8 * R, pready = sdone + 16 * NT;
  Ctl* ctl = reinterpret_cast<Ctl*>(bars + 1 + 2 * R + 4 * NT);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, wg = tid >> 7, row = tid & 127;
  const int warp_u = uniform_warp();
  const uint32_t lead = elect_one();
  const int nqb = (g.tq + NT * kTileRows - 1) / (NT * kTileRows);
  const int n = (int)(blockIdx.x % g.n);
  const int ib = (nqb - 1 - (int)(blockIdx.x / g.n)) * NT;                  // (first) query tile
  // half tiles of keys that a tile's queries see; none for a tile behind the last query
  auto half_tiles = [&](int tile) {
    const int i0 = (ib + tile) * kTileRows;
    return i0 < g.tq ? min(g.tk - 1, g.q_off + i0 + kTileRows - 1) / 64 + 1 : 0;
  };
  const int nh0 = half_tiles(0), nh1 = NT == 2 ? half_tiles(1) : 0, nh = max(nh0, nh1);

  if (tid == 0) {
    ctl->abort = 0;
    for (int i = 0; i < 1 + 2 * R + 2 * NT; ++i) mbar_init(qfull + 8 * i, 1);          // qfull, kfull[R], kfree[R], sdone[2 NT]
    for (int i = 0; i < 2 * NT; ++i) mbar_init(pready + 8 * i, 4);
    fence_barrier_init();
  }
  __syncwarp();
  if (warp == 0) tmem_alloc(smem_u32(&ctl->tmem), kTmem);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = uniform(ctl->tmem);

  if (warp_u == 8 * NT) {
    // ------------------------------------------------------------ the issuing warp
    constexpr uint32_t id_s = instr_desc(128, 64, 0, 0), id_p = instr_desc(128, kAcc, 0, 1);
    const Desc dQ = make_desc(sQ, 16, 1024), dK = make_desc(sK, 16, 1024), dB = make_desc(sB, HSub, 1024);
    auto load_keys = [&](int h) {
      const int st = h % R;
      if (!lead) return;
      mbar_expect_tx(kfull + 8 * st, MODE * HB);
      tma_load_rows<W>(sK + HB * st, &map_k, h * 64, n, kfull + 8 * st, HSub);
      if (MODE == 2) tma_load_rows<W>(sB + HB * st, &map_v, h * 64, n, kfull + 8 * st, HSub);
    };
    const int tiles = nh1 > 0 ? 2 : 1;
    if (lead) {
      mbar_expect_tx(qfull, tiles * TB);
      for (int i = 0; i < tiles; ++i) tma_load_rows<W>(sQ + TB * i, &map_q, (ib + i) * kTileRows, n, qfull);
    }
    for (int h = 0; h < R && h < nh; ++h) load_keys(h);
    mbar_wait_warp(qfull, 0, ctl, &g_status, kErrWaitTma);
    for (int h = 0; h < nh + 2; ++h) {
      if (h < nh) mbar_wait_warp(kfull + 8 * (h % R), (h / R) & 1, ctl, &g_status, kErrWaitTma);
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        const int w = 2 * i + (h & 1), nt = i ? nh1 : nh0;
        const uint32_t tS = tmem + kWg * w;
        if (nt == 0 || h >= nt + 2) continue;
        if (h >= 2) {
          mbar_wait_warp(pready + 8 * w, ((h >> 1) - 1) & 1, ctl, &g_status, kErrWaitTile);
          tc_fence_after();
#pragma unroll
          for (int pl = 0; pl < Rows<W>::kPlanes; ++pl)
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)                        // 16 keys per instruction: 16 rows of 128 B = 128 units
              mma_ts(lead, tS + 64, tS + 32 * pl + 8 * kk, dB, (HB >> 4) * ((h - 2) % R) + 128 * kk, id_p, 1);
        }
        if (h < nt) {
          tc_fence_after();
          mma_scores_wide<W>(lead, tS, Desc{dQ.lo + (TB >> 4) * i, dQ.hi}, kTileBytes, Desc{dK.lo + (HB >> 4) * (h % R), dK.hi}, HSub, id_s);
        }
        mma_commit(lead, sdone + 8 * w);                          // P~ B of h - 2 and the scores of h, one of them or none
      }
      if (h >= 2) mma_commit(lead, kfree + 8 * ((h - 2) % R));
      // half tile h - 3, whose products were issued one round ago, makes room for h - 3 + R
      if (h >= 3 && h - 3 + R < nh) {
        mbar_wait_warp(kfree + 8 * ((h - 3) % R), ((h - 3) / R) & 1, ctl, &g_status, kErrWaitMma);
        load_keys(h - 3 + R);
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ the compute warps: lane = query
    const uint32_t tS = tmem + kWg * wg + ((uint32_t)((warp & 3) * 32) << 16), tO = tS + 64;
    {
      uint32_t z[16];
#pragma unroll
      for (int c = 0; c < 16; ++c) z[c] = 0u;
#pragma unroll
      for (int c = 0; c < kAcc / 16; ++c) tmem_st16(tO + 16 * c, z);
      tmem_st_wait();
    }
    const int tile = NT == 2 ? wg >> 1 : 0, half = wg & 1, nt = tile ? nh1 : nh0;
    const int i = (ib + tile) * kTileRows + row, q0 = g.q_off + (ib + tile) * kTileRows, ia = q0 + row;
    float m_ref = -INFINITY, s = 0.f;
    int t = 0;                                                // the warpgroup's own count of half tiles
    for (int h = half; h < nt; h += 2, ++t) {
      mbar_wait_warp(sdone + 8 * wg, t & 1, ctl, &g_status, kErrWaitMma);
      tc_fence_after();
      const bool edge = ((h | 1) * 64 + 63 > q0) || (((h | 1) + 1) * 64 > g.tk);      // (by whole tiles, as there)
      row_half_tile<W>(tS, tO, g, h * 64, ia, edge, m_ref, s);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(pready + 8 * wg);
    }
    if (nt > 0) mbar_wait_warp(sdone + 8 * wg, t & 1, ctl, &g_status, kErrWaitMma);
    tc_fence_after();
    // every product has read the K stages, which the merge goes over
    asm volatile("bar.sync 1, %0;" ::"n"(256 * NT) : "memory");
    // merge area [2][128][half a row] and statistics [2][128] of this tile
    float* sX = reinterpret_cast<float*>(smem + NT * TB) + tile * 128 * Rows<W>::kHead;
    float4* sStat = reinterpret_cast<float4*>(smem + Form::kOperands) + 256 * tile;
    auto sync = [tile] {
      if (NT == 1 || tile == 0) asm volatile("bar.sync 2, 256;" ::: "memory");
      else asm volatile("bar.sync 3, 256;" ::: "memory");
    };
    if (nt > 0 && half == 0) row_merge<MODE, 0, W>(tO, g, n, i, row, m_ref, s, sStat, sX, rmax, rden, out, sync);
    else if (nt > 0) row_merge<MODE, 1, W>(tO, g, n, i, row, m_ref, s, sStat, sX, rmax, rden, out, sync);
  }
  drain_if_aborted(ctl);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_free(tmem, kTmem);
}

// Key half of the softmax-Jacobian correction alone (the reference's BC, kernels.py:777-809),
// for a backward that has pk saved:  dk = dk_main - scale * P^T (ghat * Q).
// grid = n * ceil(t/128) key blocks; S^T = K Q^T, lane = key; W = p * ghat goes back into TMEM
// over the consumed score columns as the A operand (M = keys) of dKc += W Q.  Nothing passes
// through shared memory and nothing is reduced across CTAs.
// The pass runs in half-steps of 64 queries: S^T [128 keys x 64 queries] needs 64 TMEM columns, so
// a CTA allocates 128 (S^T 64 + dKc 64) and four CTAs share an SM (32 warps to hide each other's
// MMA round trips, as in the column-sum pass; a version with 128-query steps and two CTAs per SM
// measured 5% slower).  The two warpgroups split a half-step's 64 query columns.
template <int W> constexpr int kCorrKey64Smem = 3 * (int)Rows<W>::kBytes + 2048 + 1024 + 256;
static_assert(5 * (kCorrKey64Smem<kNarrow> + 1024) > 233472, "at most four CTAs of the half-step correction pass share an SM");

// TOut: element type of dk (bf16, or float for kSplit).
template <int W = kNarrow, typename TOut = __nv_bfloat16>
__global__ void __launch_bounds__(256, W == kNarrow ? 4 : 2) backward_key_correction64_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, Geom g,
    const float* __restrict__ rmax, const float* __restrict__ rden, const float* __restrict__ ghat,
    const float* __restrict__ dk_main, TOut* __restrict__ dk) {
  constexpr uint32_t TB = Rows<W>::kBytes;
  constexpr int kAcc = Rows<W>::kCols, kTmem = W == kNarrow ? 128 : 256;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  const uint32_t sK = smem_u32(smem), sQ0 = sK + TB;
  float2* sStat = reinterpret_cast<float2*>(smem + 3 * TB);           // [2][128] (lse, ghat)
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 3 * TB + 2048);
  Ctl* ctl = reinterpret_cast<Ctl*>(bars + 8);
  const uint32_t qfull = smem_u32(bars), sdone = smem_u32(bars + 2);

  const int tid = threadIdx.x, warp = tid >> 5, wg = tid >> 7, row = tid & 127;
  const int warp_u = uniform_warp();
  const uint32_t lead = elect_one();
  const int nqb = (g.tq + kTileRows - 1) / kTileRows;
  const int n = (int)(blockIdx.x % g.n);
  const int jb = (int)(blockIdx.x / g.n);
  const int k0 = jb * kTileRows;
  const int nsteps = nqb - jb, nhalf = 2 * nsteps;
  const int64_t row_base = (int64_t)n * g.tq;

  if (tid == 0) {
    ctl->abort = 0;
    for (int i = 0; i < 3; ++i) mbar_init(qfull + 8 * i, 1);
    fence_barrier_init();
  }
  __syncwarp();
  if (warp == 0) tmem_alloc(smem_u32(&ctl->tmem), kTmem);
  if (wg == 1) {
    const int i = jb * kTileRows + row;
    float2 st = make_float2(INFINITY, 0.f);
    if (i < g.tq) st = make_float2(rmax[row_base + i] + log2f(rden[row_base + i]), ghat[row_base + i]);
    sStat[row] = st;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = uniform(ctl->tmem);
  const uint32_t tS = tmem, tDK = tmem + 64;
  constexpr uint32_t id_s = instr_desc(128, 64, 0, 0), id_kd = instr_desc(128, kAcc, 0, 1);
  // scores of half-step (stage, odd): queries 64*odd.. of the Q tile in that stage (K-major: a
  // row is 128 B)
  auto issue_scores = [&](int stage, int odd) {
    mma_scores_wide<W>(lead, tS, make_desc(sK, 16, 1024), kTileBytes,
                       make_desc(sQ0 + TB * stage + 8192 * odd, 16, 1024), kTileBytes, id_s);
  };

  if (tid == 0) {
    mbar_expect_tx(qfull, 2 * TB);
    tma_load_rows<W>(sK, &map_k, k0, n, qfull);
    tma_load_rows<W>(sQ0, &map_q, jb * kTileRows, n, qfull);
    if (nsteps > 1) {
      mbar_expect_tx(qfull + 8, TB);
      tma_load_rows<W>(sQ0 + TB, &map_q, (jb + 1) * kTileRows, n, qfull + 8);
    }
  }
  if (warp_u == 0) {
    __syncwarp();
    mbar_wait(qfull, 0, ctl, &g_status, kErrWaitTma);
    tc_fence_after();
    issue_scores(0, 0);
    mma_commit(lead, sdone);
  }
  __syncwarp();

  const int ja = k0 + row;
  const bool dead = ja >= g.tk;
  const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
  const uint32_t tcol = tS + lane_base + 32 * wg;
  for (int h = 0; h < nhalf; ++h) {
    const int t = h >> 1, odd = h & 1, ib = jb + t, b = t & 1;
    float nx_max = INFINITY, nx_den = 1.f, nx_gh = 0.f;
    const bool fetch = odd == 0 && wg == 1 && t + 1 < nsteps;
    if (fetch && (ib + 1) * kTileRows + row < g.tq) {
      const int64_t i = row_base + (ib + 1) * kTileRows + row;
      nx_max = rmax[i];
      nx_den = rden[i];
      nx_gh = ghat[i];
    }
    // scores of this half-step are ready; every earlier dKc product has completed
    mbar_wait(sdone, h & 1, ctl, &g_status, kErrWaitMma);
    tc_fence_after();
    if (tid == 0 && odd == 0 && t >= 1 && t + 1 < nsteps) {      // the Q stage of step t-1 is free
      mbar_expect_tx(qfull + 8 * (b ^ 1), TB);
      tma_load_rows<W>(sQ0 + TB * (b ^ 1), &map_q, (ib + 1) * kTileRows, n, qfull + 8 * (b ^ 1));
    }
    __syncwarp();
    const int i0 = ib * kTileRows + 64 * odd + 32 * wg;           // first query of this thread's 32
    constexpr bool END = kMaskEnd<W, kBidSoftmax>;
    const bool masked = dead || t == 0 || (END && i0 + 32 > g.tq);
    const float4* St4 = reinterpret_cast<const float4*>(sStat + b * 128 + 64 * odd + 32 * wg);
    float vs[32];
    uint32_t wt[16], wr[Rows<W>::kPlanes == 2 ? 16 : 1];
    tmem_ld32(tcol, vs);
    tmem_ld_wait(vs);
    auto tile = [&](auto mask_tag) {
      constexpr bool MASK = decltype(mask_tag)::value;
#pragma unroll
      for (int e2 = 0; e2 < 16; ++e2) {
        const float4 st = St4[e2];                                // (lse, ghat) of two queries
        float p0 = fast_exp2(fmaf(vs[2 * e2], g.zscale, -st.x));
        float p1 = fast_exp2(fmaf(vs[2 * e2 + 1], g.zscale, -st.z));
        if (MASK) {
          const int i = i0 + 2 * e2;
          if (dead || ja > i || (END && i >= g.tq)) p0 = 0.f;
          if (dead || ja > i + 1 || (END && i + 1 >= g.tq)) p1 = 0.f;
        }
        wt[e2] = pack_bf16(p0 * st.y, p1 * st.w);
        if (Rows<W>::kPlanes == 2) wr[e2] = pack_bf16_rest(p0 * st.y, p1 * st.w, wt[e2]);
      }
    };
    if (masked) tile(std::true_type{}); else tile(std::false_type{});
    tmem_st16(tcol, wt);            // W over the first 16 of the 32 consumed columns (its lo plane over the others)
    if (Rows<W>::kPlanes == 2) tmem_st16(tcol + 16, wr);
    if (fetch) sStat[(b ^ 1) * 128 + row] = make_float2(nx_max + log2f(nx_den), nx_gh);
    tmem_st_wait();
    tc_fence_before();
    __syncthreads();
    if (warp_u == 0) {
      tc_fence_after();
      const Desc dQm = make_desc(sQ0 + TB * b, kTileBytes, 1024);
#pragma unroll
      for (int pl = 0; pl < Rows<W>::kPlanes; ++pl)
#pragma unroll
        for (int kq = 0; kq < 4; ++kq)        // 16 queries per instruction: 16 rows of 128 B = 128 units
          mma_ts(lead, tDK, tS + 32 * (kq >> 1) + 16 * pl + 8 * (kq & 1), dQm, 128 * (4 * odd + kq), id_kd,
                 (h > 0 || pl > 0 || kq > 0));
      if (h + 1 < nhalf) {
        if (odd) {                          // the next half-step opens step t+1
          mbar_wait(qfull + 8 * (b ^ 1), ((t + 1) >> 1) & 1, ctl, &g_status, kErrWaitTma);
          tc_fence_after();
          issue_scores(b ^ 1, 0);
        } else {
          issue_scores(b, 1);
        }
      }
      mma_commit(lead, sdone);
    }
    __syncwarp();
  }
  mbar_wait_warp(sdone, nhalf & 1, ctl, &g_status, kErrWaitMma);
  tc_fence_after();
  // lane = key: each warpgroup finishes half of the columns of dk, 32 at a time
  constexpr int kHead = Rows<W>::kHead, kHalf = kHead / 2;
#pragma unroll
  for (int c0 = kHalf * wg; c0 < kHalf * (wg + 1); c0 += 32) {
    float a[32];
    tmem_ld32(tDK + lane_base + c0, a);
    tmem_ld_wait(a);
    if (W == kSplit) {                                          // W Q_hi + W Q_lo
      float lo[32];
      tmem_ld32(tDK + lane_base + 64 + c0, lo);
      tmem_ld_wait(lo);
#pragma unroll
      for (int e = 0; e < 32; ++e) a[e] += lo[e];
    }
    if (!dead) {
      const float* src = dk_main + ((int64_t)n * g.tk + ja) * kHead + c0;
      const int d = W == kSplit ? g.d : kHead;
      TOut* dst = dk + ((int64_t)n * g.tk + ja) * d + c0;
      float m[32];
#pragma unroll
      for (int e = 0; e < 32; e += 4) {
        const float4 x = *reinterpret_cast<const float4*>(src + e);
        m[e] = x.x - g.scale * a[e];
        m[e + 1] = x.y - g.scale * a[e + 1];
        m[e + 2] = x.z - g.scale * a[e + 2];
        m[e + 3] = x.w - g.scale * a[e + 3];
      }
      store_row32<W>(dst, m, d - c0);
    }
  }
  drain_if_aborted(ctl);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_free(tmem, kTmem);
}

// dq = bf16(dq_main - ghat * pk): the query half of the correction from the saved pk
// (the reference's dq epilogue, kernels.py:814-826; pk already carries the scale).
template <int HEAD = kHeadDim>
__global__ void dq_from_pk_kernel(const float* __restrict__ dq_main, const float* __restrict__ pk,
                                  const float* __restrict__ ghat, __nv_bfloat16* __restrict__ dq, int64_t n4) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n4) return;
  const float4 a = reinterpret_cast<const float4*>(dq_main)[i];
  const float4 b = reinterpret_cast<const float4*>(pk)[i];
  const float gh = ghat[i / (HEAD / 4)];
  reinterpret_cast<uint2*>(dq)[i] = make_uint2(pack_bf16(fmaf(-gh, b.x, a.x), fmaf(-gh, b.y, a.y)),
                                               pack_bf16(fmaf(-gh, b.z, a.z), fmaf(-gh, b.w, a.w)));
}

// ---------------------------------------------------------------- host launchers
// Narrow row passes that take rowpass_issuer_kernel: rows of kRowPairsFrom tokens in kRowPairs blocks of 256 queries.  Its CTAs have an
// SM to themselves, with their start and end unhidden, and 96 registers.  Calls without a pause, rowpass_product_kernel / it, in us,
// with pk: n = 64, T = 16384 3109 / 2901, n = 64, T = 8192 782 / 768, n = 8, T = 8192 (256 blocks) 115.5 / 97.1, n = 64, T = 6144
// 455.6 / 454.5, n = 20, T = 6144 149.3 / 145.6, n = 64, T = 5120 326 / 328, n = 64, T = 4096 217 / 221, n = 128, T = 2048 131 / 143.
// Softmax: n = 64, T = 16384 3409 / 3043, n = 64, T = 8192 851 / 800, n = 1, T = 131072 2915 / 2765, n = 8, T = 8192 106 / 99, n = 64,
// T = 6144 479 / 470, n = 20, T = 6144 147.5 / 146.2, n = 64, T = 5120 338 / 335, n = 64, T = 4096 220.5 / 221.5, n = 128, T = 2048 130 / 137,
// and with fewer blocks than SMs n = 2, T = 3000 32.8 / 40.4.
constexpr int kRowPairsFrom = 6144, kRowPairs = 256;
inline int64_t tile_pairs(const Geom& g) { return g.n * ((g.tq + 2 * kTileRows - 1) / (2 * kTileRows)); }
inline bool row_issuer(const Geom& g) { return g.q_off + g.tq >= kRowPairsFrom && tile_pairs(g) >= kRowPairs; }

// Pass 1 with the saved query correction: rmax, rden and pk = scale * softmax(q k^T) k.
inline int rowstats_pk(const void* q, const void* k, const Geom& g, float* rmax, float* rden, float* pk,
                       cudaStream_t st, char* err, size_t errlen) {
  CUtensorMap mq, mk;
  const bool issuer = row_issuer(g);
  if (int rc = make_map(&mq, q, g.n, g.tq, err, errlen)) return rc;
  if (int rc = make_map(&mk, k, g.n, g.tk, err, errlen, kHeadDim, issuer ? 64 : kTileRows)) return rc;
  if (issuer) {
    using Form = RowIssuer<1, kNarrow>;
    auto kern = rowpass_issuer_kernel<1, float, kNarrow>;
    if (int rc = set_smem_attr((const void*)kern, Form::kBytes, err, errlen)) return rc;
    kern<<<(unsigned)tile_pairs(g), Form::kThreads, Form::kBytes, st>>>(mq, mk, mk, g, rmax, rden, pk);
    return launch_status("tc rowstats_pk", err, errlen);
  }
  const int nqb = (g.tq + kTileRows - 1) / kTileRows;
  auto kern = rowpass_product_kernel<1, float>;
  constexpr int smem = RowpassSmem<1>::kBytes > kTwoPerSm ? RowpassSmem<1>::kBytes : kTwoPerSm;
  if (int rc = set_smem_attr((const void*)kern, smem, err, errlen)) return rc;
  kern<<<(unsigned)(g.n * nqb), 256, smem, st>>>(mq, mk, mk, g, rmax, rden, pk);
  return launch_status("tc rowstats_pk", err, errlen);
}

// Softmax pass, blocks above which one lane of the issuing warp polls for the next tiles instead of 32: where two CTAs share
// every SM for long, it is the faster form, on a chip that is not full the other, whose scores are issued sooner.  All lanes polling /
// one: n = 4, T = 16384 (512 blocks) 196 / 193, n = 16, T = 2048 (256) 25.8 / 27.2, n = 2, T = 3000 (48) 32.9 / 34.9.
constexpr unsigned kOnePollsAbove = 2 * 148;

// Causal softmax attention forward: out = softmax(q k^T * scale) v in bf16; rmax / rden
// (optional) as pass 1 writes them.
inline int softmax_forward(const void* q, const void* k, const void* v, const Geom& g, float* rmax,
                           float* rden, void* out, cudaStream_t st, char* err, size_t errlen) {
  CUtensorMap mq, mk, mv;
  const bool issuer = row_issuer(g);
  const int key_rows = issuer ? 64 : kTileRows;
  if (int rc = make_map(&mq, q, g.n, g.tq, err, errlen)) return rc;
  if (int rc = make_map(&mk, k, g.n, g.tk, err, errlen, kHeadDim, key_rows)) return rc;
  if (int rc = make_map(&mv, v, g.n, g.tk, err, errlen, kHeadDim, key_rows)) return rc;
  if (issuer) {
    using Form = RowIssuer<2, kNarrow>;
    auto kern = rowpass_issuer_kernel<2, __nv_bfloat16, kNarrow>;
    static_assert(Form::kBytes <= 232448, "fits an SM");
    if (int rc = set_smem_attr((const void*)kern, Form::kBytes, err, errlen)) return rc;
    kern<<<(unsigned)tile_pairs(g), Form::kThreads, Form::kBytes, st>>>(mq, mk, mv, g, rmax, rden, (__nv_bfloat16*)out);
    return launch_status("tc softmax_forward", err, errlen);
  }
  const int nqb = (g.tq + kTileRows - 1) / kTileRows;
  const unsigned grid = (unsigned)(g.n * nqb);
  auto kern = grid > kOnePollsAbove ? rowpass_product_kernel<2, __nv_bfloat16, true>
                                    : rowpass_product_kernel<2, __nv_bfloat16>;
  constexpr int smem = RowpassSmem<2>::kBytes;
  static_assert(2 * (smem + 1024) <= 233472 && 3 * (smem + 1024) > 233472, "two CTAs of the softmax pass fit one SM");
  if (int rc = set_smem_attr((const void*)kern, smem, err, errlen)) return rc;
  kern<<<grid, 256, smem, st>>>(mq, mk, mv, g, rmax, rden, (__nv_bfloat16*)out);
  return launch_status("tc softmax_forward", err, errlen);
}

// The tail of the backward when pk was saved by the forward: key correction + dq epilogue.
inline int backward_tail_with_pk(const CUtensorMap& mq, const CUtensorMap& mk, const Geom& g, const float* rmax,
                                 const float* rden, const float* ghat, const float* dk_main,
                                 const float* dq_main, const float* pk, void* dq, void* dk, cudaStream_t st,
                                 char* err, size_t errlen, void (*mark)(const char*, cudaStream_t, int)) {
  const int nkb = (g.tk + kTileRows - 1) / kTileRows;
  constexpr int smem = kCorrKey64Smem<kNarrow>;
  if (int rc = set_smem_attr((const void*)backward_key_correction64_kernel<>, smem, err, errlen)) return rc;
  mark("tc_backward_key_correction", st, 0);
  backward_key_correction64_kernel<><<<(unsigned)(g.n * nkb), 256, smem, st>>>(mq, mk, g, rmax, rden, ghat,
                                                                           dk_main, (__nv_bfloat16*)dk);
  mark("tc_backward_key_correction", st, 1);
  if (int rc = launch_status("tc backward_key_correction", err, errlen)) return rc;
  const int64_t n4 = g.n * g.tq * kHeadDim / 4;
  mark("tc_dq_from_pk", st, 0);
  dq_from_pk_kernel<><<<(unsigned)((n4 + 255) / 256), 256, 0, st>>>(dq_main, pk, ghat, (__nv_bfloat16*)dq, n4);
  mark("tc_dq_from_pk", st, 1);
  return launch_status("tc dq_from_pk", err, errlen);
}

}  // namespace tc
}  // namespace dil
