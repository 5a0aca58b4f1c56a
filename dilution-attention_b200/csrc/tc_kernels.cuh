// bf16 tensor-core path (dot_precision "bf16", bf16 inputs, head_dim 64):
// tcgen05.mma with accumulators in TMEM, operands staged by TMA, 128x128 tiles.
//
// Which axis sits on the TMEM lanes decides what is cheap per thread:
//   pass 1 (row statistics)   S  = Q K^T : lane = query, so row max / row sum
//                                          are private to a thread;
//   passes 2-4 (column work)  S^T = K Q^T: lane = key, so the cumulative demand
//                                          of a key is a running sum in ONE
//                                          register while the thread walks the
//                                          queries of the tile in order; the
//                                          per-query statistics it needs are
//                                          warp-uniform and come from shared
//                                          memory as broadcasts.
// A training forward runs passes 2 and 3 as one key-stationary sweep (tc_fused_forward.cuh);
// forward-only calls, sequence-parallel prefill and the bid / share variants run them separately.
// Warp w of a CTA reads TMEM lanes 32*(w%4)..32*(w%4)+31.  The forward passes and the
// correction pass run 256 threads (two warpgroups that split a tile's columns), thread 0
// issuing TMA and MMA, two to four CTAs per SM hiding each other's MMA/TMA latency; the
// main reverse pass runs 384 threads, one CTA per SM, with a dedicated issuing warpgroup.
#pragma once

#include <mutex>
#include <type_traits>

#include "once_per_device.cuh"
#include "tc_common.cuh"

namespace dil {
namespace tc {

__device__ int g_status = 0;   // first bounded wait that ran out (0 = none)

inline bool supported(int dtype, int precision, int d, int64_t q_offset) {
  return dtype == 1 && precision == 2 && d == kHeadDim && (q_offset % kTileRows) == 0;
}

// ---------------------------------------------------------------- host: tensor maps
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return (EncodeTiledFn)p;
  }();
  return fn;
}

// cuTensorMapEncodeTiled is a driver entry point and wants a current context.  A thread that
// has only selected the device (an autograd engine thread calling the backward first) may
// not have one yet: a runtime call that touches the device binds the primary context.
inline void ensure_context() {
  static thread_local bool bound = false;
  if (!bound) {
    cudaFree(nullptr);
    bound = true;
  }
}

// Encoded maps are kept: a map depends only on (base, n, t, element type, box), and the same
// tensors come back on every step of a training loop or every pass of a forward.
struct MapKey {
  const void* base;
  int64_t n, t;
  int kind;      // 0: bf16 box {64, rows, 1}; 1: fp32 box {32, rows, 1}, swizzled; 2: the same, not swizzled
  int box_rows;
  int feat;      // row length of the tensor in elements
  bool operator==(const MapKey& o) const {
    return base == o.base && n == o.n && t == o.t && kind == o.kind && box_rows == o.box_rows && feat == o.feat;
  }
};
struct MapCache {
  static constexpr int kSlots = 64;
  std::mutex mu;
  MapKey keys[kSlots];
  CUtensorMap maps[kSlots];
  int used = 0, next = 0;
  bool find(const MapKey& k, CUtensorMap* out) {
    std::lock_guard<std::mutex> lk(mu);
    for (int i = 0; i < used; ++i)
      if (keys[i] == k) { *out = maps[i]; return true; }
    return false;
  }
  void put(const MapKey& k, const CUtensorMap& m) {
    std::lock_guard<std::mutex> lk(mu);
    const int i = used < kSlots ? used++ : (next = (next + 1) % kSlots);
    keys[i] = k;
    maps[i] = m;
  }
};
inline MapCache& map_cache() {
  static MapCache c;
  return c;
}

// (n, t, feat) bf16 row-major -> 3-D map {feat, t, n}, box {64, rows, 1}, 128-byte swizzle.
// Rows past t read as zero, and a box never crosses into the next (batch, head) row.
inline int make_map(CUtensorMap* map, const void* base, int64_t n, int64_t t, char* err, size_t errlen,
                    int feat = kHeadDim, int box_rows = kTileRows) {
  const MapKey key{base, n, t, 0, box_rows, feat};
  if (map_cache().find(key, map)) return 0;
  ensure_context();
  EncodeTiledFn fn = encode_fn();
  if (!fn) {
    snprintf(err, errlen, "cuTensorMapEncodeTiled is not available from the driver");
    return 3;
  }
  if ((uintptr_t)base & 15) {
    snprintf(err, errlen, "bf16 tensor-core path needs 16-byte aligned q/k/v");
    return 1;
  }
  const cuuint64_t dims[3] = {(cuuint64_t)feat, (cuuint64_t)t, (cuuint64_t)n};
  const cuuint64_t strides[2] = {(cuuint64_t)feat * 2, (cuuint64_t)t * feat * 2};
  const cuuint32_t box[3] = {(cuuint32_t)kHeadDim, (cuuint32_t)box_rows, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides,
                        box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    snprintf(err, errlen, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return 3;
  }
  map_cache().put(key, *map);
  return 0;
}

// (n, t, feat) fp32 row-major -> 3-D map {feat, t, n}, box {32, rows, 1} (128 bytes wide), with the
// 128-byte swizzle or (swizzle = false) plain rows: the target of the O and dQ tile reductions.
inline int make_map_f32(CUtensorMap* map, const void* base, int64_t n, int64_t t, char* err, size_t errlen,
                        int feat = kHeadDim, int box_rows = kTileRows, bool swizzle = true) {
  const MapKey key{base, n, t, swizzle ? 1 : 2, box_rows, feat};
  if (map_cache().find(key, map)) return 0;
  ensure_context();
  EncodeTiledFn fn = encode_fn();
  if (!fn) {
    snprintf(err, errlen, "cuTensorMapEncodeTiled is not available from the driver");
    return 3;
  }
  const cuuint64_t dims[3] = {(cuuint64_t)feat, (cuuint64_t)t, (cuuint64_t)n};
  const cuuint64_t strides[2] = {(cuuint64_t)feat * 4, (cuuint64_t)t * feat * 4};
  const cuuint32_t box[3] = {32, (cuuint32_t)box_rows, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims, strides, box,
                        estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    snprintf(err, errlen, "cuTensorMapEncodeTiled (fp32) failed (%d)", (int)r);
    return 3;
  }
  map_cache().put(key, *map);
  return 0;
}

// ---------------------------------------------------------------- forward kernels
// Common shape of passes 1-3: 256 threads = two warpgroups.  Warp w reads TMEM
// lanes 32*(w%4).., so both warpgroups see all 128 lanes of a 128x128 score tile
// and split its COLUMNS: warpgroup 0 takes columns 0-63, warpgroup 1 columns 64-127.
// Thread 0 issues TMA and MMA.  One score buffer in TMEM per CTA; several CTAs per
// SM overlap each other's MMA/TMA latency.

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// bf16 pair of what `hi` (a packed pair of the rounded values) leaves of (a, b): the lo plane of a split value.
__device__ __forceinline__ uint32_t pack_bf16_rest(float a, float b, uint32_t hi) {
  return pack_bf16(a - __uint_as_float(hi << 16), b - __uint_as_float(hi & 0xffff0000u));
}

// Both parts of two fp32 values that come from outside, hi + lo.  An infinity is +-1 + +-inf: the products with another value
// that are taken (hi hi, hi lo, lo hi) then add up to what the infinity itself gives, of the right sign, NaN with 0
// — as inf + 0 the hi lo product would be inf * 0, as inf + (inf - inf) all of them are NaN.  A finite value past the largest
// bf16 is cut, not rounded to inf.  Everything else is rounded.
__device__ __forceinline__ void split_pair(float a, float b, uint32_t& hi, uint32_t& lo) {
  constexpr float kRoundsToInf = 3.3961775292304601e38f;   // 2^128 - 2^119: half a unit past the largest bf16
  float x[2] = {a, b}, rest[2];
  bool inf[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    inf[i] = isinf(x[i]);
    rest[i] = x[i];
    if (inf[i]) x[i] = copysignf(1.f, x[i]);
    else if (fabsf(x[i]) >= kRoundsToInf) x[i] = __uint_as_float(__float_as_uint(x[i]) & 0xffff0000u);
  }
  hi = pack_bf16(x[0], x[1]);
  if (!inf[0]) rest[0] -= __uint_as_float(hi << 16);
  if (!inf[1]) rest[1] -= __uint_as_float(hi & 0xffff0000u);
  lo = pack_bf16(rest[0], rest[1]);
}

// 32 columns of one output row; kSplit rows end after `left` columns (a multiple of 16).
template <int W>
__device__ __forceinline__ void store_row32(float* dst, const float* m, int left) {
#pragma unroll
  for (int e = 0; e < 32; e += 4)
    if (W != kSplit || e < left) *reinterpret_cast<float4*>(dst + e) = make_float4(m[e], m[e + 1], m[e + 2], m[e + 3]);
}
template <int W>
__device__ __forceinline__ void store_row32(__nv_bfloat16* dst, const float* m, int) {
#pragma unroll
  for (int e = 0; e < 32; e += 8)
    *reinterpret_cast<uint4*>(dst + e) = make_uint4(pack_bf16(m[e], m[e + 1]), pack_bf16(m[e + 2], m[e + 3]),
                                                    pack_bf16(m[e + 4], m[e + 5]), pack_bf16(m[e + 6], m[e + 7]));
}

// 1/a and 1/b, two consecutive demands of a key.  PAIR: from one special-function operation, of which the passes that form
// shares are short, and the product of the two, instead of two; a NaN b leaves 1/a alone.  For demands between 1e-18 and
// 1e18 (pair_demands); two more roundings, 1e-7.  Main pass of the sigmoid bid 0.883 -> 0.777 ms (n = 32, T = 8192), of
// 384 rows of 1024 tokens 206 -> 197 us.  In the reverse passes, whose two warps per scheduler wait for each other
// rather than for that unit, it loses: 10.5 -> 10.9 ms (n = 64, T = 16384).
template <bool PAIR>
__device__ __forceinline__ float2 rcp_two(float a, float b) {
  if (!PAIR) return make_float2(fast_rcp(a), fast_rcp(b));
  const float m = fminf(b, 1e18f);
  const float r = fast_rcp(a * m);
  return mul2(make_float2(r, r), make_float2(m, a));
}
// Whether every demand of a call stays in that range: eps in front, bids of at most 1 (expshift has no row sum: any size).
// Demands that a caller hands in (carry_base) are held at the upper end, where a share is nothing: capped_demand.
inline bool pair_demands(const Geom& g) {
  return g.eps >= 1e-18f && g.eps <= 1e18f && (g.normalised || g.bid == kBidSigmoid);
}
template <bool PAIR, int SHARE>
__device__ __forceinline__ float capped_demand(float d) {
  return PAIR && SHARE == kShareInclusive && d > 1e18f ? 1e18f : d;      // (a NaN stays one)
}

// Byte offset of the 16-byte chunk holding queries [q, q+8) of `key` in an
// MN-major [128 keys][128 queries] bf16 tile (q a multiple of 8): two 64-query
// sub-tiles of 16 KB, rows of 128 B, 16-byte chunks XOR-swizzled by the row.
__device__ __forceinline__ uint32_t share_chunk_offset(int key, int q) {
  return (uint32_t)((q >> 6) * (int)kTileBytes + key * 128 + ((((q & 63) >> 3) ^ (key & 7)) << 4));
}

// f of the f(a) / rowsum(f) bids up to a constant (mass_scale) that sits in the per-query factor:
// relu max(s, 0), relu2 the same before the square, softplus log2(1 + 2^z) with z = s * zscale.
// POLY: the exponential on the FMA pipe.
template <int BID, bool POLY = false>
__device__ __forceinline__ float mass_term(float s, float zscale) {
  if (BID != kBidSoftplus) return fmaxf(s, 0.f);
  const float z = s * zscale;
  const float e = POLY ? poly_exp2<4>(-fabsf(z)) : fast_exp2(-fabsf(z));
  float top;                                           // max(z, 0) that keeps a NaN, which the polynomial does not
  asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(top) : "f"(z));
  return top + fast_log2(1.f + e);
}
template <int BID> __device__ __forceinline__ float mass_power(float f) { return BID == kBidRelu2 ? f * f : f; }
__device__ __forceinline__ float mass_factor(float mass, int i, float mass_scale) {
  // (a NaN mass stays one: mass_bid hands it on)
  return mass > 0.f ? mass_scale / mass : mass <= 0.f ? -1.f / (float)(i + 1) : mass;
}
__device__ __forceinline__ float mass_bid(float fp, float l) { return l >= 0.f ? fp * l : -l; }

// Whether the masks of a kernel end at the last query too.  A query behind it is a row of zeros with a log-sum-exp of +inf, so
// that it bids 0 for every finite key, but zero times an infinite key is NaN.  The element-wise bids and softmax of
// bf16 heads of 64 leave that out: in a long row's passes it is 1% (24.4 -> 24.6 ms at n = 64, T = 16384).
template <int W, int BID> constexpr bool kMaskEnd = W != kNarrow || row_sum_bid(BID);

// log2-domain log-sum-exp of query i (+inf past the end, so that its p is 0).  The sigmoid bid
// and the shifted bids have no row statistics: their "lse" is log2 of the shift (0 for the plain
// sigmoid) for a query that exists and +inf past the end.
//
// An f(a) / rowsum(f) bid (q_off = 0) has one factor per query instead: l = lshift / (row mass), with lshift the
// constant that turns mass_term into f, so that the bid is mass_term * l; -1 / (keys in the window) for a row
// without mass, which bids that uniformly; 0 past the end.
template <int BID = kBidSoftmax>
__device__ __forceinline__ float load_lse(const float* __restrict__ rmax, const float* __restrict__ rden,
                                          int64_t row_base, int i, int tq, float lshift = 0.f) {
  if (row_sum_bid(BID)) return i < tq ? mass_factor(rden[row_base + i], i, lshift) : 0.f;
  if (BID == kBidSigmoid || rmax == nullptr) return i < tq ? lshift : INFINITY;   // no row statistics
  return i < tq ? rmax[row_base + i] + log2f(rden[row_base + i]) : INFINITY;
}

// The bid of one raw score s (kernels_bid.py:191-204) given the row's lse l:
// softmax 2^(s*zscale - l); sigmoid 1 / (1 + 2^(l - s*zscale)), which is 0 for l = +inf.  POLY: softplus's exponential on
// the FMA pipe.
template <int BID, bool POLY = false>
__device__ __forceinline__ float bid_p(float s, float zscale, float l) {
  if (row_sum_bid(BID)) return mass_bid(mass_power<BID>(mass_term<BID, POLY>(s, zscale)), l);
  if (BID == kBidSigmoid) return fast_rcp(1.f + fast_exp2(fmaf(s, -zscale, l)));
  return fast_exp2(fmaf(s, zscale, -l));
}

// ---------------------------------------------------------------- pass 1: row statistics
// grid = n * ceil(tq/128), longest rows first.  S = Q K^T, lane = query: each
// thread reduces its 64 key columns of the tile with an online max / sum; the two
// halves of a row are merged once at the end.  TMEM: 128 columns; 4 CTAs per SM.
template <int W> constexpr int kRowstatsSmem = 3 * (int)Rows<W>::kBytes + 1024 + 1024 + 256;

// BID: an f(a) / rowsum(f) bid takes the row's mass instead (rmax is 0 then, rden the mass).
template <int W = kNarrow, int BID = kBidSoftmax>
__global__ void __launch_bounds__(256, W == kNarrow ? 4 : 2) rowstats_kernel(const __grid_constant__ CUtensorMap map_q,
                                                          const __grid_constant__ CUtensorMap map_k,
                                                          Geom g, float* __restrict__ rmax,
                                                          float* __restrict__ rden) {
  constexpr uint32_t TB = Rows<W>::kBytes;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  const uint32_t sQ = smem_u32(smem), sK0 = sQ + TB;
  float2* sMerge = reinterpret_cast<float2*>(smem + 3 * TB);          // [128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 3 * TB + 1024);
  Ctl* ctl = reinterpret_cast<Ctl*>(bars + 8);
  const uint32_t kfull = smem_u32(bars), sdone = smem_u32(bars + 2);

  const int tid = threadIdx.x, warp = tid >> 5, wg = tid >> 7, row = tid & 127;
  const int warp_u = uniform_warp();
  const uint32_t lead = elect_one();
  const int nqb = (g.tq + kTileRows - 1) / kTileRows;
  const int n = (int)(blockIdx.x % g.n);
  const int ib = nqb - 1 - (int)(blockIdx.x / g.n);
  const int q0 = g.q_off + ib * kTileRows;
  const int njb = min(g.tk - 1, q0 + kTileRows - 1) / kTileRows + 1;

  if (tid == 0) {
    ctl->abort = 0;
    for (int i = 0; i < 3; ++i) mbar_init(kfull + 8 * i, 1);
    fence_barrier_init();
  }
  __syncwarp();
  if (warp == 0) tmem_alloc(smem_u32(&ctl->tmem), 128);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = uniform(ctl->tmem);

  if (tid == 0) {
    mbar_expect_tx(kfull, 2 * TB);
    tma_load_rows<W>(sQ, &map_q, ib * kTileRows, n, kfull);
    tma_load_rows<W>(sK0, &map_k, 0, n, kfull);
    if (njb > 1) {
      mbar_expect_tx(kfull + 8, TB);
      tma_load_rows<W>(sK0 + TB, &map_k, kTileRows, n, kfull + 8);
    }
  }
  float m = -INFINITY, s = 0.f;
  const int ia = q0 + row;
  const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + 64 * wg;
  for (int jb = 0; jb < njb; ++jb) {
    const int b = jb & 1;
    if (warp_u == 0) {
      mbar_wait(kfull + 8 * b, (jb >> 1) & 1, ctl, &g_status, kErrWaitTma);
      tc_fence_after();
      mma_scores_w<W>(lead, tmem, sQ, sK0 + TB * b, 128);
      mma_commit(lead, sdone);
    }
    __syncwarp();
    mbar_wait(sdone, jb & 1, ctl, &g_status, kErrWaitMma);
    tc_fence_after();
    if (tid == 0 && jb + 2 < njb) {     // this K stage is free again
      mbar_expect_tx(kfull + 8 * b, TB);
      tma_load_rows<W>(sK0 + TB * b, &map_k, (jb + 2) * kTileRows, n, kfull + 8 * b);
    }
    __syncwarp();
    const bool edge = (jb * kTileRows + kTileRows - 1 > q0) || ((jb + 1) * kTileRows > g.tk);
    // the mask arithmetic exists only in the instantiation used for edge tiles
    auto tile = [&](auto edge_tag) {
      constexpr bool EDGE = decltype(edge_tag)::value;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        float v[32];
        tmem_ld32(taddr + 32 * c, v);
        tmem_ld_wait(v);
        if (row_sum_bid(BID)) {
          float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            const int ja = jb * kTileRows + wg * 64 + c * 32 + e;
            float f = (e & 3) == 3 ? mass_term<BID, true>(v[e], g.zscale) : mass_term<BID>(v[e], g.zscale);
            if (EDGE && (ja > ia || ja >= g.tk)) f = 0.f;
            part[e & 3] += mass_power<BID>(f);
          }
          s += (part[0] + part[1]) + (part[2] + part[3]);
          continue;
        }
        float cmax = -INFINITY;          // max of the raw scores (zscale > 0 keeps the order)
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          if (EDGE) {
            const int ja = jb * kTileRows + wg * 64 + c * 32 + e;
            if (ja > ia || ja >= g.tk) v[e] = -INFINITY;
          }
          cmax = fmaxf(cmax, v[e]);
        }
        // No branch on the scores: a row without a finite one so far (a NaN query, all scores -inf) takes the path of
        // every other row with the reference 0, and what it adds up is scaled by 0 once a reference exists.  A lane
        // that went another way would still be apart from its warp at the warp-wide tcgen05.ld of the next
        // chunk and at the tcgen05.dealloc behind the last one.
        const float nm = fmaxf(m, cmax * g.zscale), ref = nm > -INFINITY ? nm : 0.f;
        float ps = 0.f;
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          // the pass is bound by the special-function unit: every fourth exponential
          // is a polynomial on the FMA pipe instead
          const float z = fmaf(v[e], g.zscale, -ref);
          ps += (e & 3) == 3 ? poly_exp2<4, W != kNarrow>(z) : fast_exp2(z);
        }
        s = s * fast_exp2(m - ref) + ps;
        m = nm;
      }
    };
    if (edge) tile(std::true_type{}); else tile(std::false_type{});
    tc_fence_before();
    __syncthreads();
  }
  if (wg == 1) sMerge[row] = make_float2(m, s);
  __syncthreads();
  const int i = ib * kTileRows + row;
  if (wg == 0 && i < g.tq) {
    const float2 o = sMerge[row];
    if (row_sum_bid(BID)) {
      rmax[(int64_t)n * g.tq + i] = 0.f;
      rden[(int64_t)n * g.tq + i] = (s + o.y) * g.lshift;
    } else {
    const float nm = fmaxf(m, o.x);          // finite: the first tile always holds key 0
    const float tot = s * fast_exp2(m - nm) + o.y * fast_exp2(o.x - nm);
    rmax[(int64_t)n * g.tq + i] = nm;
    rden[(int64_t)n * g.tq + i] = tot;
    }
  }
  drain_if_aborted(ctl);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_free(tmem, 128);
}

// ---------------------------------------------------------------- pass 2: column sums + scan
// grid = n * ceil(tk/128), key blocks with the most query blocks first.
// S^T = K Q^T, lane = key.  The CTA keeps its K tile and walks the query blocks
// in causal order.  Each warpgroup sums p over its 64 queries of the tile, 32 at a
// time; the thread of warpgroup 0 owns the key's running sum — the exclusive scan —
// and stores one checkpoint per CR query rows, one tile behind the sums.  CR = 32 when
// a backward will read the checkpoints (two threads per key there, 32 queries each),
// 64 for forward-only calls (the main forward pass starts its two warpgroups at queries
// 0 and 64 of a tile): half the scratch and half the checkpoint stores.
template <int W> constexpr int kColsumSmem = 3 * (int)Rows<W>::kBytes + 1024 + 2048 + 1024 + 256;

template <int CR, int BID = kBidSoftmax, int W = kNarrow>
__global__ void __launch_bounds__(256, W != kNarrow ? 2 : row_sum_bid(BID) ? 3 : 4) colsum_scan_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, Geom g,
    const float* __restrict__ rmax, const float* __restrict__ rden,
    const float* __restrict__ carry_base, float* __restrict__ carry, float* __restrict__ total) {
  static_assert(CR == 32 || CR == 64, "checkpoints every 32 or 64 query rows");
  constexpr int kPerTile = kTileRows / CR;                                      // 4 or 2
  constexpr uint32_t TB = Rows<W>::kBytes;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  const uint32_t sK = smem_u32(smem), sQ0 = sK + TB;
  float* sL = reinterpret_cast<float*>(smem + 3 * TB);                 // [2][128]
  float2* sCs = reinterpret_cast<float2*>(smem + 3 * TB + 1024);       // [2][128] the two sums of warpgroup 1
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 3 * TB + 3072);
  Ctl* ctl = reinterpret_cast<Ctl*>(bars + 8);
  const uint32_t qfull = smem_u32(bars), sdone = smem_u32(bars + 2);

  const int tid = threadIdx.x, warp = tid >> 5, wg = tid >> 7, row = tid & 127;
  const int warp_u = uniform_warp();
  const uint32_t lead = elect_one();
  const int nqb = (g.tq + kTileRows - 1) / kTileRows;
  const int ncb = (g.tq + CR - 1) / CR;
  const int n = (int)(blockIdx.x % g.n);
  const int jb = (int)(blockIdx.x / g.n);
  const int k0 = jb * kTileRows;
  const int ib0 = k0 > g.q_off ? (k0 - g.q_off) / kTileRows : 0;     // first block that sees these keys
  const int nib = nqb - ib0;                                          // may be <= 0
  const int64_t row_base = (int64_t)n * g.tq;

  if (tid == 0) {
    ctl->abort = 0;
    for (int i = 0; i < 3; ++i) mbar_init(qfull + 8 * i, 1);
    fence_barrier_init();
  }
  __syncwarp();
  if (warp == 0) tmem_alloc(smem_u32(&ctl->tmem), 128);
  if (nib > 0 && wg == 0) sL[row] = load_lse<BID>(rmax, rden, row_base, ib0 * kTileRows + row, g.tq, g.lshift);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = uniform(ctl->tmem);

  if (tid == 0 && nib > 0) {
    mbar_expect_tx(qfull, 2 * TB);
    tma_load_rows<W>(sK, &map_k, k0, n, qfull);
    tma_load_rows<W>(sQ0, &map_q, ib0 * kTileRows, n, qfull);
    if (nib > 1) {
      mbar_expect_tx(qfull + 8, TB);
      tma_load_rows<W>(sQ0 + TB, &map_q, (ib0 + 1) * kTileRows, n, qfull + 8);
    }
  }
  const int ja = k0 + row;
  const bool live = ja < g.tk;
  const float base = (carry_base != nullptr && live) ? carry_base[(int64_t)n * g.tk + ja] : 0.f;
  float local = 0.f, prev0 = 0.f, prev1 = 0.f;   // warpgroup 0: scan state, its two sums of the previous tile
  // the checkpoints of 128-row tile `tile` (in front of its queries 0, 32, 64, 96 — or 0 and 64),
  // and the scan moved past it
  auto store_checkpoints = [&](int tile, float2 w1) {
    const int rb = tile * kPerTile;
    const float c0 = base + local, c1 = c0 + prev0, c2 = c1 + prev1, c3 = c2 + w1.x;
    if (live) {
      const int64_t o = ((int64_t)n * ncb + rb) * g.tk + ja;
      if (CR == 32) {
        if (rb < ncb) carry[o] = c0;
        if (rb + 1 < ncb) carry[o + g.tk] = c1;
        if (rb + 2 < ncb) carry[o + 2 * (int64_t)g.tk] = c2;
        if (rb + 3 < ncb) carry[o + 3 * (int64_t)g.tk] = c3;
      } else {
        if (rb < ncb) carry[o] = c0;
        if (rb + 1 < ncb) carry[o + g.tk] = c2;
      }
    }
    local += (prev0 + prev1) + (w1.x + w1.y);
  };
  const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + 64 * wg;
  for (int it = 0; it < nib; ++it) {
    const int ib = ib0 + it, b = it & 1;
    if (warp_u == 0) {
      mbar_wait(qfull + 8 * b, (it >> 1) & 1, ctl, &g_status, kErrWaitTma);
      tc_fence_after();
      mma_scores_w<W>(lead, tmem, sK, sQ0 + TB * b, 128);
      mma_commit(lead, sdone);
    }
    __syncwarp();
    // while the MMA runs: next tile's statistics, and the checkpoints of the previous tile
    float lse_next = 0.f;
    if (wg == 1 && it + 1 < nib) lse_next = load_lse<BID>(rmax, rden, row_base, (ib + 1) * kTileRows + row, g.tq, g.lshift);
    if (wg == 0 && it > 0) store_checkpoints(ib - 1, sCs[((it - 1) & 1) * 128 + row]);
    mbar_wait(sdone, it & 1, ctl, &g_status, kErrWaitMma);
    tc_fence_after();
    if (tid == 0 && it + 2 < nib) {
      mbar_expect_tx(qfull + 8 * b, TB);
      tma_load_rows<W>(sQ0 + TB * b, &map_q, (ib + 2) * kTileRows, n, qfull + 8 * b);
    }
    __syncwarp();
    const int i0 = g.q_off + ib * kTileRows + 64 * wg;   // absolute position of this half's first query
    const int qend = g.q_off + g.tq;
    const bool edge = i0 < k0 + kTileRows - 1 ||                      // part of the diagonal tile, or a ragged last one
                      (kMaskEnd<W, BID> && i0 + 64 > qend);
    const float4* L4 = reinterpret_cast<const float4*>(sL + 128 * b + 64 * wg);
    float colsum0 = 0.f, colsum1 = 0.f;      // queries 0-31 and 32-63 of this warpgroup's half
    auto tile = [&](auto edge_tag) {
      constexpr bool EDGE = decltype(edge_tag)::value;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        float v[32];
        tmem_ld32(taddr + 32 * c, v);
        tmem_ld_wait(v);
        float part[4] = {0.f, 0.f, 0.f, 0.f};     // four independent sums
#pragma unroll
        for (int e4 = 0; e4 < 8; ++e4) {
          const float4 l = L4[c * 8 + e4];
          const float ls[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            float p = bid_p<BID>(v[e4 * 4 + u], g.zscale, ls[u]);
            const int i = i0 + c * 32 + e4 * 4 + u;
            if (EDGE && (ja > i || (kMaskEnd<W, BID> && i >= qend))) p = 0.f;
            part[u] += p;
          }
        }
        const float cs = (part[0] + part[1]) + (part[2] + part[3]);
        if (c == 0) colsum0 = cs; else colsum1 = cs;
      }
    };
    if (edge) tile(std::true_type{}); else tile(std::false_type{});
    if (wg == 0) {
      prev0 = colsum0;
      prev1 = colsum1;
    } else {
      sCs[b * 128 + row] = make_float2(colsum0, colsum1);
    }
    if (wg == 1 && it + 1 < nib) sL[128 * (b ^ 1) + row] = lse_next;
    tc_fence_before();
    __syncthreads();
  }
  if (wg == 0 && live) {
    if (nib > 0) store_checkpoints(nqb - 1, sCs[((nib - 1) & 1) * 128 + row]);
    total[(int64_t)n * g.tk + ja] = local;
  }
  drain_if_aborted(ctl);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_free(tmem, 128);
}

// ---------------------------------------------------------------- pass 3: main pass
// grid = n * ceil(tq/128), longest rows first.  S^T = K Q^T, lane = key.
// Each thread walks 64 queries of the tile in order (warpgroup 1 starts from the
// mid-block checkpoint) with its key's demand in one register:
//     den += p;  share = p / den          (den = committed + p + eps)
// and writes its half of the bf16 share tile to shared memory as an MN-major
// operand ([key][query]).  Two MMAs consume the tile:
//   O   [query x d ] += share * V      (A = share MN-major, B = V MN-major)
//   rs  [query x 16] += share * ones   (row sums of the SAME bf16 shares)
// so the final divide out = O / (rs + eps) normalises exactly what was summed.
// TMEM: S^T 128 columns, O 64, rs 16 (256 allocated; two CTAs per SM).
// Q, K[2], V, ones, shares (two 64-query sub-tiles per plane); exact: the base must already be 1024-aligned
template <int W> constexpr int kMainSmem =
    4 * (int)Rows<W>::kBytes + (1 + 2 * Rows<W>::kPlanes) * (int)kTileBytes + 512 + 128;

// BID: softmax, or expshift, whose log-sum-exp is a constant and whose bids have no upper end.  SHARE selects the ablations of
// kernels_bid.py (exclusive or absent share step, :254-262); the default instantiation is the operator.
template <int SHARE = kShareInclusive, bool PAIR = true, int BID = kBidSoftmax>
__global__ void __launch_bounds__(256, 2) forward_main_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
    const __grid_constant__ CUtensorMap map_v, Geom g, const float* __restrict__ rmax,
    const float* __restrict__ rden, const float* __restrict__ carry,
    const float* __restrict__ carry_base, float* __restrict__ out, float* __restrict__ ssum) {
  constexpr int W = kNarrow;
  constexpr uint32_t TB = Rows<W>::kBytes;
  constexpr int kOCols = Rows<W>::kCols + 16;        // O and the row sums: one tile
  constexpr int kTmem = 256;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if (smem_u32(smem) & 1023u) {                      // no slack is requested: refuse instead of overrunning
    if (threadIdx.x == 0) atomicCAS(&g_status, 0, kErrAlign);
    return;
  }
  const uint32_t sQ = smem_u32(smem), sK0 = sQ + TB, sV = sQ + 3 * TB;
  // a [128 keys][64] bf16 tile of ones right behind V: the last 64-column group of the B
  // operand of share @ [V | ones] (N = 80), so the row sums come out of the same MMA
  const uint32_t sOnes = sQ + 4 * TB, sSh = sOnes + kTileBytes;
  uint8_t* ones_ptr = smem + 4 * TB;
  float* sL = reinterpret_cast<float*>(smem + 4 * TB + 3 * kTileBytes);
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(sL) + 512);
  Ctl* ctl = reinterpret_cast<Ctl*>(bars + 8);
  const uint32_t kfull = smem_u32(bars), vfull = smem_u32(bars + 2), sdone = smem_u32(bars + 3);

  const int tid = threadIdx.x, warp = tid >> 5, wg = tid >> 7, row = tid & 127;
  const int warp_u = uniform_warp();
  const uint32_t lead = elect_one();
  const int nqb = (g.tq + kTileRows - 1) / kTileRows;
  const int ncb = (g.tq + g.carry_rows - 1) / g.carry_rows;
  const int n = (int)(blockIdx.x % g.n);
  const int ib = nqb - 1 - (int)(blockIdx.x / g.n);
  const int q0 = g.q_off + ib * kTileRows;
  const int njb = min(g.tk - 1, q0 + kTileRows - 1) / kTileRows + 1;

  if (tid == 0) {
    ctl->abort = 0;
    for (int i = 0; i < 4; ++i) mbar_init(kfull + 8 * i, 1);
    fence_barrier_init();
  }
  __syncwarp();
  if (warp == 0) tmem_alloc(smem_u32(&ctl->tmem), kTmem);
  if (wg == 0) sL[row] = load_lse<kBidSoftmax>(rmax, rden, (int64_t)n * g.tq, ib * kTileRows + row, g.tq, g.lshift);
  else {
#pragma unroll
    for (int c = 0; c < 8; ++c)
      reinterpret_cast<uint4*>(ones_ptr)[row * 8 + c] = make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u);
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = uniform(ctl->tmem);
  const uint32_t tS = tmem, tO = tmem + 128, tR = tO + Rows<W>::kCols;

  if (tid == 0) {
    mbar_expect_tx(kfull, 2 * TB);
    tma_load_rows<W>(sQ, &map_q, ib * kTileRows, n, kfull);
    tma_load_rows<W>(sK0, &map_k, 0, n, kfull);
    mbar_expect_tx(vfull, TB);
    tma_load_rows<W>(sV, &map_v, 0, n, vfull);
    if (njb > 1) {
      mbar_expect_tx(kfull + 8, TB);
      tma_load_rows<W>(sK0 + TB, &map_k, kTileRows, n, kfull + 8);
    }
  }
  if (warp_u == 0) {
    __syncwarp();
    mbar_wait(kfull, 0, ctl, &g_status, kErrWaitTma);
    tc_fence_after();
    mma_scores_w<W>(lead, tS, sK0, sQ, 128);
    mma_commit(lead, sdone);
  }
  __syncwarp();

  // the checkpoint row this warpgroup starts from: the one in front of query 0 / query 64 of the block
  const int rb = (ib * kTileRows + 64 * wg) / g.carry_rows;
  const bool have_rows = rb < ncb;                 // false only for a ragged last half block
  const int64_t carry_row = ((int64_t)n * ncb + (have_rows ? rb : 0)) * g.tk;
  const float4* L4 = reinterpret_cast<const float4*>(sL + 64 * wg);
  const uint32_t taddr = tS + ((uint32_t)((warp & 3) * 32) << 16) + 64 * wg;
  const int qh = q0 + 64 * wg;                     // absolute position of this half's first query
  auto load_den = [&](int jbx) {
    const int jx = jbx * kTileRows + row;
    float d = g.eps;
    if (SHARE != kShareNone && jx < g.tk && have_rows) {      // no share step: no demand is read
      d += carry[carry_row + jx];
      if (carry_base != nullptr) d += carry_base[(int64_t)n * g.tk + jx];
    }
    return capped_demand<PAIR, SHARE>(d);
  };
  float den_next = load_den(0);
  for (int jb = 0; jb < njb; ++jb) {
    const int b = jb & 1;
    const int ja = jb * kTileRows + row;
    float den = den_next;
    mbar_wait(sdone, jb & 1, ctl, &g_status, kErrWaitMma);
    tc_fence_after();
    if (tid == 0) {
      if (jb >= 1) {                      // the V buffer is free: the previous share*V finished
        mbar_expect_tx(vfull, TB);
        tma_load_rows<W>(sV, &map_v, jb * kTileRows, n, vfull);
      }
      if (jb >= 1 && jb + 1 < njb) {      // K stage of tile jb-1 is free
        mbar_expect_tx(kfull + 8 * (b ^ 1), TB);
        tma_load_rows<W>(sK0 + TB * (b ^ 1), &map_k, (jb + 1) * kTileRows, n, kfull + 8 * (b ^ 1));
      }
    }
    __syncwarp();
    if (jb + 1 < njb) den_next = load_den(jb + 1);   // lands while this tile is processed
    const bool diag = jb * kTileRows + kTileRows - 1 > qh;
    const bool dead = ja >= g.tk;
    auto tile = [&](auto mask_tag) {
    constexpr bool MASK = decltype(mask_tag)::value;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      float v[32];
      tmem_ld32(taddr + 32 * c, v);
      tmem_ld_wait(v);
      // the statistics of group e8+1 are read before group e8 is stored: shared-memory
      // loads cannot be hoisted above the stores by the compiler
      float4 lnext[2] = {L4[c * 8], L4[c * 8 + 1]};
#pragma unroll
      for (int e8 = 0; e8 < 4; ++e8) {
        uint32_t packed[4];
        const float4 lcur[2] = {lnext[0], lnext[1]};
        if (e8 < 3) {
          lnext[0] = L4[c * 8 + e8 * 2 + 2];
          lnext[1] = L4[c * 8 + e8 * 2 + 3];
        }
        // two special-function ops per score bind this pass: every fourth exponential of the
        // softmax bid is a polynomial on the FMA pipe (79.7 -> 75.3 ms at the 128K prefill shape)
        float2 fourth = make_float2(fmaf(v[e8 * 8 + 3], g.zscale, -lcur[0].w), fmaf(v[e8 * 8 + 7], g.zscale, -lcur[1].w));
        if (BID == kBidExpshift) {                           // exponents past 128: as in the fused sweep
          fourth = poly_exp2_two<4>(make_float2(min_nan(fourth.x - 1.f, 128.f), min_nan(fourth.y - 1.f, 128.f)));
          fourth = add2(fourth, fourth);
        } else {
          fourth = poly_exp2_two<4>(fourth);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float ls[4] = {lcur[h].x, lcur[h].y, lcur[h].z, lcur[h].w};
          float sh[4], dn[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int e = e8 * 8 + h * 4 + u;
            float p = u < 3 ? bid_p<kBidSoftmax>(v[e], g.zscale, ls[u]) : h == 0 ? fourth.x : fourth.y;
            if (MASK && (dead || ja > qh + c * 32 + e)) p = 0.f;
            if (SHARE == kShareInclusive) {
              den += p;
              sh[u] = p;
              dn[u] = den;
            } else if (SHARE == kShareExclusive) {     // earlier queries' demand only
              sh[u] = p * fast_rcp(den);
              den += p;
            } else {                                   // no share step
              sh[u] = p;
            }
          }
          if (SHARE == kShareInclusive) {
#pragma unroll
            for (int u = 0; u < 4; u += 2) {
              const float2 s2 = mul2(make_float2(sh[u], sh[u + 1]), rcp_two<PAIR>(dn[u], dn[u + 1]));
              sh[u] = s2.x;
              sh[u + 1] = s2.y;
            }
          }
          packed[h * 2 + 0] = pack_bf16(sh[0], sh[1]);
          packed[h * 2 + 1] = pack_bf16(sh[2], sh[3]);
        }
        const uint32_t dst = sSh + share_chunk_offset(row, wg * 64 + c * 32 + e8 * 8);
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(packed[0]),
                     "r"(packed[1]), "r"(packed[2]), "r"(packed[3])
                     : "memory");
      }
    }
    };
    // (by whole warps: the TMEM loads are warp-wide, and the keys of a row may end in the middle of one)
    if (__any_sync(0xffffffffu, diag || dead)) tile(std::true_type{}); else tile(std::false_type{});
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    if (warp_u == 0) {
      tc_fence_after();
      mbar_wait(vfull, jb & 1, ctl, &g_status, kErrWaitTma);
      tc_fence_after();
      constexpr uint32_t id_o = instr_desc(128, kOCols, 1, 1);
      // descriptors are built once per tile; a k-step is a constant 2048 B (128 units) further
      const Desc dSh = make_desc(sSh, kTileBytes, 1024), dVm = make_desc(sV, kTileBytes, 1024);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) mma_ss(lead, tO, dSh, 128 * kk, dVm, 128 * kk, id_o, (jb > 0 || kk > 0));
      if (jb + 1 < njb) {
        mbar_wait(kfull + 8 * (b ^ 1), ((jb + 1) >> 1) & 1, ctl, &g_status, kErrWaitTma);
        tc_fence_after();
        mma_scores_w<W>(lead, tS, sK0 + TB * (b ^ 1), sQ, 128);
      }
      mma_commit(lead, sdone);
    }
    __syncwarp();
  }
  mbar_wait_warp(sdone, njb & 1, ctl, &g_status, kErrWaitMma);
  tc_fence_after();
  {
    // lane = query now: each warpgroup stores half of the output columns of row `row`, 32 at a time
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    constexpr int kHalf = kHeadDim / 2;
    const int i = ib * kTileRows + row;
    float rs;
    tmem_ld1(tR + lane_base, &rs);
    tmem_ld_wait1(&rs);
    float o[32];
    tmem_ld32(tO + lane_base + kHalf * wg, o);
    tmem_ld_wait(o);
    const float inv = 1.f / (rs + g.eps);
    if (i < g.tq) {
      float4* dst = reinterpret_cast<float4*>(out + ((int64_t)n * g.tq + i) * kHeadDim + kHalf * wg);
#pragma unroll
      for (int c = 0; c < 8; ++c) dst[c] = make_float4(o[4 * c] * inv, o[4 * c + 1] * inv, o[4 * c + 2] * inv, o[4 * c + 3] * inv);
    }
    if (i < g.tq && wg == 0) ssum[(int64_t)n * g.tq + i] = rs;
  }
  drain_if_aborted(ctl);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_free(tmem, kTmem);
}

// The main pass with its own issuing warp, for rows that leave room for one CTA per SM (W != kNarrow) and the
// bids of sigmoid form (sigmoid, sigshift).  The arithmetic is forward_main_kernel's.  A ninth warp issues every copy and product, so that
// no compute warp waits for another one's turn at the tensor pipe: the scores of tile jb + 1 are issued as soon as
// all warps have read those of tile jb (half of the arithmetic still ahead of them), and share V of tile jb runs under
// the arithmetic of tile jb + 1, whose first 32 shares per thread wait in registers until it has read the share tile.
// Where one CTA fills an SM nothing else hides those round trips: bf16 heads of 128 0.39 -> 0.30 ms (n = 32, T = 4096),
// softplus bid 1.55 -> 1.26 ms (n = 32, T = 8192); with two CTAs: sigmoid bid 0.98 -> 0.89 ms.  The softmax bid of heads
// of 64 stays on forward_main_kernel: its long rows run at the card's power limit, where this form is 1 to 3% slower
// (145.2 -> 148 ms for the passes of a 128K prompt, 16 heads).
// Compute warpgroups: with one CTA per SM two are two warps per scheduler, which leave it idle while they wait for each
// other's hand-over; four take 32 queries of a tile per thread instead of 64 (bf16 heads of 128 0.303 -> 0.277 ms, fp32 heads of
// 64 0.306 -> 0.277, softplus bid 1.205 -> 1.164 ms at the sizes above, both with reciprocals by pairs).  Where two CTAs share
// an SM there are four per scheduler already.
template <int W> constexpr int kMainGroups = W == kNarrow ? 2 : 4;
template <int W> constexpr int kMainThreads = 128 * kMainGroups<W> + 32;

// Shares as hi + lo make NaN of an infinite value (lo may be negative or 0).  Where an output is NaN and its row sum is not, the
// value is to blame: the output becomes the sum of the infinities that the row sees, NaN if they are of both signs or a
// value is NaN.  out: this lane's row, columns [col0, col1), if `row` says that there is one; i: its position, -1 where the row
// sum is NaN; vinf: where a row of v, `stride` apart, holds what is infinite (its lo plane under kSplit); keys: up to the
// warp's last row.  The warp walks in step, whatever the values: its release of TMEM follows.
__device__ __noinline__ void restore_infinities(float* out, const __nv_bfloat16* vinf, int stride, int keys, int i, bool row,
                                                int col0, int col1) {
  for (int c = col0; c < col1; ++c) {
    const float x = row ? out[c] : 0.f;
    const bool want = x != x && i >= 0;
    if (!__any_sync(0xffffffffu, want)) continue;
    float sum = 0.f;
    for (int j = 0; j < keys; ++j) {
      const float v = __bfloat162float(vinf[(int64_t)j * stride + c]);
      sum += j <= i && !(fabsf(v) < INFINITY) ? v : 0.f;
      if ((j & 63) == 63 && __all_sync(0xffffffffu, sum != sum || !want)) break;
    }
    const float y = want && sum != 0.f ? sum : x;
    if (row) out[c] = y;
  }
  __syncwarp();
}

template <int BID = kBidSoftmax, int SHARE = kShareInclusive, int W = kNarrow, bool PAIR = true>
__global__ void __launch_bounds__(kMainThreads<W>, W == kNarrow ? 2 : 1) forward_main_async_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
    const __grid_constant__ CUtensorMap map_v, Geom g, const float* __restrict__ rmax,
    const float* __restrict__ rden, const float* __restrict__ carry,
    const float* __restrict__ carry_base, const __nv_bfloat16* __restrict__ v_rows, float* __restrict__ out,
    float* __restrict__ ssum) {
  constexpr uint32_t TB = Rows<W>::kBytes;
  constexpr int P = Rows<W>::kPlanes;
  constexpr int NW = kMainGroups<W>, CW = kTileRows / NW;      // queries of a tile per thread
  constexpr int kOCols = Rows<W>::kCols + 16;        // O and the row sums: one tile
  constexpr int kTmem = W == kNarrow ? 256 : 512;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if (smem_u32(smem) & 1023u) {                      // no slack is requested: refuse instead of overrunning
    if (threadIdx.x == 0) atomicCAS(&g_status, 0, kErrAlign);
    return;
  }
  const uint32_t sQ = smem_u32(smem), sK0 = sQ + TB, sV = sQ + 3 * TB;
  // a [128 keys][64] bf16 tile of ones right behind V: the last 64-column group of the B
  // operand of share @ [V | ones] (N = 80 or 144), so the row sums come out of the same MMA
  const uint32_t sOnes = sQ + 4 * TB, sSh = sOnes + kTileBytes;
  uint8_t* ones_ptr = smem + 4 * TB;
  float* sL = reinterpret_cast<float*>(smem + 4 * TB + (1 + 2 * P) * kTileBytes);
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(sL) + 512);
  Ctl* ctl = reinterpret_cast<Ctl*>(bars + 8);
  const uint32_t kfull = smem_u32(bars), vfull = smem_u32(bars + 2), sdone = smem_u32(bars + 3);
  const uint32_t odone = smem_u32(bars + 4), sfree = smem_u32(bars + 5), shready = smem_u32(bars + 6);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, wg = tid >> 7, row = tid & 127;
  const int warp_u = uniform_warp();
  const uint32_t lead = elect_one();
  const int nqb = (g.tq + kTileRows - 1) / kTileRows;
  const int ncb = (g.tq + g.carry_rows - 1) / g.carry_rows;
  const int n = (int)(blockIdx.x % g.n);
  const int ib = nqb - 1 - (int)(blockIdx.x / g.n);
  const int q0 = g.q_off + ib * kTileRows;
  const int njb = min(g.tk - 1, q0 + kTileRows - 1) / kTileRows + 1;

  if (tid == 0) {
    ctl->abort = 0;
    for (int i = 0; i < 5; ++i) mbar_init(kfull + 8 * i, 1);      // kfull[2], vfull, sdone, odone
    mbar_init(sfree, 4 * NW);
    mbar_init(shready, 4 * NW);
    fence_barrier_init();
  }
  __syncwarp();
  if (warp == 0) tmem_alloc(smem_u32(&ctl->tmem), kTmem);
  if (wg == 0) sL[row] = load_lse<BID>(rmax, rden, (int64_t)n * g.tq, ib * kTileRows + row, g.tq, g.lshift);
  else if (wg == 1) {
#pragma unroll
    for (int c = 0; c < 8; ++c)
      reinterpret_cast<uint4*>(ones_ptr)[row * 8 + c] = make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u);
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = uniform(ctl->tmem);
  const uint32_t tS = tmem, tO = tmem + 128, tR = tO + Rows<W>::kCols;

  if (warp_u == 4 * NW) {
    if (lead) {
      mbar_expect_tx(kfull, 2 * TB);
      tma_load_rows<W>(sQ, &map_q, ib * kTileRows, n, kfull);
      tma_load_rows<W>(sK0, &map_k, 0, n, kfull);
      mbar_expect_tx(vfull, TB);
      tma_load_rows<W>(sV, &map_v, 0, n, vfull);
      if (njb > 1) {
        mbar_expect_tx(kfull + 8, TB);
        tma_load_rows<W>(sK0 + TB, &map_k, kTileRows, n, kfull + 8);
      }
    }
    {
      constexpr uint32_t id_s = instr_desc(128, 128, 0, 0), id_o = instr_desc(128, kOCols, 1, 1);
      // descriptors are built once; a k-step of O is a constant 2048 B (128 units) further
      const Desc dK0 = make_desc(sK0, 16, 1024), dK1 = make_desc(sK0 + TB, 16, 1024), dQ = make_desc(sQ, 16, 1024);
      const Desc dSh = make_desc(sSh, kTileBytes, 1024), dVm = make_desc(sV, kTileBytes, 1024);
      mbar_wait_warp(kfull, 0, ctl, &g_status, kErrWaitTma);
      tc_fence_after();
      mma_scores_wide<W>(lead, tS, dK0, kTileBytes, dQ, kTileBytes, id_s);
      mma_commit(lead, sdone);
      for (int jb = 0; jb < njb; ++jb) {
        const int b = jb & 1;
        if (jb + 1 < njb) {
          mbar_wait_warp(kfull + 8 * (b ^ 1), ((jb + 1) >> 1) & 1, ctl, &g_status, kErrWaitTma);
          mbar_wait_warp(sfree, jb & 1, ctl, &g_status, kErrWaitTile);
          tc_fence_after();
          mma_scores_wide<W>(lead, tS, b ? dK0 : dK1, kTileBytes, dQ, kTileBytes, id_s);
          mma_commit(lead, sdone);
          if (lead && jb + 2 < njb) {     // the scores of jb have been read, so its K stage is free
            mbar_expect_tx(kfull + 8 * b, TB);
            tma_load_rows<W>(sK0 + TB * b, &map_k, (jb + 2) * kTileRows, n, kfull + 8 * b);
          }
        }
        if (jb >= 1) {                    // V is free once the previous share V has completed
          mbar_wait_warp(odone, (jb - 1) & 1, ctl, &g_status, kErrWaitMma);
          if (lead) {
            mbar_expect_tx(vfull, TB);
            tma_load_rows<W>(sV, &map_v, jb * kTileRows, n, vfull);
          }
        }
        mbar_wait_warp(shready, jb & 1, ctl, &g_status, kErrWaitTile);
        mbar_wait_warp(vfull, jb & 1, ctl, &g_status, kErrWaitTma);
        tc_fence_after();
#pragma unroll
        for (int pl = 0; pl < P; ++pl)
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            mma_ss(lead, tO, dSh, 2048 * pl + 128 * kk, dVm, 128 * kk, id_o, (jb > 0 || pl > 0 || kk > 0));
        mma_commit(lead, odone);
      }
    }
    __syncwarp();
  } else {
  // the checkpoint row this warpgroup starts from: the one in front of its first query of the block
  const int rb = (ib * kTileRows + CW * wg) / g.carry_rows;
  const bool have_rows = rb < ncb;                 // false only in a ragged last block
  const int64_t carry_row = ((int64_t)n * ncb + (have_rows ? rb : 0)) * g.tk;
  const float4* L4 = reinterpret_cast<const float4*>(sL + CW * wg);
  const uint32_t taddr = tS + ((uint32_t)((warp & 3) * 32) << 16) + CW * wg;
  const int qh = q0 + CW * wg;                     // absolute position of this warpgroup's first query
  auto load_den = [&](int jbx) {
    const int jx = jbx * kTileRows + row;
    float d = g.eps;
    if (SHARE != kShareNone && jx < g.tk && have_rows) {      // no share step: no demand is read
      d += carry[carry_row + jx];
      if (carry_base != nullptr) d += carry_base[(int64_t)n * g.tk + jx];
    }
    return capped_demand<PAIR, SHARE>(d);
  };
  float den_next = load_den(0);
  for (int jb = 0; jb < njb; ++jb) {
    const int ja = jb * kTileRows + row;
    float den = den_next;
    if (jb + 1 < njb) den_next = load_den(jb + 1);   // lands while this tile is processed
    const bool dead = ja >= g.tk;
    const bool masked = dead || jb * kTileRows + kTileRows - 1 > qh;
    mbar_wait_warp(sdone, jb & 1, ctl, &g_status, kErrWaitMma);
    tc_fence_after();
#pragma unroll
    for (int c = 0; c < CW / 32; ++c) {
      float v[32];
      uint32_t packed[16], rest[P == 2 ? 16 : 1];
      tmem_ld32(taddr + 32 * c, v);
      tmem_ld_wait(v);
      if (c == CW / 32 - 1) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(sfree);
      }
      auto chunk = [&](auto mask_tag) {
        constexpr bool MASK = decltype(mask_tag)::value;
#pragma unroll
        for (int e8 = 0; e8 < 4; ++e8) {
          const float4 la = L4[c * 8 + 2 * e8], lb = L4[c * 8 + 2 * e8 + 1];
          const float ls[8] = {la.x, la.y, la.z, la.w, lb.x, lb.y, lb.z, lb.w};
          float p[8], r[8];
          if (BID == kBidSoftmax) {
            const float2 zs = make_float2(g.zscale, g.zscale);
            float2 z[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
              z[i] = fma2(make_float2(v[e8 * 8 + 2 * i], v[e8 * 8 + 2 * i + 1]), zs, make_float2(-ls[2 * i], -ls[2 * i + 1]));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              p[2 * i] = fast_exp2(z[i].x);
              p[2 * i + 1] = (i & 1) ? poly_exp2<4, W != kNarrow>(z[i].y) : fast_exp2(z[i].y);
            }
          } else {
#pragma unroll
            for (int u = 0; u < 8; ++u)
              p[u] = (u & 3) == 3 ? bid_p<BID, true>(v[e8 * 8 + u], g.zscale, ls[u]) : bid_p<BID>(v[e8 * 8 + u], g.zscale, ls[u]);
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            if (MASK && (dead || ja > qh + c * 32 + e8 * 8 + u)) p[u] = 0.f;
            if (SHARE == kShareExclusive) {            // earlier queries' demand only
              r[u] = fast_rcp(den);
              den += p[u];
            } else if (SHARE == kShareInclusive) {
              den += p[u];
              r[u] = den;
            }
          }
          if (SHARE == kShareInclusive) {
#pragma unroll
            for (int u = 0; u < 8; u += 2) {
              const float2 i2 = rcp_two<PAIR>(r[u], r[u + 1]);
              r[u] = i2.x;
              r[u + 1] = i2.y;
            }
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float2 s2 = make_float2(p[2 * i], p[2 * i + 1]);
            if (SHARE != kShareNone) s2 = mul2(s2, make_float2(r[2 * i], r[2 * i + 1]));
            const int o = 4 * e8 + i;
            packed[o] = pack_bf16(s2.x, s2.y);
            if (P == 2) rest[P == 2 ? o : 0] = pack_bf16_rest(s2.x, s2.y, packed[o]);
          }
        }
      };
      if (masked) chunk(std::true_type{}); else chunk(std::false_type{});
      if (c == 0 && jb >= 1) mbar_wait_warp(odone, (jb - 1) & 1, ctl, &g_status, kErrWaitMma);
#pragma unroll
      for (int e8 = 0; e8 < 4; ++e8) {
        const uint32_t dst = sSh + share_chunk_offset(row, wg * CW + c * 32 + e8 * 8);
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(packed[4 * e8]),
                     "r"(packed[4 * e8 + 1]), "r"(packed[4 * e8 + 2]), "r"(packed[4 * e8 + 3])
                     : "memory");
        if (P == 2)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + 2 * kTileBytes), "r"(rest[P == 2 ? 4 * e8 : 0]),
                       "r"(rest[P == 2 ? 4 * e8 + 1 : 0]), "r"(rest[P == 2 ? 4 * e8 + 2 : 0]), "r"(rest[P == 2 ? 4 * e8 + 3 : 0])
                       : "memory");
      }
    }
    fence_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(shready);
  }
  mbar_wait_warp(odone, (njb - 1) & 1, ctl, &g_status, kErrWaitMma);
  tc_fence_after();
  if (wg < 2) {
    // lane = query now: each of two warpgroups stores half of the output columns of row `row`, 32 at a time
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    constexpr int kHalf = Rows<W>::kHead / 2;
    const int i = ib * kTileRows + row;
    float rs;
    tmem_ld1(tR + lane_base, &rs);
    tmem_ld_wait1(&rs);
    const float inv = 1.f / (rs + g.eps);
    __syncwarp();                                     // (a division has paths of its own for NaN and the like)
    const int d = W == kSplit ? g.d : Rows<W>::kHead;
    bool nan = false;
#pragma unroll
    for (int c0 = 0; c0 < kHalf; c0 += 32) {
      const int col = kHalf * wg + c0;
      float o[32];
      tmem_ld32(tO + lane_base + col, o);
      tmem_ld_wait(o);
      if (W == kSplit) {                              // share V_hi + share V_lo
        float lo[32];
        tmem_ld32(tO + lane_base + 64 + col, lo);
        tmem_ld_wait(lo);
#pragma unroll
        for (int e = 0; e < 32; ++e) o[e] += lo[e];
      }
      if (i < g.tq) {
        float4* dst = reinterpret_cast<float4*>(out + ((int64_t)n * g.tq + i) * d + col);
#pragma unroll
        for (int c = 0; c < 8; ++c)
          if (W != kSplit || col + 4 * c < d)
            dst[c] = make_float4(o[4 * c] * inv, o[4 * c + 1] * inv, o[4 * c + 2] * inv, o[4 * c + 3] * inv);
      }
      if (P == 2) {
#pragma unroll
        for (int e = 0; e < 32; ++e) nan |= o[e] != o[e];
      }
    }
    if (i < g.tq && wg == 0) ssum[(int64_t)n * g.tq + i] = rs;
    if (P == 2) {
      if (__any_sync(0xffffffffu, nan && rs == rs && i < g.tq))
        restore_infinities(out + ((int64_t)n * g.tq + i) * d, v_rows + (int64_t)n * g.tk * (64 * Rows<W>::kSub) + (W == kSplit ? 64 : 0),
                           64 * Rows<W>::kSub, min(g.tk, (i | 31) + 1), rs == rs ? i : -1, i < g.tq, kHalf * wg,
                           min(d, kHalf * (wg + 1)));
    }
  }
  }
  drain_if_aborted(ctl);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_free(tmem, kTmem);
}

// ---------------------------------------------------------------- pass 4: backward
// Pre-pass, one warp per query row: sinv = 1/(ssum+eps); dbar' = sinv * (dout . out);
// do' = bf16(sinv * dout); zeroes the dq / ghat accumulators.  Folding sinv into dO
// turns  ds = (do.v - dbar) * sinv  into  do'.v - dbar'  and  dv = attn^T do  into
// share^T do', so the main pass never multiplies by sinv per element.
template <typename TD>
__global__ void backward_prep_kernel(const TD* __restrict__ dout, const float* __restrict__ out,
                                     const float* __restrict__ ssum, float eps, int64_t rows,
                                     float* __restrict__ dbarp, __nv_bfloat16* __restrict__ dop,
                                     float* __restrict__ ghat, float* __restrict__ dq_main) {
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  float2 a;
  if (std::is_same<TD, float>::value) {
    a = reinterpret_cast<const float2*>(dout + row * kHeadDim)[lane];
  } else {
    const uint32_t raw = reinterpret_cast<const uint32_t*>(dout + row * kHeadDim)[lane];
    a = make_float2(__uint_as_float(raw << 16), __uint_as_float(raw & 0xffff0000u));
  }
  const float2 b = reinterpret_cast<const float2*>(out + row * kHeadDim)[lane];
  const float sinv = 1.f / (ssum[row] + eps);
  const float dot = warp_sum(a.x * b.x + a.y * b.y);
  reinterpret_cast<uint32_t*>(dop + row * kHeadDim)[lane] = pack_bf16(a.x * sinv, a.y * sinv);
  reinterpret_cast<float2*>(dq_main + row * kHeadDim)[lane] = make_float2(0.f, 0.f);
  if (lane == 0) {
    dbarp[row] = dot * sinv;
    ghat[row] = 0.f;
  }
}

// The factor da / (dp - ghat) of an f(a) / rowsum(f) bid from mass_term and the query's l, f'(a) / (row mass)
// (kernels_bid.py:206-225): zero for a row without mass (l < 0) and, under MASK, for a masked query (f < 0).
template <int BID, bool MASK>
__device__ __forceinline__ float mass_jac(float f, float l, const Geom& g) {
  float d;                                             // f' up to the constant in l
  if (BID == kBidSoftplus) d = 1.f - fast_exp2(-f);    // sigmoid(a) = 1 - e^-softplus(a)
  else if (BID == kBidRelu2) d = f + f;
  else d = f > 0.f ? 1.f : 0.f;
  if (MASK && f < 0.f) d = 0.f;
  // l is (mass_scale / mass), and mass_scale is ln 2 (softplus), scale (relu), scale^2 (relu2: f' = 2 scale^2 s / scale)
  return d * fmaxf(l, 0.f) * (BID == kBidSoftplus ? kLog2e : g.rscale);
}

// One thread's 32 queries of the main reverse pass: vs holds their raw scores against the thread's key, vd
// dO' . v; incle is the key's demand (+ eps) in front of them, R the suffix of dk_share behind them, and query
// e sees the key when e >= first_q and, under END, e < end_q (MASK; all of them do otherwise).  Afterwards shp holds the shares as
// bf16 pairs (SPLIT: their lo plane behind them), vs the Jacobian factor, vd that factor times dp, and R the suffix in front of the
// queries.  Two sweeps.  Forwards: p and 1/(committed+p+eps), the demand
// accumulated from the checkpoint in front exactly as the forward pass did.  Backwards: the
// suffix of dk_share (kernels.py:763-764), accumulated from the last query to the first as
// the reference does — its terms grow towards a key's first bidders, so the other order
// loses the small ones.
//
// PASS: 0 = the Jacobian correction (if any) follows in a pass of its own.  An f(a) / rowsum(f) bid, whose factor is
// unbounded, takes two passes: 1 leaves p and p * dp in vs and vd, the terms of ghat; 2 subtracts ghat (Gh4) from dp
// before the factor multiplies.  These bids keep mass_term of a query between the sweeps (-1 where the query does not
// see the key), which gives p and the factor both.
template <int BID, int SHARE, bool MASK, bool SPLIT, bool END, int PASS = 0>
__device__ __forceinline__ void reverse_sweeps(float (&vs)[32], float (&vd)[32], uint32_t* shp, float& R, float incle,
                                               const float4* Lse4, const float4* Dbar4, const Geom& g,
                                               bool dead, int first_q, int end_q, const float4* Gh4 = nullptr) {
  constexpr bool MASS = row_sum_bid(BID);
  float inv[32];
#pragma unroll
  for (int e4 = 0; e4 < 8; ++e4) {
    const float4 l4 = Lse4[e4];
    const float lse[4] = {l4.x, l4.y, l4.z, l4.w};
    // softmax: z = s*zscale - lse, p = 2^z;  sigmoid: z = lse - s*zscale, p = 1/(1 + 2^z)
    const float zsign = BID == kBidSigmoid ? -g.zscale : g.zscale;
    const float lsign = BID == kBidSigmoid ? 1.f : -1.f;
    const float2 zs = make_float2(zsign, zsign);
    const float2 z01 = fma2(make_float2(vs[e4 * 4], vs[e4 * 4 + 1]), zs, make_float2(lsign * lse[0], lsign * lse[1]));
    const float2 z23 = fma2(make_float2(vs[e4 * 4 + 2], vs[e4 * 4 + 3]), zs, make_float2(lsign * lse[2], lsign * lse[3]));
    const float z[4] = {z01.x, z01.y, z23.x, z23.y};
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = e4 * 4 + u;
      float p, keep;
      if (MASS) {
        keep = u == 3 ? mass_term<BID, true>(vs[e], g.zscale) : mass_term<BID>(vs[e], g.zscale);
        p = mass_bid(mass_power<BID>(keep), lse[u]);
        if (MASK && (dead || first_q > e || (END && e >= end_q))) keep = -1.f;
      } else {
        p = fast_exp2(z[u]);
      }
      if (BID == kBidSigmoid) p = fast_rcp(1.f + p);
      if (MASK) {
        if (dead || first_q > e || (END && e >= end_q)) p = 0.f;
      }
      if (SHARE == kShareInclusive) {
        incle += p;
        inv[e] = fast_rcp(incle);
      } else if (SHARE == kShareExclusive) {     // the demand of earlier queries only
        inv[e] = fast_rcp(incle);
        incle += p;
      } else {
        inv[e] = 1.f;
      }
      vs[e] = MASS ? keep : p;
    }
  }
#pragma unroll
  for (int e4 = 7; e4 >= 0; --e4) {
    const float4 d4 = Dbar4[e4];
    const float dbr[4] = {d4.x, d4.y, d4.z, d4.w};
    float lr[4], gh[4];
    if (MASS) {
      const float4 l4 = Lse4[e4];
      lr[0] = l4.x; lr[1] = l4.y; lr[2] = l4.z; lr[3] = l4.w;
      if (PASS == 2) {
        const float4 g4 = Gh4[e4];
        gh[0] = g4.x; gh[1] = g4.y; gh[2] = g4.z; gh[3] = g4.w;
      }
    }
    // with inv = 1/(committed+p+eps), share = p*inv and w = ds*inv:
    //   ds*(committed+eps)*inv^2 = w*(1-share),  dk_share = -w*share,
    //   dp = w - w*share + (suffix before this query) = w + (suffix after it)
    // (element-wise parts two queries per instruction; the suffix itself is serial).
    // Exclusive share step (inv = 1/(committed+eps)): the direct term is w itself, so
    // dp = w + (suffix BEFORE this query); no share step: dp = ds, no suffix at all.
    // The Jacobian factor is p for the softmax bid and p(1-p) for the sigmoid
    // (kernels_bid.py:196-204, 735-754); vs keeps it for the later suffix fix-up.
#pragma unroll
    for (int h = 1; h >= 0; --h) {
      const int e = e4 * 4 + 2 * h;
      float2 p2 = make_float2(vs[e], vs[e + 1]);
      float2 jac2;
      if (MASS) {
        jac2 = make_float2(mass_jac<BID, MASK>(p2.x, lr[2 * h], g), mass_jac<BID, MASK>(p2.y, lr[2 * h + 1], g));
        p2 = make_float2(mass_bid(mass_power<BID>(p2.x), lr[2 * h]), mass_bid(mass_power<BID>(p2.y), lr[2 * h + 1]));
        if (MASK) {
          if (vs[e] < 0.f) p2.x = 0.f;
          if (vs[e + 1] < 0.f) p2.y = 0.f;
        }
        if (PASS == 1) jac2 = p2;
      }
      const float2 i2 = make_float2(inv[e], inv[e + 1]);
      const float2 w2 = mul2(sub2(make_float2(vd[e], vd[e + 1]), make_float2(dbr[2 * h], dbr[2 * h + 1])), i2);
      const float2 s2 = mul2(p2, i2);
      if (!MASS) jac2 = p2;
      if (BID == kBidSigmoid) jac2 = mul2(p2, sub2(make_float2(1.f, 1.f), p2));
      float2 pd2;
      if (SHARE == kShareInclusive) {
        const float r1 = fmaf(-w2.y, s2.y, R);
        R = fmaf(-w2.x, s2.x, r1);
        pd2 = add2(w2, make_float2(R, r1));
      } else if (SHARE == kShareExclusive) {
        const float r1 = fmaf(-w2.y, s2.y, R);
        pd2 = add2(w2, make_float2(r1, R));
        R = fmaf(-w2.x, s2.x, r1);
      } else {
        pd2 = w2;
      }
      if (PASS == 2) pd2 = sub2(pd2, make_float2(gh[2 * h], gh[2 * h + 1]));
      pd2 = mul2(jac2, pd2);
      vd[e] = pd2.x;
      vd[e + 1] = pd2.y;
      if (BID == kBidSigmoid || MASS) {
        vs[e] = jac2.x;
        vs[e + 1] = jac2.y;
      }
      if (PASS == 1) continue;
      shp[e4 * 2 + h] = pack_bf16(s2.x, s2.y);
      if (SPLIT) shp[16 + e4 * 2 + h] = pack_bf16_rest(s2.x, s2.y, shp[e4 * 2 + h]);
    }
  }
}

// x[l] summed over the warp, in lane l: each of the five steps halves the values that a lane holds (31 shuffles for 32
// sums).  Overwrites x.
__device__ __forceinline__ float sum_over_lanes(float (&x)[32], int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int e = 0; e < o; ++e) {
      const float give = lane & o ? x[e] : x[e + o], mine = lane & o ? x[e + o] : x[e];
      x[e] = mine + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  return x[0];
}

// Main reverse pass (the reference's BA, kernels.py:677-775).  grid = n * ceil(t/128),
// key blocks with the most query blocks first; one CTA per SM, three warpgroups: two of
// compute warps and one whose first warp issues every TMA copy and every MMA and whose
// four warps move the finished dQ tiles out.
// TMEM (496 of 512 columns): two stages of S^T (64 columns each) | two stages of dOV^T
// (64 each) | dV 64 | dK 64 | dQ 64 + ghat 16 as one 80-column tile | the V tile as a
// bf16 A operand (32).
// The CTA keeps K (shared memory) and V (TMEM) of 128 keys and walks the queries from
// last to first in half-steps of 64: S^T = K Q^T and (dO' V^T)^T = V dO'^T are
// [128 keys x 64 queries], lane = key.  Two threads share a key and take 32 queries of a
// half-step each; the key's demand is stored every 32 query rows, so each starts from a
// stored checkpoint.  Each thread sweeps its 32 queries twice:
//   forwards for p and 1/(committed + p + eps), the demand accumulated from the checkpoint
//     exactly as the forward pass did (walking it backwards by subtraction cancels
//     catastrophically once attention is peaked);
//   backwards for the suffix sum of dk_share (kernels.py:763-764), in the reference's order:
//     its terms grow towards a key's first bidders, so a forward prefix would lose the small
//     ones.  Warpgroup 0 (queries 63..32) starts from the suffix behind the half-step;
//     warpgroup 1 (31..0) starts from zero, keeps p and pdp = p * dp in registers, and after
//     one barrier of the compute warps adds p * (the suffix warpgroup 0 ended with): dp is
//     linear in the suffix.
// Per half-step each thread writes 32 shares and 32 pdp values as bf16 pairs over TMEM
// columns it has already read: lane = key is the M index, so they are the A operands of
// dV += share^T dO' and dK += pdp^T Q without passing through shared memory.  pdp also goes
// to shared memory as the MN-major A operand (M = queries) of one N = 80 MMA per 128
// queries against B = [K | ones], which yields dQ = pdp K in 64 columns and ghat = pdp 1
// in the next 16.
// The issuing warp runs two half-steps ahead of the arithmetic: when the tiles of
// half-step h are complete it issues dV, dK (and dQ | ghat after the second half) of h and
// the score MMAs of h + 2 into the stage h has just left, so the tensor pipe works under
// the arithmetic of h + 1.  Q and dO' tiles are triple-buffered.  After setup the third
// warpgroup gives registers up (setmaxnreg) and the compute warpgroups take them.
constexpr int kBwdThreads = 384;
constexpr int kBwdRegs = 168;      // per thread at launch, by the launch bounds; the reverse passes' splits stay within them
static_assert(128 + 2 * 184 <= 3 * kBwdRegs && 104 + 2 * 200 <= 3 * kBwdRegs, "setmaxnreg hands out what the block was launched with");
constexpr int kBwdSmem = 12 * kTileBytes + 2048 + 2048 + 256 + 1024;

// PASS 1 (reverse_sweeps; pass 2 is wide_backward_main_kernel) forms only the scores and adds up ghat, p * dp over the
// 32 keys of a warp by shuffles (31 for 32 queries) and over warps by atomics, all in fp32.  Its do' is
// [hi | lo] as in pass 2, so that ghat is the sum of exactly the dp it will be subtracted from; the lo tiles take the
// shared memory of the pdp and dQ tiles.
template <int BID = kBidSoftmax, int SHARE = kShareInclusive, int PASS = 0>
__global__ void __launch_bounds__(kBwdThreads, 1) backward_main_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
    const __grid_constant__ CUtensorMap map_do, const __grid_constant__ CUtensorMap map_dq, Geom g,
    const __nv_bfloat16* __restrict__ v,
    const float* __restrict__ rmax, const float* __restrict__ rden, const float* __restrict__ dbarp,
    const float* __restrict__ carry, const float* __restrict__ total, float* __restrict__ dq_main,
    float* __restrict__ dk_main, __nv_bfloat16* __restrict__ dv, float* __restrict__ ghat) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  const uint32_t sK = smem_u32(smem);
  // a [128 keys][64] bf16 tile of ones: the second 64-column group of the dQ MMA's B operand
  // (N = 80 = 64 columns of K + 16 of ones), so ghat comes out of the same instruction
  const uint32_t sOnes = sK + kTileBytes;
  uint8_t* ones_ptr = smem + kTileBytes;
  const uint32_t sQ0 = sK + 2 * kTileBytes, sD0 = sK + 5 * kTileBytes;        // [3] each
  const uint32_t sPd = sK + 8 * kTileBytes;                                    // 32 KB
  const uint32_t sDq = sK + 10 * kTileBytes;                                   // 32 KB: fp32 dQ staging
  float* sLse = reinterpret_cast<float*>(smem + 12 * kTileBytes);              // [2][128] log-sum-exp of a step's queries
  float* sDbar = sLse + 256;                                                   // [2][128] their dbar'
  float* sG = reinterpret_cast<float*>(smem + 12 * kTileBytes + 2048);         // [2][2][128] sums of dk_share
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 12 * kTileBytes + 4096);
  Ctl* ctl = reinterpret_cast<Ctl*>(bars + 12);
  static_assert(PASS == 0 || PASS == 1, "pass 2 runs on wide_backward_main_kernel");
  constexpr uint32_t kStageTx = (PASS == 1 ? 3 : 2) * kTileBytes;
  const uint32_t kfull = smem_u32(bars), qfull = smem_u32(bars + 1);           // qfull[3]
  const uint32_t sdone = smem_u32(bars + 4), tiles = smem_u32(bars + 6);       // [2] each
  const uint32_t dqdone = smem_u32(bars + 8);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, wg = tid >> 7, row = tid & 127;
  const int warp_u = uniform_warp();
  const uint32_t lead = elect_one();
  const int nqb = (g.tq + kTileRows - 1) / kTileRows;
  const int ncb = (g.tq + kCarryRows - 1) / kCarryRows;
  const int n = (int)(blockIdx.x % g.n);
  const int jb = (int)(blockIdx.x / g.n);
  const int k0 = jb * kTileRows;
  const int nsteps = nqb - jb;                     // query blocks jb .. nqb-1, visited in reverse
  const int nhalf = 2 * nsteps;
  const int64_t row_base = (int64_t)n * g.tq;
  const int ja = k0 + row;
  const bool dead = ja >= g.tk;

  auto load_stats = [&](int ib) {
    const int i = ib * kTileRows + row;
    float2 st = make_float2(row_sum_bid(BID) ? 0.f : INFINITY, 0.f);
    if (i < g.tq) st = make_float2(load_lse<BID>(rmax, rden, row_base, i, g.tq, g.lshift), dbarp[row_base + i]);
    return st;
  };

  if (tid == 0) {
    ctl->abort = 0;
    for (int i = 0; i < 6; ++i) mbar_init(kfull + 8 * i, 1);      // kfull, qfull[3], sdone[2]
    mbar_init(tiles, 8);
    mbar_init(tiles + 8, 8);
    mbar_init(dqdone, 1);
    fence_barrier_init();
  }
  __syncwarp();
  if (warp == 0) tmem_alloc(smem_u32(&ctl->tmem), 512);
  if (wg == 0) {
    const float2 st = load_stats(nqb - 1);
    sLse[row] = st.x;
    sDbar[row] = st.y;
  }
  else if (wg == 1) {
#pragma unroll
    for (int c = 0; c < 8; ++c)
      reinterpret_cast<uint4*>(ones_ptr)[row * 8 + c] = make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u);
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = uniform(ctl->tmem);
  const uint32_t tS0 = tmem, tDOV0 = tmem + 128, tDV = tmem + 256, tDK = tmem + 320, tDQ = tmem + 384,
                 tG = tmem + 448, tV = tmem + 464;
  const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;

  if (wg == 0) {
    // this key's V row as an A operand: two head-dim elements per 32-bit column
    uint32_t w[32];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      uint4 x = make_uint4(0u, 0u, 0u, 0u);
      if (!dead) x = reinterpret_cast<const uint4*>(v + ((int64_t)n * g.tk + ja) * kHeadDim)[c];
      w[4 * c] = x.x; w[4 * c + 1] = x.y; w[4 * c + 2] = x.z; w[4 * c + 3] = x.w;
    }
    tmem_st16(tV + lane_base, w);
    tmem_st16(tV + lane_base + 16, w + 16);
  }
  if (wg < 2) {
    // dV and dK start from zero, so that every MMA into them accumulates
    uint32_t z[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) z[c] = 0u;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      tmem_st16(tDV + lane_base + 32 * wg + 16 * c, z);
      tmem_st16(tDK + lane_base + 32 * wg + 16 * c, z);
    }
    tmem_st_wait();
  }
  if (tid == 256) {
    mbar_expect_tx(kfull, kTileBytes);
    tma_load_tile(sK, &map_k, k0, n, kfull);
    for (int s = 0; s < 3 && s < nsteps; ++s) {
      mbar_expect_tx(qfull + 8 * s, kStageTx);
      tma_load_tile(sQ0 + kTileBytes * s, &map_q, (nqb - 1 - s) * kTileRows, n, qfull + 8 * s);
      tma_load_tile(sD0 + kTileBytes * s, &map_do, (nqb - 1 - s) * kTileRows, n, qfull + 8 * s);
      if (PASS == 1) tma_load_tile(sPd + kTileBytes * s, &map_do, (nqb - 1 - s) * kTileRows, n, qfull + 8 * s, 64);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  if (wg == 2) {
    // ------------------------------------------------------------ warpgroup 2: issue and dQ read-out
    // Warp 8 issues every MMA and TMA copy.  After the second half-step of a step all
    // four warps (lane = query) move the finished dQ | ghat tile out, so that the compute
    // warps never touch it.  The warpgroup hands most of its registers to the other two.
    asm volatile("setmaxnreg.dec.sync.aligned.u32 128;");
    constexpr uint32_t id_s = instr_desc(128, 64, 0, 0);     // scores: both operands K-major
    constexpr uint32_t id_kd = instr_desc(128, 64, 0, 1);    // dV, dK: A from TMEM (M = keys), B MN-major
    constexpr uint32_t id_qd = instr_desc(128, 80, 1, 1);    // dQ | ghat: A MN-major (M = queries)
    // every descriptor is built once; inside the loop tile, stage and k-step are constant
    // offsets (in 16-byte units: a tile is 1024, an MN-major k-step 128, a K-major one 2)
    const Desc dKk = make_desc(sK, 16, 1024);                 // K, K-major: A of the scores
    const Desc dKm = make_desc(sK, sOnes - sK, 1024);         // [K | ones], MN-major: B of dQ | ghat
    const Desc dPm = make_desc(sPd, kTileBytes, 1024);        // pdp, MN-major: A of dQ | ghat
    const Desc dQk = make_desc(sQ0, 16, 1024), dQm = make_desc(sQ0, kTileBytes, 1024);
    const Desc dDk = make_desc(sD0, 16, 1024), dDm = make_desc(sD0, kTileBytes, 1024);
    // scores of a half-step in stage ST of Q and dO'; even half-steps take queries 64..127
    auto issue_scores = [&](auto odd_c, auto st_c) {
      constexpr int ODD = decltype(odd_c)::value, ST = decltype(st_c)::value;
      constexpr uint32_t off = ST * 1024 + (ODD ? 0 : 512);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) mma_ss(lead, tS0 + 64 * ODD, dKk, 2 * kk, dQk, off + 2 * kk, id_s, kk > 0);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) mma_ts(lead, tDOV0 + 64 * ODD, tV + 8 * kk, dDk, off + 2 * kk, id_s, kk > 0);
#pragma unroll
      for (int kk = 0; PASS == 1 && kk < 4; ++kk)            // + V (lo part of do')^T
        mma_ts(lead, tDOV0 + 64 * ODD, tV + 8 * kk, make_desc(sPd, 16, 1024), off + 2 * kk, id_s, 1);
    };
    if (warp_u == 8) {
      mbar_wait_warp(kfull, 0, ctl, &g_status, kErrWaitTma);
      mbar_wait_warp(qfull, 0, ctl, &g_status, kErrWaitTma);
      tc_fence_after();
      issue_scores(std::integral_constant<int, 0>{}, std::integral_constant<int, 0>{});
      mma_commit(lead, sdone);
      issue_scores(std::integral_constant<int, 1>{}, std::integral_constant<int, 0>{});
      mma_commit(lead, sdone + 8);
    }
    __syncwarp();
    // half-step h = 2s + ODD of step s, whose Q and dO' tiles sit in stage ST = s % 3
    auto half = [&](auto odd_c, auto st_c, int s) {
      constexpr int ODD = decltype(odd_c)::value, ST = decltype(st_c)::value;
      constexpr int ST1 = (ST + 1) % 3, ST2 = (ST + 2) % 3;
      if (warp_u == 8) {
        mbar_wait_warp(tiles + 8 * ODD, s & 1, ctl, &g_status, kErrWaitTile);
        tc_fence_after();
#pragma unroll
        for (int kq = 0; PASS != 1 && kq < 4; ++kq) {       // contraction over the 64 queries
          // queries [16kq, 16kq+16) of the half-step: 8 columns at the start of the owning
          // warpgroup's 32-column range (warpgroup 1 owns queries 0..31)
          constexpr uint32_t base = ST * 1024 + (ODD ? 0 : 4) * 128;
          const uint32_t col = 64 * ODD + 32 * (kq >> 1) + 8 * (kq & 1);
          mma_ts(lead, tDV, tS0 + col, dDm, base + 128 * kq, id_kd, 1);
          mma_ts(lead, tDK, tDOV0 + col, dQm, base + 128 * kq, id_kd, 1);
        }
        if (ODD && PASS != 1) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)                    // contraction over the 128 keys
            mma_ss(lead, tDQ, dPm, 128 * kk, dKm, 128 * kk, id_qd, kk > 0);
          mma_commit(lead, dqdone);
        }
        if (s + 1 < nsteps) {                               // half-step h + 2 belongs to step s + 1
          if (!ODD) {
            mbar_wait_warp(qfull + 8 * ST1, ((s + 1) / 3) & 1, ctl, &g_status, kErrWaitTma);
            tc_fence_after();
          }
          issue_scores(odd_c, std::integral_constant<int, ST1>{});
        }
        mma_commit(lead, sdone + 8 * ODD);
        if (!ODD && s >= 1 && s + 2 < nsteps) {
          // every MMA of step s-1 has completed once the commit of its second half-step has:
          // its Q and dO' stage takes step s+2
          mbar_wait_warp(sdone + 8, s & 1, ctl, &g_status, kErrWaitMma);
          if (lead) {
            mbar_expect_tx(qfull + 8 * ST2, kStageTx);
            tma_load_tile(sQ0 + kTileBytes * ST2, &map_q, (nqb - 3 - s) * kTileRows, n, qfull + 8 * ST2);
            tma_load_tile(sD0 + kTileBytes * ST2, &map_do, (nqb - 3 - s) * kTileRows, n, qfull + 8 * ST2);
            if (PASS == 1) tma_load_tile(sPd + kTileBytes * ST2, &map_do, (nqb - 3 - s) * kTileRows, n, qfull + 8 * ST2, 64);
          }
        }
      }
      __syncwarp();
      if (ODD && PASS != 1) {
        // dQ and ghat of the step's 128 queries: lane = query.  The fp32 tile is staged in
        // shared memory in the copy engine's swizzled layout and added to dq_main by two
        // tensor reductions of 32 columns.
        if (lane == 0) mbar_wait(dqdone, s & 1, ctl, &g_status, kErrWaitMma);
        __syncwarp();
        tc_fence_after();
        if (tid == 256) tma_wait_read_all();            // the previous reductions have read the staging buffer
        asm volatile("bar.sync 2, 128;" ::: "memory");
        const uint32_t stage = sDq + row * 128;
#pragma unroll 1
        for (int j = 0; j < 4; ++j) {                   // 16 columns at a time
          float dq[16];
          tmem_ld16(tDQ + lane_base + 16 * j, dq);
          tmem_ld_wait16(dq);
#pragma unroll
          for (int c = 0; c < 4; ++c)
            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(stage + kTileBytes * (j >> 1) + (((4 * (j & 1) + c) ^ (row & 7)) << 4)),
                         "f"(dq[4 * c] * g.scale), "f"(dq[4 * c + 1] * g.scale), "f"(dq[4 * c + 2] * g.scale),
                         "f"(dq[4 * c + 3] * g.scale)
                         : "memory");
        }
        float gh;
        tmem_ld1(tG + lane_base, &gh);
        tmem_ld_wait1(&gh);
        fence_async_smem();
        tc_fence_before();
        asm volatile("bar.sync 2, 128;" ::: "memory");
        const int ibq = nqb - 1 - s;
        if (tid == 256) {
          tc_fence_after();
          tma_reduce_add_tile(&map_dq, sDq, 0, ibq * kTileRows, n);
          tma_reduce_add_tile(&map_dq, sDq + kTileBytes, 32, ibq * kTileRows, n);
        }
        const int i = ibq * kTileRows + row;
        if (PASS == 0 && i < g.tq) atomicAdd(ghat + row_base + i, gh);
      }
    };
    using C0 = std::integral_constant<int, 0>;
    using C1 = std::integral_constant<int, 1>;
    using C2 = std::integral_constant<int, 2>;
    for (int s = 0; s < nsteps; s += 3) {
      half(C0{}, C0{}, s);
      half(C1{}, C0{}, s);
      if (s + 1 < nsteps) {
        half(C0{}, C1{}, s + 1);
        half(C1{}, C1{}, s + 1);
      }
      if (s + 2 < nsteps) {
        half(C0{}, C2{}, s + 2);
        half(C1{}, C2{}, s + 2);
      }
    }
    if (tid == 256) tma_wait_read_all();
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 184;");
    // ------------------------------------------------------------ the compute warps
    const int cw = 32 * (1 - wg);                    // this warpgroup's columns of a stage
    // demand of this thread's key in front of its 32 queries of half-step h (exclusive of the
    // first): the stored checkpoint of that 32-row block (past the end: any value, p is 0 there)
    auto load_edge = [&](int h) {
      if (dead || SHARE == kShareNone) return 0.f;         // no share step: no demand is read
      const int rb = 4 * (nqb - 1 - (h >> 1)) + ((h & 1) ? 0 : 2) + (wg == 0 ? 1 : 0);
      return rb < ncb ? carry[((int64_t)n * ncb + rb) * g.tk + ja] : total[(int64_t)n * g.tk + ja];
    };
    float sigma = 0.f;                               // suffix of dk_share behind the half-step
    // the checkpoints are read once from a buffer far larger than L2: each load is issued two
    // half-steps before its value is used
    float incl = load_edge(0);
    float incl_next = nhalf > 1 ? load_edge(1) : 0.f;
    for (int h = 0; h < nhalf; ++h) {
      const int s = h >> 1, odd = h & 1, ib = nqb - 1 - s, b = s & 1;
      // fetch what the coming half-steps need before waiting for this one
      float incl_next2 = 0.f;
      float st_max = INFINITY, st_den = 1.f, st_dbar = 0.f;
      if (h + 2 < nhalf) incl_next2 = load_edge(h + 2);
      const bool fetch_stats = !odd && wg == 0 && s + 1 < nsteps;
      if (fetch_stats) {
        const int i = (ib - 1) * kTileRows + row;     // ib >= 1 here, so i < tq
        if (row_sum_bid(BID)) {
          st_den = rden[row_base + i];
        } else if (BID == kBidSoftmax && rmax != nullptr) {
          st_max = rmax[row_base + i];
          st_den = rden[row_base + i];
        } else {
          st_max = g.lshift;                          // no row statistics: lse = log2(shift) + log2(1)
        }
        st_dbar = dbarp[row_base + i];
      }
      mbar_wait_warp(sdone + 8 * odd, s & 1, ctl, &g_status, kErrWaitMma);
      tc_fence_after();
      float vs[32], vd[32];
      const uint32_t tcol = lane_base + 64 * odd + cw;
      tmem_ld32(tS0 + tcol, vs);
      tmem_ld32(tDOV0 + tcol, vd);
      tmem_ld_wait(vs);
      tmem_ld_wait(vd);
      const int qc = (odd ? 0 : 64) + cw;             // first query column of this thread in the step's tile
      const int iq0 = ib * kTileRows + qc;            // its position (q_off == 0 here)
      const bool masked_tile = dead || (ib * kTileRows + (odd ? 0 : 64) < k0 + kTileRows - 1) ||
                               (kMaskEnd<kNarrow, BID> && iq0 + 32 > g.tq);
      const float4* Lse4 = reinterpret_cast<const float4*>(sLse + b * 128 + qc);
      const float4* Dbar4 = reinterpret_cast<const float4*>(sDbar + b * 128 + qc);
      uint32_t shp[16];                                // 32 shares as bf16 pairs
      // warpgroup 0 (queries 32..63) knows the suffix of dk_share behind its queries; warpgroup 1
      // starts from zero and adds p * (the suffix warpgroup 0 ends with) afterwards: dp is linear in it
      float R = wg == 0 ? sigma : 0.f;
      auto chunk = [&](auto mask_tag) {
        reverse_sweeps<BID, SHARE, decltype(mask_tag)::value, false, kMaskEnd<kNarrow, BID>, PASS>(
            vs, vd, shp, R, incl + g.eps, Lse4, Dbar4, g, dead, ja - iq0, g.tq - iq0);
      };
      if (masked_tile) chunk(std::true_type{}); else chunk(std::false_type{});
      // warpgroup 0: the suffix behind query 32; warpgroup 1: minus its own sum of -dk_share
      sG[(odd * 2 + wg) * 128 + row] = R;
      // the shares stay in TMEM, over score columns this thread has consumed
      if (PASS != 1) tmem_st16(tS0 + tcol, shp);
      asm volatile("bar.sync 1, 256;" ::: "memory");   // the compute warps
      const float rother = sG[(odd * 2 + (1 - wg)) * 128 + row];
      const float fix = wg == 1 ? rother : 0.f;
      sigma = R + rother;                              // the suffix behind the next half-step
      if (PASS == 1) {
        // p * dp summed over the warp's 32 keys
#pragma unroll
        for (int e = 0; e < 32; ++e) vd[e] = fmaf(vs[e], fix, vd[e]);
        const float sum = sum_over_lanes(vd, lane);
        if (iq0 + lane < g.tq) atomicAdd(ghat + row_base + iq0 + lane, sum);
      } else {
        // the dQ MMAs of the previous 128 queries read the pdp buffer that is written next
        if (!odd && s >= 1) mbar_wait_warp(dqdone, (s - 1) & 1, ctl, &g_status, kErrWaitMma);
        uint32_t pdt[16];                              // 32 pdp values as bf16 pairs
#pragma unroll
        for (int e8 = 0; e8 < 4; ++e8) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int e = e8 * 8 + 2 * u;
            const float2 f2 = fma2(make_float2(vs[e], vs[e + 1]), make_float2(fix, fix), make_float2(vd[e], vd[e + 1]));
            pdt[e8 * 4 + u] = pack_bf16(f2.x, f2.y);
          }
          // shared memory: the MN-major A operand of dQ | ghat (M = queries)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sPd + share_chunk_offset(row, qc + e8 * 8)),
                       "r"(pdt[e8 * 4]), "r"(pdt[e8 * 4 + 1]), "r"(pdt[e8 * 4 + 2]), "r"(pdt[e8 * 4 + 3])
                       : "memory");
        }
        // TMEM, over consumed dOV^T columns: the A operand of dK (M = keys)
        tmem_st16(tDOV0 + tcol, pdt);
      }
      if (fetch_stats) {
        sLse[(b ^ 1) * 128 + row] = row_sum_bid(BID) ? mass_factor(st_den, (ib - 1) * kTileRows + row, g.lshift)
                                                     : st_max + log2f(st_den);
        sDbar[(b ^ 1) * 128 + row] = st_dbar;
      }
      incl = incl_next;
      incl_next = incl_next2;
      tmem_st_wait();
      fence_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tiles + 8 * odd);
    }
  }
  mbar_wait_warp(sdone + 8, nsteps & 1, ctl, &g_status, kErrWaitMma);
  tc_fence_after();
  if (PASS != 1 && warp < 8) {
    // lane = key: each warpgroup stores 32 of the 64 columns of dk_main and dv
    float a[32];
    const int64_t o = ((int64_t)n * g.tk + ja) * kHeadDim + 32 * wg;
    tmem_ld32(tDK + lane_base + 32 * wg, a);
    tmem_ld_wait(a);
    if (!dead) {
#pragma unroll
      for (int e = 0; e < 32; e += 4)
        *reinterpret_cast<float4*>(dk_main + o + e) =
            make_float4(a[e] * g.scale, a[e + 1] * g.scale, a[e + 2] * g.scale, a[e + 3] * g.scale);
    }
    tmem_ld32(tDV + lane_base + 32 * wg, a);
    tmem_ld_wait(a);
    if (!dead) {
#pragma unroll
      for (int e = 0; e < 32; e += 8)
        *reinterpret_cast<uint4*>(dv + o + e) =
            make_uint4(pack_bf16(a[e], a[e + 1]), pack_bf16(a[e + 2], a[e + 3]),
                       pack_bf16(a[e + 4], a[e + 5]), pack_bf16(a[e + 6], a[e + 7]));
    }
  }
  drain_if_aborted(ctl);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_free(tmem, 512);
}

// The forward half of reverse_sweeps for a thread's 32 queries and the sigmoid's bid: scores become bids in vs, and inv takes
// 1/(committed + p + eps) (the exclusive share step: 1/(committed + eps)).  incle is the key's demand (+ eps) in front of the queries.
template <int SHARE, bool MASK>
__device__ __forceinline__ void bids_and_inverses(float (&vs)[32], float (&inv)[32], float incle, const Geom& g, bool dead, int first_q) {
  const float2 zs = make_float2(-g.zscale, -g.zscale), lse = make_float2(g.lshift, g.lshift);
#pragma unroll
  for (int e = 0; e < 32; e += 2) {
    const float2 z2 = fma2(make_float2(vs[e], vs[e + 1]), zs, lse);
    const float z[2] = {z2.x, z2.y};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      float p = fast_rcp(1.f + fast_exp2(z[u]));
      if (MASK && (dead || first_q > e + u)) p = 0.f;
      if (SHARE == kShareInclusive) incle += p;
      inv[e + u] = fast_rcp(incle);
      if (SHARE == kShareExclusive) incle += p;
      vs[e + u] = p;
    }
  }
}

// The backward half for 8 of them, last to first: vd holds their dO' . v, R the suffix of dk_share behind them and, afterwards, in
// front of them.  shp takes their shares as bf16 pairs, p the Jacobian factor, inv that factor times dp.  The formulas stand in
// reverse_sweeps.
template <int SHARE>
__device__ __forceinline__ void suffix_of_eight(float* p, float* inv, const float* vd, const float4* Dbar4, float& R, uint32_t* shp) {
#pragma unroll
  for (int c = 1; c >= 0; --c) {
    const float4 d4 = Dbar4[c];
    const float dbr[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
    for (int h = 1; h >= 0; --h) {
      const int e = 4 * c + 2 * h;
      const float2 p2 = make_float2(p[e], p[e + 1]), i2 = make_float2(inv[e], inv[e + 1]);
      const float2 w2 = mul2(sub2(make_float2(vd[e], vd[e + 1]), make_float2(dbr[2 * h], dbr[2 * h + 1])), i2), s2 = mul2(p2, i2);
      const float r1 = fmaf(-w2.y, s2.y, R), r0 = fmaf(-w2.x, s2.x, r1);
      const float2 jac2 = mul2(p2, sub2(make_float2(1.f, 1.f), p2));
      const float2 pd2 = mul2(jac2, add2(w2, SHARE == kShareInclusive ? make_float2(r0, r1) : make_float2(r1, R)));
      R = r0;
      shp[2 * c + h] = pack_bf16(s2.x, s2.y);
      p[e] = jac2.x;
      p[e + 1] = jac2.y;
      inv[e] = pd2.x;
      inv[e + 1] = pd2.y;
    }
  }
}

// Main reverse pass (the reference's BA, kernels.py:677-775) of the sigmoid's bid with a share step.
// grid = n * ceil(t/128), key blocks with the most queries first; one CTA per SM, five warpgroups: four of compute warps, and one
// whose last warp issues every TMA copy and MMA while its first two move the finished dQ tiles out.
//
// The CTA keeps K and V of 128 keys (both as TMEM operands) and walks the queries from last to first in slices of 32, which the
// compute warpgroups take in turn, one thread per key.  The demand of a key is stored every 32 query rows, so every slice starts
// from a stored checkpoint; what a slice needs of the one behind it is the key's suffix of dk_share, one float per key, which is
// handed from warp to warp (the four warps of a scheduler hold the same 32 keys): nothing in the loop waits for the whole CTA.  Per
// slice:
//   S^T, (dO' V^T)^T   [128 keys x 32 queries] each: 4 + 4 MMAs of N = 32, A = K, V in TMEM
//   forwards           p and 1/(committed + p + eps), the demand accumulated from the checkpoint exactly as the forward pass did
//   backwards          the suffix of dk_share from the slice's end in the reference's order (kernels.py:763-764); the suffix behind
//                      the slice is added afterwards, dp being linear in it
//   dV, dK             += share^T dO', pdp^T Q: shares and pdp go back into TMEM as bf16 pairs over the scores that were read, where
//                      they are A operands (M = keys): 2 + 2 MMAs
// and per 64 queries dQ^T = [K | 0]^T pdp, M = 64 features (and 64 rows of zeros), from the pdp that every thread also writes to
// shared memory: 8 MMAs of N = 64 into one tile of 64 columns, moved out by TMA tensor reductions as in the fused forward.
// TMEM: [S^T 32 | dOV^T 32] per warpgroup, dV 64, dK 64, V 32, K 32, dQ^T 64 = 512 columns.
//
// Against backward_main_kernel, whose eight compute warps go through a half-step together: whole backward, n = 32, T = 8192
// 1673 -> 1437 us, n = 8, T = 4096 127 -> 107, n = 64, T = 2048 294 -> 271, n = 16, T = 1777 69.9 -> 65.7, but n = 384, T = 1024
// 604 -> 609 and n = 256, T = 512 163 -> 168, where a block's start and end weigh more.  The three special-function operations of a
// sigmoid score leave the card below its power limit; the softmax bid's passes of long rows run at it (1.72 GHz), and there this
// form, which executes more instructions, gained nothing (14.5 / 14.6 ms at n = 64, T = 16384; n = 384, T = 1024 672 / 705 us).
constexpr int kSliceRegs = 96;          // per thread at launch, by the launch bounds
static_assert(4 * 104 + 64 <= 5 * kSliceRegs, "setmaxnreg hands out what the block was launched with");
constexpr int kSliceThreads = 640;
constexpr int kSliceRing = 6;                                     // half tiles (64 queries) of q and of do'
constexpr int kSliceFrom = 1536;                                  // tokens of a row from which it is the faster one
// K zeros | Q[6] dO'[6] (8 KB each) | pdp[2] | staging[2] (16 KB each) | dbar [4][64] | suffixes [4][128] | barriers
constexpr int kSliceSmem = (2 + kSliceRing + 2 + 2) * kTileBytes + 1024 + 2048 + 512 + 1024;

template <int SHARE>
__global__ void __launch_bounds__(kSliceThreads, 1) backward_slices_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
    const __grid_constant__ CUtensorMap map_do, const __grid_constant__ CUtensorMap map_dq, Geom g,
    const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ v,
    const float* __restrict__ dbarp, const float* __restrict__ carry, const float* __restrict__ total, float* __restrict__ dk_main,
    __nv_bfloat16* __restrict__ dv) {
  constexpr int R = kSliceRing;
  constexpr uint32_t HB = kTileBytes / 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  const uint32_t sK = smem_u32(smem), sZero = sK + kTileBytes;               // A of dQ^T: [K | 0], MN-major
  const uint32_t sQ = sZero + kTileBytes, sD = sQ + R * HB, sPd = sD + R * HB;
  const uint32_t sStage = sPd + 2 * kTileBytes;                              // [2][2 warps][64 queries][32 features] fp32
  float* sDbar = reinterpret_cast<float*>(smem + (sStage - sK) + 2 * kTileBytes);   // [4][64] dbar' of a half tile's queries
  float* sG = sDbar + 256;                                                   // [4][128] suffix in front of a warpgroup's slice
  uint64_t* bars = reinterpret_cast<uint64_t*>(sG + 512);
  const uint32_t kfull = smem_u32(bars), fin = kfull + 8, qfull = fin + 8, sdone = qfull + 8 * R, dqdone = sdone + 32,
                 tiles = dqdone + 16, dqfree = tiles + 32, chain = dqfree + 8;            // 1, 1, [R], [4], [2], [4], 1, [4][4]
  Ctl* ctl = reinterpret_cast<Ctl*>(bars + 13 + R + 16);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, wg = tid >> 7, row = tid & 127;
  const int warp_u = uniform_warp();
  const uint32_t lead = elect_one();
  const int ncb = (g.tq + kCarryRows - 1) / kCarryRows;
  const int n = (int)(blockIdx.x % g.n);
  const int k0 = (int)(blockIdx.x / g.n) * kTileRows;
  const int hl = (g.tq + 63) / 64 - 1, nh = hl - k0 / 64 + 1;   // half tiles hl .. k0 / 64 of queries: the u-th one is hl - u
  const int64_t row_base = (int64_t)n * g.tq;
  const int ja = k0 + row;
  const bool dead = ja >= g.tk;

  if (tid == 0) {
    ctl->abort = 0;
    for (int i = 0; i < 8 + R; ++i) mbar_init(kfull + 8 * i, 1);            // kfull, fin, qfull[R], sdone[4], dqdone[2]
    for (int i = 0; i < 4; ++i) mbar_init(tiles + 8 * i, 4);
    mbar_init(dqfree, 3);
    for (int i = 0; i < 16; ++i) mbar_init(chain + 8 * i, 1);
    fence_barrier_init();
  }
  __syncwarp();
  if (warp == 0) tmem_alloc(smem_u32(&ctl->tmem), 512);
  if (tid < 256) {
    // of the first four half tiles (a negative row belongs to no half tile of this block)
    const int i = (hl - (tid >> 6)) * 64 + (tid & 63);
    sDbar[tid] = i >= 0 && i < g.tq ? dbarp[row_base + i] : 0.f;
  } else if (wg == 2) {
#pragma unroll
    for (int c = 0; c < 8; ++c) reinterpret_cast<uint4*>(smem + kTileBytes)[row * 8 + c] = make_uint4(0u, 0u, 0u, 0u);
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = uniform(ctl->tmem);
  const uint32_t tS = tmem, tDV = tmem + 256, tDK = tmem + 320, tV = tmem + 384, tK = tmem + 416, tQ = tmem + 448;
  const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;

  if (wg < 2) {
    // this key's row as an A operand: two head-dim elements per 32-bit column
    uint32_t w[32];
    const __nv_bfloat16* src = (wg == 0 ? v : k) + ((int64_t)n * g.tk + ja) * kHeadDim;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      uint4 x = make_uint4(0u, 0u, 0u, 0u);
      if (!dead) x = reinterpret_cast<const uint4*>(src)[c];
      w[4 * c] = x.x; w[4 * c + 1] = x.y; w[4 * c + 2] = x.z; w[4 * c + 3] = x.w;
    }
    __syncwarp();
    tmem_st16(tV + 32 * wg + lane_base, w);
    tmem_st16(tV + 32 * wg + lane_base + 16, w + 16);
    tmem_st_wait();
  } else if (wg < 4) {
    // dV and dK start from zero, so that every MMA into them accumulates
    uint32_t z[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) z[c] = 0u;
#pragma unroll
    for (int c = 0; c < 4; ++c) tmem_st16(tDV + 64 * (wg - 2) + lane_base + 16 * c, z);
    tmem_st_wait();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  if (wg == 4) {
    // ------------------------------------------------------------ issue (its last warp), and the dQ read-out
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    if (warp_u == 19) {
      constexpr uint32_t id_s = instr_desc(128, 32, 0, 0);     // scores: A from TMEM, B K-major
      constexpr uint32_t id_kd = instr_desc(128, 64, 0, 1);    // dV, dK: A from TMEM (M = keys), B MN-major
      constexpr uint32_t id_q = instr_desc(128, 64, 1, 1);     // dQ^T: A and B MN-major
      const Desc dKm = make_desc(sK, sZero - sK, 1024), dPd = make_desc(sPd, kTileBytes, 1024);
      const Desc dQk = make_desc(sQ, 16, 1024), dQm = make_desc(sQ, kTileBytes, 1024);
      const Desc dDk = make_desc(sD, 16, 1024), dDm = make_desc(sD, kTileBytes, 1024);
      auto load_rows = [&](int u) {
        const int st = u % R;
        if (!lead) return;
        mbar_expect_tx(qfull + 8 * st, 2 * HB);
        tma_load_tile(sQ + HB * st, &map_q, (hl - u) * 64, n, qfull + 8 * st);
        tma_load_tile(sD + HB * st, &map_do, (hl - u) * 64, n, qfull + 8 * st);
      };
      // Place in the ring and warpgroup are compile-time (half tile u is the J-th of a round of the ring), so that an MMA's
      // operands are constants away from uniform registers.
      // scores of slice ODD of a half tile: queries 32..63 for ODD = 0, 0..31 for 1
      auto issue_scores = [&](auto j_c, auto odd_c) {
        constexpr int J = decltype(j_c)::value, ODD = decltype(odd_c)::value, W = (2 * J + ODD) & 3;
        constexpr uint32_t off = (HB >> 4) * J + (ODD ? 0 : 256);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) mma_ts(lead, tS + 64 * W, tK + 8 * kk, dQk, off + 2 * kk, id_s, kk > 0);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) mma_ts(lead, tS + 64 * W + 32, tV + 8 * kk, dDk, off + 2 * kk, id_s, kk > 0);
        mma_commit(lead, sdone + 8 * W);
      };
      using C0 = std::integral_constant<int, 0>;
      using C1 = std::integral_constant<int, 1>;
      if (lead) {
        mbar_expect_tx(kfull, kTileBytes);
        tma_load_tile(sK, &map_k, k0, n, kfull);
      }
      for (int u = 0; u < R && u < nh; ++u) load_rows(u);
      mbar_wait_warp(qfull, 0, ctl, &g_status, kErrWaitTma);
      tc_fence_after();
      issue_scores(C0{}, C0{});
      issue_scores(C0{}, C1{});
      if (nh > 1) {
        mbar_wait_warp(qfull + 8, 0, ctl, &g_status, kErrWaitTma);
        tc_fence_after();
        issue_scores(C1{}, C0{});
        issue_scores(C1{}, C1{});
      }
      mbar_wait_warp(kfull, 0, ctl, &g_status, kErrWaitTma);
      auto half = [&](auto j_c, int u) {
        constexpr int J = decltype(j_c)::value, J2 = (J + 2) % R;
        auto slice = [&](auto odd_c) {
          constexpr int ODD = decltype(odd_c)::value, W = (2 * J + ODD) & 3;
          constexpr uint32_t off = (HB >> 4) * J + (ODD ? 0 : 256);
          mbar_wait_warp(tiles + 8 * W, (u >> 1) & 1, ctl, &g_status, kErrWaitTile);
          tc_fence_after();
#pragma unroll
          for (int kk = 0; kk < 2; ++kk) {                     // contraction over the 32 queries
            mma_ts(lead, tDV, tS + 64 * W + 8 * kk, dDm, off + 128 * kk, id_kd, 1);
            mma_ts(lead, tDK, tS + 64 * W + 32 + 8 * kk, dQm, off + 128 * kk, id_kd, 1);
          }
          if (u + 2 < nh) {
            if (!ODD) {
              mbar_wait_warp(qfull + 8 * J2, ((u + 2) / R) & 1, ctl, &g_status, kErrWaitTma);
              tc_fence_after();
            }
            issue_scores(std::integral_constant<int, J2>{}, odd_c);
          }
        };
        slice(C0{});
        slice(C1{});
        // both slices of the half tile exist.  Once dQ^T of the one before is out, its queries' places in the ring are free, and
        // dbar' of half tile u + 3 is in its place (its scores are issued in the turn for u + 1)
        if (u >= 1) {
          mbar_wait_warp(dqfree, (u - 1) & 1, ctl, &g_status, kErrWaitDrain);
          tc_fence_after();
          if (u - 1 + R < nh) load_rows(u - 1 + R);
        }
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)                         // contraction over the 128 keys
          mma_ss(lead, tQ, dKm, 128 * kk, dPd, (kTileBytes >> 4) * (J & 1) + 128 * kk, id_q, kk > 0);
        mma_commit(lead, dqdone + 8 * (J & 1));
      };
      static_assert(R == 6, "a round of the ring is six half tiles, an even number");
      for (int u = 0; u < nh; u += R) {
        half(C0{}, u);
        if (u + 1 < nh) half(C1{}, u + 1);
        if (u + 2 < nh) half(std::integral_constant<int, 2>{}, u + 2);
        if (u + 3 < nh) half(std::integral_constant<int, 3>{}, u + 3);
        if (u + 4 < nh) half(std::integral_constant<int, 4>{}, u + 4);
        if (u + 5 < nh) half(std::integral_constant<int, 5>{}, u + 5);
      }
      mma_commit(lead, fin);
      __syncwarp();
    } else {
      // dQ^T of half tile u to global memory by two warps, lane = feature (staging is doubled: a tile does not wait for the copy
      // engine to have read the one before).  The third keeps dbar': that of half tile u + 4 takes the place of half tile u, whose
      // last use lies in front of dqdone; the issuing warp waits for the release of u at the end of its turn for u + 1, in front of the
      // scores of u + 4.
      if (warp_u == 18) {
        float next[2] = {0.f, 0.f};
        auto fetch = [&](int u) {                              // (every row of an earlier half tile exists)
          next[0] = dbarp[row_base + (hl - u) * 64 + lane];
          next[1] = dbarp[row_base + (hl - u) * 64 + 32 + lane];
        };
        if (4 < nh) fetch(4);
        for (int u = 0; u < nh; ++u) {
          if (lane == 0) mbar_wait(dqdone + 8 * (u & 1), (u >> 1) & 1, ctl, &g_status, kErrWaitMma);
          __syncwarp();
          if (u + 4 < nh) {
            sDbar[64 * (u & 3) + lane] = next[0];
            sDbar[64 * (u & 3) + 32 + lane] = next[1];
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(dqfree);
          if (u + 5 < nh) fetch(u + 5);
        }
      } else {
        const uint32_t tile = tQ + lane_base;
        for (int u = 0; u < nh; ++u) {
          const uint32_t stage = sStage + kTileBytes * (u & 1) + HB * (warp & 1);
          if (lane == 0) mbar_wait(dqdone + 8 * (u & 1), (u >> 1) & 1, ctl, &g_status, kErrWaitMma);
          if (lane == 0) tma_wait_read_all_but_one();          // the last reduction but one has read this staging
          __syncwarp();
          tc_fence_after();
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            float o[32];
            tmem_ld32(tile + 32 * c, o);
            tmem_ld_wait(o);
            if (c == 1) {
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(dqfree);              // this warp has read the tile
            }
#pragma unroll
            for (int e = 0; e < 32; ++e)
              asm volatile("st.shared.f32 [%0], %1;" ::"r"(stage + lane * 4 + (32 * c + e) * 128), "f"(o[e] * g.scale) : "memory");
          }
          fence_async_smem();
          __syncwarp();
          if (lane == 0) tma_reduce_add_tile(&map_dq, stage, 32 * (warp & 1), (hl - u) * 64, n);
        }
      }
      if (lane == 0) tma_wait_read_all();
      __syncwarp();
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    // ------------------------------------------------------------ the compute warps: lane = key
    const uint32_t tSw = tS + 64 * wg + lane_base, tDw = tSw + 32;
    const uint32_t mine = chain + 8 * (4 * wg + (warp & 3)), behind = chain + 8 * (4 * ((wg + 3) & 3) + (warp & 3));
    const float* sBehind = sG + 128 * ((wg + 3) & 3) + row;
    // demand of the thread's key in front of slice i (exclusive of its first query): the stored checkpoint of that 32-row block
    // (past the end: any value.  Queries behind the last one are rows of zeros in Q, dO' and dbar': their bids multiply zeros, and
    // what they add to a demand no query in front of them sees)
    const int rb = 2 * hl + 1 - wg;                            // of the warpgroup's first slice; four less for every other
    const float* edge = carry + ((int64_t)n * ncb + rb) * g.tk + ja;
    float incl = 0.f;
    if (!dead && wg < 2 * nh) incl = rb < ncb ? *edge : total[(int64_t)n * g.tk + ja];
    for (int i = wg; i < 2 * nh; i += 4) {
      const int u = i >> 1, q0 = (hl - u) * 64 + ((i & 1) ? 0 : 32);
      float incl_next = 0.f;                                   // read once, from a buffer far larger than L2
      edge -= 4 * (int64_t)g.tk;
      if (!dead && i + 4 < 2 * nh) incl_next = *edge;
      const float4* Dbar4 = reinterpret_cast<const float4*>(sDbar + 64 * (u & 3) + ((i & 1) ? 0 : 32));
      mbar_wait_warp(sdone + 8 * wg, (i >> 2) & 1, ctl, &g_status, kErrWaitMma);
      tc_fence_after();
      float p[32], inv[32];
      tmem_ld32(tSw, p);
      tmem_ld_wait(p);
      if (dead || q0 < k0 + kTileRows - 1) bids_and_inverses<SHARE, true>(p, inv, incl + g.eps, g, dead, ja - q0);
      else bids_and_inverses<SHARE, false>(p, inv, incl + g.eps, g, dead, ja - q0);
      __syncwarp();
      float suffix = 0.f;                                      // of the slice alone
#pragma unroll
      for (int c = 1; c >= 0; --c) {
        float vd[16];
        uint32_t shp[8];
        tmem_ld16(tDw + 16 * c, vd);
        tmem_ld_wait16(vd);
        suffix_of_eight<SHARE>(p + 16 * c + 8, inv + 16 * c + 8, vd + 8, Dbar4 + 4 * c + 2, suffix, shp + 4);
        suffix_of_eight<SHARE>(p + 16 * c, inv + 16 * c, vd, Dbar4 + 4 * c, suffix, shp);
        tmem_st8(tSw + 8 * c, shp);
      }
      float base = 0.f;                                        // the suffix behind the slice: dp is linear in it
      if (i > 0) {
        mbar_wait(behind, ((i - 1) >> 2) & 1, ctl, &g_status, kErrWaitTile);
        base = *sBehind;
      }
      sG[128 * wg + row] = base + suffix;
      __syncwarp();
      if (lane == 0) mbar_arrive(mine);
      uint32_t pdt[16];
#pragma unroll
      for (int e = 0; e < 32; e += 2) {
        const float2 pd2 = fma2(make_float2(p[e], p[e + 1]), make_float2(base, base), make_float2(inv[e], inv[e + 1]));
        pdt[e >> 1] = pack_bf16(pd2.x, pd2.y);
      }
      // the products of half tile u - 2 have read the pdp buffer that is written next
      if (u >= 2) mbar_wait_warp(dqdone + 8 * (u & 1), ((u >> 1) - 1) & 1, ctl, &g_status, kErrWaitMma);
#pragma unroll
      for (int c = 0; c < 4; ++c)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sPd + kTileBytes * (u & 1) +
                                                                      share_chunk_offset(row, ((i & 1) ? 0 : 32) + 8 * c)),
                     "r"(pdt[4 * c]), "r"(pdt[4 * c + 1]), "r"(pdt[4 * c + 2]), "r"(pdt[4 * c + 3])
                     : "memory");
      tmem_st16(tDw, pdt);
      incl = incl_next;
      tmem_st_wait();
      fence_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tiles + 8 * wg);
    }
  }
  mbar_wait(fin, 0, ctl, &g_status, kErrWaitMma);
  __syncwarp();
  tc_fence_after();
  if (wg < 4) {
    // lane = key: each warpgroup stores 16 of the 64 columns of dk_main and dv
    float a[16], b[16];
    const int64_t o = ((int64_t)n * g.tk + ja) * kHeadDim + 16 * wg;
    tmem_ld16(tDK + lane_base + 16 * wg, a);
    tmem_ld16(tDV + lane_base + 16 * wg, b);
    tmem_ld_wait16(a);
    tmem_ld_wait16(b);
    if (!dead) {
#pragma unroll
      for (int e = 0; e < 16; e += 4)
        *reinterpret_cast<float4*>(dk_main + o + e) =
            make_float4(a[e] * g.scale, a[e + 1] * g.scale, a[e + 2] * g.scale, a[e + 3] * g.scale);
#pragma unroll
      for (int e = 0; e < 16; e += 8)
        *reinterpret_cast<uint4*>(dv + o + e) =
            make_uint4(pack_bf16(b[e], b[e + 1]), pack_bf16(b[e + 2], b[e + 3]), pack_bf16(b[e + 4], b[e + 5]),
                       pack_bf16(b[e + 6], b[e + 7]));
    }
  }
  drain_if_aborted(ctl);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_free(tmem, 512);
}

// Barrier of the 128 threads of one warpgroup (named barriers 1 and 2).
__device__ __forceinline__ void wg_barrier(int wg) {
  if (wg == 0) asm volatile("bar.sync 1, 128;" ::: "memory");
  else asm volatile("bar.sync 2, 128;" ::: "memory");
}

// Softmax-Jacobian corrections (the reference's BC + dq epilogue, kernels.py:777-826):
//   dk = dk_main - scale * P^T (ghat * Q)        (accumulated here per key block)
//   dq = dq_main - scale * ghat * (P K)          (added to dq_main with vector reductions;
//                                                 the reference reads a saved pk instead)
// One bf16 tile W[key][query] = p * ghat serves both products: K-major it is the A
// operand with M = keys, MN-major the A operand with M = queries.
// grid = n * ceil(t/128); 256 threads, the two warpgroups split the tile's query
// columns; TMEM: S^T 128, dKc 64, dQc 64 (256; two CTAs per SM).
constexpr int kCorrSmem = 3 * kTileBytes + 2 * kTileBytes + 2048 + 1024 + 256;

__global__ void __launch_bounds__(256, 2) backward_correction_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
    const __grid_constant__ CUtensorMap map_dq, Geom g, const float* __restrict__ rmax,
    const float* __restrict__ rden, const float* __restrict__ ghat, const float* __restrict__ dk_main,
    __nv_bfloat16* __restrict__ dk) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  const uint32_t sK = smem_u32(smem), sQ0 = sK + kTileBytes, sW = sK + 3 * kTileBytes;
  float2* sStat = reinterpret_cast<float2*>(smem + 5 * kTileBytes);           // [2][128] (lse, ghat)
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 5 * kTileBytes + 2048);
  Ctl* ctl = reinterpret_cast<Ctl*>(bars + 8);
  const uint32_t qfull = smem_u32(bars), sdone = smem_u32(bars + 2), dqdone = smem_u32(bars + 3);

  const int tid = threadIdx.x, warp = tid >> 5, wg = tid >> 7, row = tid & 127;
  const int warp_u = uniform_warp();
  const uint32_t lead = elect_one();
  const int nqb = (g.tq + kTileRows - 1) / kTileRows;
  const int n = (int)(blockIdx.x % g.n);
  const int jb = (int)(blockIdx.x / g.n);
  const int k0 = jb * kTileRows;
  const int nsteps = nqb - jb;
  const int64_t row_base = (int64_t)n * g.tq;

  auto load_stats = [&](int ib) {
    const int i = ib * kTileRows + row;
    float2 st = make_float2(INFINITY, 0.f);
    if (i < g.tq) st = make_float2(rmax[row_base + i] + log2f(rden[row_base + i]), ghat[row_base + i]);
    return st;
  };

  if (tid == 0) {
    ctl->abort = 0;
    for (int i = 0; i < 4; ++i) mbar_init(qfull + 8 * i, 1);
    fence_barrier_init();
  }
  __syncwarp();
  if (warp == 0) tmem_alloc(smem_u32(&ctl->tmem), 256);
  if (wg == 1) sStat[row] = load_stats(jb);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = uniform(ctl->tmem);
  const uint32_t tS = tmem, tDK = tmem + 128, tDQ = tmem + 192;

  if (tid == 0) {
    mbar_expect_tx(qfull, 2 * kTileBytes);
    tma_load_tile(sK, &map_k, k0, n, qfull);
    tma_load_tile(sQ0, &map_q, jb * kTileRows, n, qfull);
    if (nsteps > 1) {
      mbar_expect_tx(qfull + 8, kTileBytes);
      tma_load_tile(sQ0 + kTileBytes, &map_q, (jb + 1) * kTileRows, n, qfull + 8);
    }
  }
  if (warp_u == 0) {
    __syncwarp();
    mbar_wait(qfull, 0, ctl, &g_status, kErrWaitTma);
    tc_fence_after();
    mma_scores_w<kNarrow>(lead, tS, sK, sQ0, 128);
    mma_commit(lead, sdone);
  }
  __syncwarp();

  const int ja = k0 + row;
  const bool dead = ja >= g.tk;
  const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
  for (int t = 0; t < nsteps; ++t) {
    const int ib = jb + t, b = t & 1;
    // next step's statistics as raw values: they are combined at the store below, when the
    // loads have long returned, so that no instruction waits for them here
    float nx_max = INFINITY, nx_den = 1.f, nx_gh = 0.f;
    if (wg == 1 && t + 1 < nsteps && (ib + 1) * kTileRows + row < g.tq) {
      const int64_t i = row_base + (ib + 1) * kTileRows + row;
      nx_max = rmax[i];
      nx_den = rden[i];
      nx_gh = ghat[i];
    }
    mbar_wait(sdone, t & 1, ctl, &g_status, kErrWaitMma);
    tc_fence_after();
    if (tid == 0 && t >= 1 && t + 1 < nsteps) {      // the Q stage of step t-1 is free
      mbar_expect_tx(qfull + 8 * (b ^ 1), kTileBytes);
      tma_load_tile(sQ0 + kTileBytes * (b ^ 1), &map_q, (ib + 1) * kTileRows, n, qfull + 8 * (b ^ 1));
    }
    __syncwarp();
    // this warpgroup's half of the W buffer doubled as its dQ staging area: the previous
    // step's reduction must have read it before it is written again
    if (row == 0) tma_wait_read_all();
    wg_barrier(wg);
    const int i0 = ib * kTileRows + 64 * wg;
    const bool masked_tile = dead || t == 0;
    const float4* St4 = reinterpret_cast<const float4*>(sStat + b * 128 + 64 * wg);
    auto tile = [&](auto mask_tag) {
    constexpr bool MASK = decltype(mask_tag)::value;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      float vs[32];
      uint32_t wt[16];                                 // this chunk's 32 W values as bf16 pairs
      tmem_ld32(tS + lane_base + 64 * wg + 32 * c, vs);
      tmem_ld_wait(vs);
      float4 snext[4];
#pragma unroll
      for (int u2 = 0; u2 < 4; ++u2) snext[u2] = St4[(c * 32) / 2 + u2];
#pragma unroll
      for (int e8 = 0; e8 < 4; ++e8) {
        float w8[8];
        float4 scur[4];
#pragma unroll
        for (int u2 = 0; u2 < 4; ++u2) scur[u2] = snext[u2];
        if (e8 < 3) {      // next group's statistics, read before this group's store
#pragma unroll
          for (int u2 = 0; u2 < 4; ++u2) snext[u2] = St4[(c * 32 + (e8 + 1) * 8) / 2 + u2];
        }
#pragma unroll
        for (int u2 = 0; u2 < 4; ++u2) {
          const float4 st = scur[u2];
          const float lse[2] = {st.x, st.z}, gh[2] = {st.y, st.w};
#pragma unroll
          for (int w = 0; w < 2; ++w) {
            const int u = u2 * 2 + w, e = e8 * 8 + u;
            float p = fast_exp2(fmaf(vs[e], g.zscale, -lse[w]));
            if (MASK && (dead || ja > i0 + c * 32 + e)) p = 0.f;
            w8[u] = p * gh[w];
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) wt[e8 * 4 + u] = pack_bf16(w8[2 * u], w8[2 * u + 1]);
        // shared memory: the MN-major A operand of dQc (M = queries)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sW + share_chunk_offset(row, wg * 64 + c * 32 + e8 * 8)),
                     "r"(wt[e8 * 4]), "r"(wt[e8 * 4 + 1]), "r"(wt[e8 * 4 + 2]), "r"(wt[e8 * 4 + 3])
                     : "memory");
      }
      // TMEM, over the score columns just consumed: the A operand of dKc (M = keys)
      tmem_st16(tS + lane_base + 64 * wg + 32 * c, wt);
    }
    };
    if (masked_tile) tile(std::true_type{}); else tile(std::false_type{});
    if (wg == 1 && t + 1 < nsteps) sStat[(b ^ 1) * 128 + row] = make_float2(nx_max + log2f(nx_den), nx_gh);
    tmem_st_wait();
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    if (warp_u == 0) {
      tc_fence_after();
      constexpr uint32_t id_kd = instr_desc(128, 64, 0, 1), id_qd = instr_desc(128, 64, 1, 1);
      // descriptors are built once per tile; a k-step is a constant 2048 B (128 units) further
      const Desc dQm = make_desc(sQ0 + kTileBytes * b, kTileBytes, 1024);
      const Desc dWm = make_desc(sW, kTileBytes, 1024), dKm = make_desc(sK, kTileBytes, 1024);
      // dQc first: its tile is what the threads read out next, and only it reads the shared-
      // memory W tile (the staging area of that read-out); dKc takes W from TMEM and runs,
      // with the next scores, under the read-out
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) mma_ss(lead, tDQ, dWm, 128 * kk, dKm, 128 * kk, id_qd, kk > 0);
      mma_commit(lead, dqdone);
#pragma unroll
      for (int kq = 0; kq < 8; ++kq)
        mma_ts(lead, tDK, tS + 64 * (kq >> 2) + 32 * ((kq & 3) >> 1) + 8 * (kq & 1), dQm, 128 * kq, id_kd,
               (t > 0 || kq > 0));
      if (t + 1 < nsteps) {
        mbar_wait(qfull + 8 * (b ^ 1), ((t + 1) >> 1) & 1, ctl, &g_status, kErrWaitTma);
        tc_fence_after();
        mma_scores_w<kNarrow>(lead, tS, sK, sQ0 + kTileBytes * (b ^ 1), 128);
      }
      mma_commit(lead, sdone);
    }
    __syncwarp();
    mbar_wait_warp(dqdone, t & 1, ctl, &g_status, kErrWaitMma);
    tc_fence_after();
    {
      // lane = query: each warpgroup owns 32 of the 64 columns.  The fp32 tile is staged in
      // the (now free) W buffer in the copy engine's swizzled layout and added to dq_main
      // by ONE tensor reduction per warpgroup: 128 B per row instead of eight scattered
      // 16-byte reductions per thread.
      float dq[32];
      tmem_ld32(tDQ + lane_base + 32 * wg, dq);
      tmem_ld_wait(dq);
      const float ns = -g.scale;
      const uint32_t stage = sW + kTileBytes * wg + row * 128;
#pragma unroll
      for (int c = 0; c < 8; ++c)
        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(stage + ((c ^ (row & 7)) << 4)),
                     "f"(dq[4 * c] * ns), "f"(dq[4 * c + 1] * ns), "f"(dq[4 * c + 2] * ns), "f"(dq[4 * c + 3] * ns)
                     : "memory");
      fence_async_smem();
      tc_fence_before();
      wg_barrier(wg);
      if (row == 0) tma_reduce_add_tile(&map_dq, sW + kTileBytes * wg, 32 * wg, ib * kTileRows, n);
    }
    tc_fence_before();
  }
  if (row == 0) tma_wait_read_all();
  mbar_wait_warp(sdone, nsteps & 1, ctl, &g_status, kErrWaitMma);
  tc_fence_after();
  {
    // lane = key: each warpgroup finishes 32 of the 64 columns of dk
    float a[32];
    const int64_t o = ((int64_t)n * g.tk + ja) * kHeadDim + 32 * wg;
    tmem_ld32(tDK + lane_base + 32 * wg, a);
    tmem_ld_wait(a);
    if (!dead) {
      float m[32];
#pragma unroll
      for (int e = 0; e < 32; e += 4) {
        const float4 x = *reinterpret_cast<const float4*>(dk_main + o + e);
        m[e] = x.x - g.scale * a[e];
        m[e + 1] = x.y - g.scale * a[e + 1];
        m[e + 2] = x.z - g.scale * a[e + 2];
        m[e + 3] = x.w - g.scale * a[e + 3];
      }
#pragma unroll
      for (int e = 0; e < 32; e += 8)
        *reinterpret_cast<uint4*>(dk + o + e) =
            make_uint4(pack_bf16(m[e], m[e + 1]), pack_bf16(m[e + 2], m[e + 3]),
                       pack_bf16(m[e + 4], m[e + 5]), pack_bf16(m[e + 6], m[e + 7]));
    }
  }
  drain_if_aborted(ctl);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_free(tmem, 256);
}

// dq = bf16(dq_main)
__global__ void cast_dq_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, int64_t n4) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n4) return;
  const float4 x = reinterpret_cast<const float4*>(src)[i];
  reinterpret_cast<uint2*>(dst)[i] = make_uint2(pack_bf16(x.x, x.y), pack_bf16(x.z, x.w));
}

// ---------------------------------------------------------------- host launchers
#define DILUTION_TC_HAS_MAIN 1
#define DILUTION_TC_HAS_BACKWARD 1

// The opt-in to more than 48 KB of dynamic shared memory is per kernel and per device: it is
// made on the first launch of that kernel on that device and remembered.
// regs: registers per thread that the kernel's setmaxnreg split needs at launch.  An increase beyond what the block was launched
// with waits for ever, so a build in which the compiler took fewer is refused here.
inline int set_smem_attr(const void* fn, int bytes, char* err, size_t errlen, int regs = 0) {
  static OncePerDevice opted_in;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) dev = -1;
  if (opted_in.done(fn, dev)) return 0;
  if (regs > 0) {
    cudaFuncAttributes at;
    const cudaError_t e = cudaFuncGetAttributes(&at, fn);
    if (e != cudaSuccess || at.numRegs < regs) {
      if (e != cudaSuccess) snprintf(err, errlen, "cudaFuncGetAttributes: %s", cudaGetErrorString(e));
      else snprintf(err, errlen, "kernel built with %d registers, its split needs %d", at.numRegs, regs);
      return 3;
    }
  }
  const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) {
    snprintf(err, errlen, "cudaFuncSetAttribute(%d): %s", bytes, cudaGetErrorString(e));
    return 3;
  }
  opted_in.set(fn, dev);
  return 0;
}

inline int launch_status(const char* what, char* err, size_t errlen) {
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    snprintf(err, errlen, "%s: %s", what, cudaGetErrorString(e));
    return 3;
  }
  return 0;
}

// Shared memory of the 256-column kernels is padded so that at most two CTAs share
// an SM (an SM has 512 TMEM columns); the 128-column kernels fit four by themselves.
constexpr int kTwoPerSm = 100 * 1024;
static_assert(5 * (kRowstatsSmem<kNarrow> + 1024) > 233472 && 5 * (kColsumSmem<kNarrow> + 1024) > 233472,
              "at most four CTAs of a 128-column kernel may share an SM");

// Compile-time bid / share of a launch from the run-time fields of its geometry.
#define DIL_TC_SHARE(g, ...)                                                                       \
  if ((g).share == kShareInclusive) { constexpr int SHARE = kShareInclusive; __VA_ARGS__; }        \
  else if ((g).share == kShareExclusive) { constexpr int SHARE = kShareExclusive; __VA_ARGS__; }   \
  else { constexpr int SHARE = kShareNone; __VA_ARGS__; }
// (only the inclusive share step takes reciprocals of consecutive demands together)
#define DIL_TC_PAIR(g, SHARE, ...)                                                                       \
  if (SHARE != kShareInclusive || pair_demands(g)) { constexpr bool PAIR = true; __VA_ARGS__; }          \
  else { constexpr bool PAIR = SHARE != kShareInclusive; __VA_ARGS__; }
#define DIL_TC_PLAIN_BID(g, ...)                                               \
  if ((g).bid == kBidSigmoid) { constexpr int BID = kBidSigmoid; __VA_ARGS__; } \
  else { constexpr int BID = kBidSoftmax; __VA_ARGS__; }
#define DIL_TC_MASS_BID(g, ...)                                                     \
  if ((g).bid == kBidRelu) { constexpr int BID = kBidRelu; __VA_ARGS__; }           \
  else if ((g).bid == kBidRelu2) { constexpr int BID = kBidRelu2; __VA_ARGS__; }    \
  else { constexpr int BID = kBidSoftplus; __VA_ARGS__; }
#define DIL_TC_BID(g, ...)                                            \
  if (row_sum_bid((g).bid)) { DIL_TC_MASS_BID(g, __VA_ARGS__) }       \
  else { DIL_TC_PLAIN_BID(g, __VA_ARGS__) }

inline int rowstats(const void* q, const void* k, const Geom& g, float* rmax, float* rden,
                    cudaStream_t st, char* err, size_t errlen) {
  CUtensorMap mq, mk;
  if (int rc = make_map(&mq, q, g.n, g.tq, err, errlen)) return rc;
  if (int rc = make_map(&mk, k, g.n, g.tk, err, errlen)) return rc;
  constexpr int smem = kRowstatsSmem<kNarrow>;
  const int nqb = (g.tq + kTileRows - 1) / kTileRows;
  auto launch = [&](auto kern) -> int {
    if (int rc = set_smem_attr((const void*)kern, smem, err, errlen)) return rc;
    kern<<<(unsigned)(g.n * nqb), 256, smem, st>>>(mq, mk, g, rmax, rden);
    return 0;
  };
  if (int rc = g.bid == kBidRelu       ? launch(rowstats_kernel<kNarrow, kBidRelu>)
               : g.bid == kBidRelu2    ? launch(rowstats_kernel<kNarrow, kBidRelu2>)
               : g.bid == kBidSoftplus ? launch(rowstats_kernel<kNarrow, kBidSoftplus>)
                                       : launch(rowstats_kernel<>)) return rc;
  return launch_status("tc rowstats", err, errlen);
}

inline int colsum_scan(const void* q, const void* k, const Geom& g, const float* rmax,
                       const float* rden, const float* carry_base, float* carry, float* total,
                       cudaStream_t st, char* err, size_t errlen) {
  CUtensorMap mq, mk;
  if (int rc = make_map(&mq, q, g.n, g.tq, err, errlen)) return rc;
  if (int rc = make_map(&mk, k, g.n, g.tk, err, errlen)) return rc;
  constexpr int smem = kColsumSmem<kNarrow>;
  const int nkb = (g.tk + kTileRows - 1) / kTileRows;
  const unsigned grid = (unsigned)(g.n * nkb);
  if (g.carry_rows == 32) {
    DIL_TC_BID(g, {
      if (int rc = set_smem_attr((const void*)colsum_scan_kernel<32, BID>, smem, err, errlen)) return rc;
      colsum_scan_kernel<32, BID><<<grid, 256, smem, st>>>(mq, mk, g, rmax, rden, carry_base, carry, total);
    })
  } else {                              // forward-only calls of the operator
    if (int rc = set_smem_attr((const void*)colsum_scan_kernel<64>, smem, err, errlen)) return rc;
    colsum_scan_kernel<64><<<grid, 256, smem, st>>>(mq, mk, g, rmax, rden, carry_base, carry, total);
  }
  return launch_status("tc colsum_scan", err, errlen);
}

inline int forward_main(const void* q, const void* k, const void* v, const Geom& g, const float* rmax,
                        const float* rden, const float* carry, const float* carry_base, float* out,
                        float* ssum, cudaStream_t st, char* err, size_t errlen) {
  CUtensorMap mq, mk, mv;
  if (int rc = make_map(&mq, q, g.n, g.tq, err, errlen)) return rc;
  if (int rc = make_map(&mk, k, g.n, g.tk, err, errlen)) return rc;
  if (int rc = make_map(&mv, v, g.n, g.tk, err, errlen)) return rc;
  constexpr int smem = kMainSmem<kNarrow>;
  static_assert(2 * (smem + 1024) <= 233472 && 3 * (smem + 1024) > 233472, "exactly two CTAs of the main pass fit one SM");
  const int nqb = (g.tq + kTileRows - 1) / kTileRows;
  const unsigned grid = (unsigned)(g.n * nqb);
  DIL_TC_SHARE(g, DIL_TC_PAIR(g, SHARE, {
    if (g.bid == kBidSigmoid) {
      auto kern = forward_main_async_kernel<kBidSigmoid, SHARE, kNarrow, PAIR>;
      if (int rc = set_smem_attr((const void*)kern, smem, err, errlen)) return rc;
      kern<<<grid, kMainThreads<kNarrow>, smem, st>>>(mq, mk, mv, g, rmax, rden, carry, carry_base, nullptr, out, ssum);
    } else {
      auto kern = g.normalised ? forward_main_kernel<SHARE, PAIR> : forward_main_kernel<SHARE, SHARE != kShareInclusive, kBidExpshift>;
      if (int rc = set_smem_attr((const void*)kern, smem, err, errlen)) return rc;
      kern<<<grid, 256, smem, st>>>(mq, mk, mv, g, rmax, rden, carry, carry_base, out, ssum);
    }
  }))
  return launch_status("tc forward_main", err, errlen);
}

int backward_tail_with_pk(const CUtensorMap& mq, const CUtensorMap& mk, const Geom& g, const float* rmax,
                          const float* rden, const float* ghat, const float* dk_main, const float* dq_main,
                          const float* pk, void* dq, void* dk, cudaStream_t st, char* err, size_t errlen,
                          void (*mark)(const char*, cudaStream_t, int));

// dop: (n, t, 64) bf16 scratch for the pre-scaled dout.  pk: the query correction saved by the
// forward (rowstats_pk), or null: the correction pass then recomputes it.
inline int backward(const void* q, const void* k, const void* v, const Geom& g, const void* dout,
                    int dout_dtype, const float* out, const float* rmax, const float* rden, const float* carry,
                    const float* total, const float* ssum, const float* pk, float* dq_main, float* dk_main,
                    float* ghat,
                    float* dbarp, void* dop, void* dq, void* dk, void* dv, cudaStream_t st, char* err,
                    size_t errlen, void (*mark)(const char*, cudaStream_t, int)) {
  CUtensorMap mq, mk;
  if (int rc = make_map(&mq, q, g.n, g.tq, err, errlen)) return rc;
  if (int rc = make_map(&mk, k, g.n, g.tk, err, errlen)) return rc;
  CUtensorMap md;
  if (int rc = make_map(&md, dop, g.n, g.tq, err, errlen)) return rc;
  const int64_t rows = g.n * g.tq;
  const int nkb = (g.tk + kTileRows - 1) / kTileRows;
  mark("tc_backward_prep", st, 0);
  if (dout_dtype == 0)
    backward_prep_kernel<float><<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(
        (const float*)dout, out, ssum, g.eps, rows, dbarp, (__nv_bfloat16*)dop, ghat, dq_main);
  else
    backward_prep_kernel<__nv_bfloat16><<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(
        (const __nv_bfloat16*)dout, out, ssum, g.eps, rows, dbarp, (__nv_bfloat16*)dop, ghat, dq_main);
  mark("tc_backward_prep", st, 1);
  if (int rc = launch_status("tc backward_prep", err, errlen)) return rc;
  CUtensorMap mdq;
  if (int rc = make_map_f32(&mdq, dq_main, g.n, g.tq, err, errlen)) return rc;
  if (g.carry_rows == 32) {
    constexpr int smem_bwd = kBwdSmem;
    static_assert(smem_bwd <= 232448 && 2 * smem_bwd > 233472, "the backward main pass runs one CTA per SM");
    const unsigned grid = (unsigned)(g.n * nkb);
    const bool slices = g.bid == kBidSigmoid && g.share != kShareNone && g.tq >= kSliceFrom;
    if (slices) {
      CUtensorMap mq64, md64, mdq64;
      if (int rc = make_map(&mq64, q, g.n, g.tq, err, errlen, kHeadDim, 64)) return rc;
      if (int rc = make_map(&md64, dop, g.n, g.tq, err, errlen, kHeadDim, 64)) return rc;
      if (int rc = make_map_f32(&mdq64, dq_main, g.n, g.tq, err, errlen, kHeadDim, 64, false)) return rc;
      if (((uintptr_t)k | (uintptr_t)v) & 15) {
        snprintf(err, errlen, "bf16 tensor-core path needs 16-byte aligned q/k/v");
        return 1;
      }
      static_assert(kSliceSmem <= 232448 && 2 * kSliceSmem > 233472, "the main reverse pass runs one CTA per SM");
      auto kern = g.share == kShareInclusive ? backward_slices_kernel<kShareInclusive> : backward_slices_kernel<kShareExclusive>;
      if (int rc = set_smem_attr((const void*)kern, kSliceSmem, err, errlen, kSliceRegs)) return rc;
      mark("tc_backward_main", st, 0);
      kern<<<grid, kSliceThreads, kSliceSmem, st>>>(mq64, mk, md64, mdq64, g, (const __nv_bfloat16*)k, (const __nv_bfloat16*)v, dbarp,
                                                    carry, total, dk_main, (__nv_bfloat16*)dv);
    } else {
      mark("tc_backward_main", st, 0);
      DIL_TC_PLAIN_BID(g, DIL_TC_SHARE(g, {
        if (int rc = set_smem_attr((const void*)backward_main_kernel<BID, SHARE>, smem_bwd, err, errlen, kBwdRegs)) return rc;
        backward_main_kernel<BID, SHARE><<<grid, kBwdThreads, smem_bwd, st>>>(
            mq, mk, md, mdq, g, (const __nv_bfloat16*)v, rmax, rden, dbarp, carry, total, dq_main, dk_main,
            (__nv_bfloat16*)dv, ghat);
      }))
    }
    mark("tc_backward_main", st, 1);
  } else {
    snprintf(err, errlen, "the tensor-core backward needs checkpoints every 32 query rows (got %d)", g.carry_rows);
    return 1;
  }
  if (int rc = launch_status("tc backward_main", err, errlen)) return rc;
  if (!g.normalised || g.share == kShareNone) {
    // no row normalisation in the bid: no Jacobian correction, dk and dq are dk_main and dq_main.
    // Without a share step the correction of the softmax bid vanishes identically:
    // ghat_i = sum_j p_ij (do_i.v_j - do_i.out_i) = do_i.out_i - do_i.out_i = 0 (out_i = sum_j p_ij v_j).
    const int64_t n4 = rows * kHeadDim / 4;
    mark("tc_cast_dk_dq", st, 0);
    cast_dq_kernel<<<(unsigned)((n4 + 255) / 256), 256, 0, st>>>(dk_main, (__nv_bfloat16*)dk, n4);
    cast_dq_kernel<<<(unsigned)((n4 + 255) / 256), 256, 0, st>>>(dq_main, (__nv_bfloat16*)dq, n4);
    mark("tc_cast_dk_dq", st, 1);
    return launch_status("tc cast_dk_dq", err, errlen);
  }
  if (pk != nullptr)
    return backward_tail_with_pk(mq, mk, g, rmax, rden, ghat, dk_main, dq_main, pk, dq, dk, st, err, errlen, mark);
  constexpr int smem = kCorrSmem > kTwoPerSm ? kCorrSmem : kTwoPerSm;
  if (int rc = set_smem_attr((const void*)backward_correction_kernel, smem, err, errlen)) return rc;
  mark("tc_backward_correction", st, 0);
  backward_correction_kernel<<<(unsigned)(g.n * nkb), 256, smem, st>>>(mq, mk, mdq, g, rmax, rden, ghat,
                                                                     dk_main, (__nv_bfloat16*)dk);
  mark("tc_backward_correction", st, 1);
  if (int rc = launch_status("tc backward_correction", err, errlen)) return rc;
  const int64_t n4 = rows * kHeadDim / 4;
  mark("tc_cast_dq", st, 0);
  cast_dq_kernel<<<(unsigned)((n4 + 255) / 256), 256, 0, st>>>(dq_main, (__nv_bfloat16*)dq, n4);
  mark("tc_cast_dq", st, 1);
  return launch_status("tc cast_dq", err, errlen);
}

// Self-test of the bounded wait: one CTA waits on an mbarrier phase that nothing will
// ever complete, with a short limit (about a millisecond).  The wait must give up,
// record kErrSelfTest and let the kernel return normally; nothing faults or hangs.
__global__ void selftest_wait_kernel(long long limit_cycles, int* __restrict__ gave_up) {
  __shared__ uint64_t bar;
  __shared__ Ctl ctl;
  if (threadIdx.x == 0) {
    ctl.abort = 0;
    mbar_init(smem_u32(&bar), 1);
    fence_barrier_init();
  }
  __syncthreads();
  const bool ok = mbar_wait(smem_u32(&bar), 0, &ctl, &g_status, kErrSelfTest, limit_cycles);
  __syncthreads();
  if (threadIdx.x == 0) *gave_up = ok ? 0 : 1;
}

inline int selftest_wait(int* gave_up_dev, cudaStream_t st, char* err, size_t errlen) {
  selftest_wait_kernel<<<1, 64, 0, st>>>(2000000LL, gave_up_dev);
  return launch_status("selftest_wait", err, errlen);
}

// Reads (and clears) the device status word; synchronises the device.
inline int read_status(int* out) {
  int v = 0;
  // kernels on non-blocking streams are not ordered before a copy on the default stream
  if (cudaDeviceSynchronize() != cudaSuccess) return 3;
  if (cudaMemcpyFromSymbol(&v, g_status, sizeof(int)) != cudaSuccess) return 3;
  if (v != 0) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_status, &zero, sizeof(int));
  }
  *out = v;
  return 0;
}

}  // namespace tc
}  // namespace dil
