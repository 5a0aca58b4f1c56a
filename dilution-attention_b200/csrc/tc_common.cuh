// Blackwell (sm_100a) building blocks for the bf16 tensor-core path: mbarriers
// with bounded waits, TMA tile loads, TMEM allocation, tcgen05.mma issue/commit
// and tcgen05.ld, plus the shared-memory and instruction descriptors they take.
//
// Conventions used by every kernel built on these:
//  * operand tiles are [128 rows][64 bf16] = 16 KB, written by TMA with the
//    128-byte swizzle; row pitch 128 B, 8-row groups 1024 B apart, tile base
//    1024-byte aligned.  Read as a K-major operand the rows are the M/N index
//    and the 64 elements the contraction index; read as an MN-major operand the
//    64 elements are the M/N index and the rows the contraction index;
//  * accumulators live in TMEM with M = 128: row r of D is TMEM lane r, column
//    c of D is TMEM column base+c (fp32);
//  * every wait on an mbarrier gives up after kWaitCycles, records a code in the
//    device status word and raises the CTA's abort flag; later waits return at
//    once, the CTA drains, frees its TMEM and exits.  Loop bounds and addresses
//    never depend on data, so an aborted CTA stays in bounds.
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace dil {
namespace tc {

constexpr int kTileRows = 128;
constexpr int kHeadDim = 64;
constexpr uint32_t kTileBytes = kTileRows * kHeadDim * 2;   // 16 KB
constexpr long long kWaitCycles = 4000000000LL;             // ~2 s: a live wait is microseconds

// How many [rows][64 bf16] sub-tiles one row of q, k, v takes, what they hold, and how exactly the kernels
// multiply the values that they form (shares, pdp, P~, W).
//   kNarrow : heads of 64 in bf16, one sub-tile; formed values rounded to bf16;
//   kWide128: heads of 128 in bf16, two sub-tiles of 64 features;
//   kPairs64: heads of 64 in bf16, one sub-tile;
//   kSplit  : heads of up to 64 in fp32, each value as hi + lo with hi = bf16(x), lo = bf16(x - hi) (split_pair):
//             sub-tile 0 holds the hi parts, sub-tile 1 the lo parts (zeros behind the head size).  A product of
//             two such operands keeps 16 bits of each (2^-17 relative), where tf32 keeps 11.
// All but kNarrow form hi + lo pairs too (kPlanes), and take do' as hi + lo: [hi | lo] sub-tiles.
// Sub-tile s of a [128 rows] tile lies kTileBytes * s behind its start.
enum : int { kNarrow = 0, kWide128 = 1, kSplit = 2, kPairs64 = 3 };
template <int W> struct Rows {
  static constexpr int kSub = W == kWide128 || W == kSplit ? 2 : 1;
  static constexpr int kPlanes = W == kNarrow ? 1 : 2;             // bf16 parts of a value the kernels form
  static constexpr int kCols = 64 * kSub;                          // accumulator columns of a product with k, v, q or dout
  static constexpr int kHead = W == kWide128 ? 128 : 64;           // head size (kSplit: padded)
  static constexpr uint32_t kBytes = kSub * kTileBytes;            // one [128 rows] tile
  // score products: sub-tile pairs (a, b) that are multiplied.  kSplit leaves out lo * lo (2^-18 of the score).
  static constexpr int kPairs = W == kSplit ? 3 : kSub;
  static __device__ constexpr int pair_a(int i) { return W == kSplit ? (i == 2) : i; }
  static __device__ constexpr int pair_b(int i) { return W == kSplit ? (i == 1) : i; }
  // the same of V do'^T, and the parts of do' that dV takes one after the other (kSplit: both in one N = 128 product)
  static constexpr int kDoSub = W == kNarrow ? 1 : W == kWide128 ? 4 : 2;
  static constexpr int kDoPairs = W == kSplit ? 3 : kDoSub;
  static __device__ constexpr int do_a(int i) { return W == kSplit ? (i == 2) : W == kWide128 ? (i & 1) : 0; }
  static __device__ constexpr int do_b(int i) { return W == kSplit ? (i == 1) : i; }
  static constexpr int kDoParts = W == kSplit || W == kNarrow ? 1 : 2;
};

enum : int { kErrWaitTma = 101, kErrWaitMma = 102, kErrWaitDrain = 103, kErrAlign = 104, kErrWaitTile = 105, kErrSelfTest = 199 };

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// ---- mbarrier ---------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Per-CTA control block in shared memory.
struct Ctl {
  volatile int abort;   // raised by the first wait that ran out
  uint32_t tmem;        // written by tcgen05.alloc
};

// Bounded wait.  Returns false (after one probe, if the CTA is already aborting) when
// the phase did not complete in time.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, Ctl* ctl, int* status,
                                          int code, long long limit = kWaitCycles) {
  if (mbar_try(bar, parity)) return true;      // the common case costs one instruction
  if (ctl->abort) return false;
  const long long t0 = clock64();
  while (!mbar_try(bar, parity)) {
    if (clock64() - t0 > limit) {
      ctl->abort = 1;
      atomicCAS(status, 0, code);
      return false;
    }
  }
  return true;
}

// The wait of a whole warp: its lanes meet behind it.  Every lane polls for itself and may leave in another turn than its
// neighbours, but TMEM loads and stores and register hand-overs want the warp whole (.sync.aligned).  In a warp that issues only
// the elected lane's MMAs, commits and copies make the barriers go on; a lane that was still polling when the phase after the next
// began would wait for a parity that comes back no more.  No such lane can exist if nothing is issued before all have seen the phase.
__device__ __forceinline__ void mbar_wait_warp(uint32_t bar, uint32_t parity, Ctl* ctl, int* status, int code) {
  mbar_wait(bar, parity, ctl, status, code);
  __syncwarp();
}

// After a wait has given up, the CTA runs to its end without waiting for anything, so copies and
// MMAs it issued may still be in flight when it gets there.  Every kernel calls this in front of its
// last CTA-wide barrier: a CTA that gave up idles for a fixed grace period (about 0.2 ms, three
// orders of magnitude above a copy's or an MMA's latency) before it frees its TMEM and returns.
__device__ __forceinline__ void drain_if_aborted(const Ctl* ctl) {
  if (ctl->abort) {
    const long long t0 = clock64();
    while (clock64() - t0 < 400000LL) {
    }
  }
}

// ---- fences -------------------------------------------------------------------
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ---- TMA ----------------------------------------------------------------------
// One [box rows][64 bf16] tile of a (n, t, 64 or 128) tensor: coordinates (col, row, n).
__device__ __forceinline__ void tma_load_tile(uint32_t dst, const CUtensorMap* map, int row, int n,
                                              uint32_t bar, int col = 0) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];"
      :
      : "r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(col), "r"(row), "r"(n)
      : "memory");
}

// All sub-tiles of one tile, `sub_bytes` apart (kTileBytes for 128 rows).
template <int W, int SUB = Rows<W>::kSub>
__device__ __forceinline__ void tma_load_rows(uint32_t dst, const CUtensorMap* map, int row, int n, uint32_t bar,
                                              uint32_t sub_bytes = kTileBytes) {
#pragma unroll
  for (int s = 0; s < SUB; ++s) tma_load_tile(dst + sub_bytes * s, map, row, n, bar, 64 * s);
}

// Element-wise add of a shared-memory tile into global memory (performed at L2), one
// instruction for the whole box; coordinates (col, row, n).  Rows/columns outside the
// tensor are dropped.  The issuing thread commits the group and, before the tile is
// overwritten, waits until the copy engine has read it.
__device__ __forceinline__ void tma_reduce_add_tile(const CUtensorMap* map, uint32_t src, int col, int row,
                                                    int n) {
  asm volatile(
      "cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.bulk_group [%0, {%2, %3, %4}], [%1];"
      :
      : "l"(reinterpret_cast<uint64_t>(map)), "r"(src), "r"(col), "r"(row), "r"(n)
      : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void tma_wait_read_all() {
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

__device__ __forceinline__ void tma_wait_read_all_but_one() {
  asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
}

// ---- TMEM -----------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t slot_smem, uint32_t cols) {   // whole warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_smem),
               "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t taddr, uint32_t cols) {         // whole warp
  __syncwarp();
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols)
               : "memory");
}

// 32 consecutive fp32 columns of this thread's lane.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32"
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15,"
      " %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31},"
      " [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
// Loads fill their registers asynchronously.  Every wait names those it is for, so that the compiler cannot move a use
// of them above it.
__device__ __forceinline__ void tmem_ld_wait(float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]),
                 "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]),
                 "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]),
                 "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]),
                 "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}

// One fp32 column of this thread's lane.
__device__ __forceinline__ void tmem_ld1(uint32_t taddr, float* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];"
               : "=r"(*reinterpret_cast<uint32_t*>(v))
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld_wait1(float* v) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(*reinterpret_cast<uint32_t*>(v)) : : "memory");
}

// 16 consecutive fp32 columns of this thread's lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32"
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait16(float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]),
                 "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]),
                 "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}

// 16 consecutive 32-bit columns of this thread's lane, written from registers.
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0],"
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      :
      : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               :
               : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// ---- descriptors ------------------------------------------------------------------
// Shared-memory matrix descriptor, 128-byte swizzle, for the 16 KB tile layout above.
//   K-major view : 8-row groups 1024 B apart (SBO); LBO unused.
//   MN-major view: the 64 contiguous elements are one MN group (LBO = distance to the
//                  next group of 64, for tiles wider than 64); 8 contraction rows per
//                  1024 B (SBO).
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;   // descriptor version of this architecture
  d |= (uint64_t)2 << 61;   // 128-byte swizzle
  return d;
}

// Instruction descriptor: bf16 x bf16 -> fp32, M x N, operand majors (0 = K-major, 1 = MN-major).
__host__ __device__ constexpr uint32_t instr_desc(int m, int n, int a_mn, int b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// Whole warps issue MMAs: every lane runs the issuing code, in step, and the instruction itself is predicated on one elected
// lane.  An MMA takes its addresses and descriptors from uniform registers; where a single lane runs the code (if (lane == 0))
// the compiler holds them in ordinary ones and moves each of them over in front of each instruction, 80 cycles per MMA in
// the row pass (8 of them and the commit: 650 cycles, as uniform code 120; n = 64, T = 8192).  Everything the operands
// are made of must be uniform in the compiler's eyes too: uniform() for what comes out of memory, uniform_warp() for the
// branch.  lead: elect_one(), asked once per thread, where the warp is in step.
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t uniform(uint32_t x) { return __shfl_sync(0xffffffffu, x, 0); }
__device__ __forceinline__ int uniform_warp() { return (int)uniform(threadIdx.x >> 5); }

// Arrive on an mbarrier once every MMA issued so far by this thread has completed.
__device__ __forceinline__ void mma_commit(uint32_t lead, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
      ::"r"(bar), "r"(lead)
      : "memory");
}

// A descriptor is kept as two 32-bit halves.  The start address sits in the low half, so
// stepping through a tile is one 32-bit add of a constant to a value built once outside
// the loop.
struct Desc {
  uint32_t lo, hi;
};
__device__ __forceinline__ Desc make_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  const uint64_t d = smem_desc(saddr, lbo_bytes, sbo_bytes);
  return Desc{(uint32_t)d, (uint32_t)(d >> 32)};
}
// D[tmem] (+)= A[smem] * B[smem]; one instruction covers 16 contraction elements.
// Offsets are added in descriptor units of 16 bytes.
__device__ __forceinline__ void mma_ss(uint32_t lead, uint32_t d_tmem, Desc a, uint32_t a_off16, Desc b, uint32_t b_off16,
                                       uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %2};\n\t"
      "mov.b64 db, {%3, %4};\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "setp.ne.b32 q, %7, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}"
      :
      : "r"(d_tmem), "r"(a.lo + a_off16), "r"(a.hi), "r"(b.lo + b_off16), "r"(b.hi), "r"(idesc),
        "r"(accumulate), "r"(lead)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]: A is an M x 16 bf16 operand held in TMEM, row m on
// lane m, two consecutive contraction elements per 32-bit column (8 columns).
__device__ __forceinline__ void mma_ts(uint32_t lead, uint32_t d_tmem, uint32_t a_tmem, Desc b, uint32_t b_off16,
                                       uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 db;\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "setp.ne.b32 q, %6, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}"
      :
      : "r"(d_tmem), "r"(a_tmem), "r"(b.lo + b_off16), "r"(b.hi), "r"(idesc), "r"(accumulate), "r"(lead)
      : "memory");
}

// S[128 x n_cols] = A[128 rows] * B[n_cols rows]^T over the features of a row, both K-major: four instructions per
// pair of sub-tiles, which lie a_sub and b_sub bytes apart.
template <int W>
__device__ __forceinline__ void mma_scores_wide(uint32_t lead, uint32_t d_tmem, Desc a, uint32_t a_sub, Desc b, uint32_t b_sub,
                                                uint32_t idesc) {
#pragma unroll
  for (int i = 0; i < Rows<W>::kPairs; ++i)
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
      mma_ss(lead, d_tmem, a, (a_sub >> 4) * Rows<W>::pair_a(i) + 2 * kk, b, (b_sub >> 4) * Rows<W>::pair_b(i) + 2 * kk, idesc,
             i > 0 || kk > 0);
}
// The same of V do'^T.
template <int W>
__device__ __forceinline__ void mma_dov_wide(uint32_t lead, uint32_t d_tmem, Desc a, uint32_t a_sub, Desc b, uint32_t b_sub, uint32_t idesc) {
#pragma unroll
  for (int i = 0; i < Rows<W>::kDoPairs; ++i)
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
      mma_ss(lead, d_tmem, a, (a_sub >> 4) * Rows<W>::do_a(i) + 2 * kk, b, (b_sub >> 4) * Rows<W>::do_b(i) + 2 * kk, idesc,
             i > 0 || kk > 0);
}
template <int W>
__device__ __forceinline__ void mma_scores_w(uint32_t lead, uint32_t d_tmem, uint32_t a_smem, uint32_t b_smem, int n_cols) {
  mma_scores_wide<W>(lead, d_tmem, make_desc(a_smem, 16, 1024), kTileBytes, make_desc(b_smem, 16, 1024), kTileBytes,
                     instr_desc(128, n_cols, 0, 0));
}

// Dynamic shared memory base rounded up to 1024 bytes.
__device__ __forceinline__ uint8_t* align1024(uint8_t* p) {
  return p + ((1024u - (smem_u32(p) & 1023u)) & 1023u);
}

}  // namespace tc
}  // namespace dil
