// Chunked-prefill attention on the 5th-generation tensor cores (tcgen05 + TMEM), 16-bit caches.
//
// An item is 128 query rows that share a KV head: 128 / n tokens times the n query heads of the head's
// group (a group wider than 128 is cut into equal ones), so that a short tail of a prompt fills rows
// with heads instead of leaving a tile per head nearly empty.  A unit of work is two neighbouring items
// of one sequence.  A cluster of two CTAs (two SMs) works through the units the host dealt to it; CTA r holds the rows of item r
// and half of every K / V tile, and one tcgen05.mma of the pair (cta_group::2, 256 rows) reads both
// halves, so each K / V byte crosses L2 once for 256 rows.
// What bounds it is the tensor pipe: 24 products of 128 x 128 x 16 per SM and 128-key tile (8 scores,
// 16 weights times V: a weight travels as two 16-bit terms), 1536 clocks.  Everything else is kept off
// that path:
//   * tensor memory holds three score / weight buffers and O (4 x 128 columns), so the scores of the
//     next tiles are issued before the weights of this one are back;
//   * one warp issues the scores, another the P V: what a warp does between two batches of MMAs (a look at
//     a barrier behind a batch takes it 330 clocks) lies under the other's products.  Each waits for one
//     barrier a step, on which everything that step needs arrives;
//   * two softmax groups of four warps take every other tile, a thread per query row: no exchange
//     within a row, and a tile's softmax has two tiles' time.  The weights are handed over in two halves;
//   * a cluster is persistent: the rows of a finished unit are taken out of tensor memory by the group that had
//     its last tile while the other is at the next unit's first, whose Q, K and V are in shared memory already,
//     and leave by TMA.
//
// Before, one CTA held two items with one score buffer each: scores -> softmax -> P V of an item were one
// chain, 4650 clocks for a tile of both (3072 of them MMAs), and a CTA's start and end (7 us) stood alone.  Now
// 1900 clocks a tile and SM (1536), bound by the loop over three buffers: scores seen, softmax 3300, P V, scores.
// Prompts with their RoPE and append, us: 28/4 heads bf16, 4 x 2048 tokens in chunks of 512 306 -> 280; 32/8 fp16,
// 777 tokens 43.4 -> 30.4; 32/8 bf16, 16384 tokens in chunks of 2048 3237 -> 2729 (power-limited, 1.75 GHz).
// Measured and dropped: an eighth or a quarter of the exponentials as polynomials on the FMA units (312 -> 315 and
// 327 us a call of 2048 tokens behind 8192: they are not what bounds a tile).
//
// Per CTA: warps 0..3 and 4..7 softmax groups; warps 8 and 11 (CTA 0 only) issue the P V and the scores of
// the pair; warp 9 requests Q and K (and stores rows), warp 10 V, by TMA, their bytes counted on CTA 0's barriers.
// The host cuts units along the keys where whole units leave SMs idle: such a part leaves unnormalised
// rows with their maximum and sum in a slot of the work area, and prefill_merge_kernel combines them.
// Every wait is bounded; a role that gives up raises its CTA's flag, the other CTA runs out of its own
// waits, tensor memory is freed on every path and the workspace status word is raised.
#include <algorithm>
#include <cstring>
#include <type_traits>
#include <vector>

#include "kpx_once.h"
#include "kpx_prefill_plan.h"
#include "kpx_tma.cuh"

namespace kpx {
namespace {

constexpr int kD = 128, kBS = 16;
constexpr float kLog2e = 1.4426950408889634f;
constexpr int kQItemB = kTile * kD * 2;     // an item's rows: two slabs of 64 elements, 128 bytes a row
constexpr int kQSlabB = kQItemB / 2;
constexpr int kHalfB = kTile * kD;          // a CTA's half of a K or V tile
constexpr int kKSlabB = kHalfB / 2;         // 64 keys x 64 elements
constexpr int kBufs = 3;  // of scores / weights in tensor memory, and of K and of V in shared memory

// A slot holds, for both items of a unit, 128 rows of O, then 128 maxima and 128 sums (floats).
constexpr int64_t kPartItemFloats = int64_t(kTile) * (kD + 2);
constexpr int64_t kPartSlotFloats = 2 * kPartItemFloats;
constexpr int kMaxClusters = 96;
// The work list of a call travels as a kernel parameter: a copy of it on the stream would be a few microseconds on the
// host and on the GPU, keep the launch from being chained, and read a list that is gone when a captured graph is
// replayed.  kInlineUnits is what the 32764 bytes of a kernel's parameters hold beside the rest; longer lists are
// laid into the work area by launches of list_kernel, a parameter full at a time.  All parameters are copied with every launch, so lists of up to kFewUnits
// go in shorter ones (a call of 8/8 heads, 8 x 100 tokens 9.1 us, 9.5 with the long list; 777 tokens, 32/8 15.0 / 15.1).
// Copied / as a parameter, us: 400 units (8/8 heads, 50 x 64 tokens behind 100) 40.3 / 34.9, 512 (32/8, 64 x 16) 34.0 /
// 27.7, (32/32, 16 x 100 behind 50) 46.4 / 40.5, 640 (8/8, 80 x 64 behind 100) 57.7 / 51.3.
constexpr int kFewUnits = 352, kInlineUnits = 960;
template <int kUnits>
struct UnitList {
  uint16_t start[kMaxClusters + 1];  // units start[c] .. start[c + 1] - 1 are cluster c's
  Unit unit[kUnits];
};
constexpr int kListPieces = 2000;  // of 16 bytes, in a parameter of list_kernel
struct ListPieces {
  uint4 piece[kListPieces];
};
struct MergeList {
  Merge merge[kMaxMerges];
};
inline int64_t align256(int64_t x) { return (x + 255) / 256 * 256; }

struct PrefillParams {
  void* out;
  const int32_t* block_table;
  const int32_t* starts;  // nullptr: the list is the parameter
  const Unit* units;
  float* partials;  // slots of kPartSlotFloats floats
  int32_t* status;
  int64_t num_blocks;
  int32_t max_blocks_per_seq, num_q_heads, group_heads, item_tokens;
  int32_t head_groups;   // groups that share a KV head
  uint32_t inv_heads;    // row / group_heads = row * inv_heads >> 16
  float qscale;  // softmax scale * log2(e)
  // Polls a bounded wait makes before it gives up (kWaitLimit), and, for the test of that path
  // only, the CTA one of whose tiles is announced to its barrier but never requested (-1: none;
  // the tile is chosen by the bits above the low 16, see the loader).
  uint32_t wait_limit;
  int32_t withhold_cta;
};

static_assert(sizeof(PrefillParams) + 64 + 4 * sizeof(CUtensorMap) + 64 + sizeof(UnitList<kInlineUnits>) <= 32764,
              "a kernel's parameters");

// ---- PTX wrappers -----------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void fence_async_proxy() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t* slot_in_smem, uint32_t columns) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot_in_smem)),
               "r"(columns)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t base, uint32_t columns) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(columns) : "memory");
}
// every MMA issued so far arrives on the barrier at this address of both CTAs when it has completed
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"(uint16_t(3))
      : "memory");
}
// the same on the barrier of this CTA alone
__device__ __forceinline__ void umma_commit_here(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
// D[tmem] (+)= A[smem] * B[smem] of the pair, 256 x 128 x 16, issued by one thread of CTA 0
__device__ __forceinline__ void umma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]: A is read from each CTA's tensor memory (row = lane, two 16-bit k
// values per 32-bit column, 8 columns per k = 16 step)
__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// the same with CTA 0's rows of D left as they are
__device__ __forceinline__ void umma_ts_cta1(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5, %6, %6, %6, %6}, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0xffffffffu), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld32(uint32_t addr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,"
      "%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(addr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t addr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(addr)
               : "memory");
  tmem_wait_ld();
}
__device__ __forceinline__ void tmem_st8(uint32_t addr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
// Arrive on the barrier that lies at this address in CTA 0.  What it announces is read by the tensor core, not by
// threads of the other CTA: tensor-memory stores ordered by tcgen05.wait::st and the fence before this, tiles that
// the TMA unit has reported on an mbarrier, rows zeroed behind a fence of their own.  With .release.cluster here and
// .acquire.cluster in the waits, an arrival took 1450 clocks and a wait that is already over 350.
__device__ __forceinline__ void arrive_at_cta0(uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %0, 0;\n\t"
      "mbarrier.arrive.shared::cluster.b64 _, [a];\n\t}" ::"r"(smem_u32(bar))
      : "memory");
}
// Tiled TMA loads into this CTA whose bytes are counted on the barrier that lies at this address in CTA 0
__device__ __forceinline__ void tma_load_3d_pair(void* dst, const void* tmap, int c0, int c1, int c2, uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %5, 0;\n\t"
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], "
      "[%1, {%2, %3, %4}], [a];\n\t}" ::"r"(smem_u32(dst)),
      "l"(tmap), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tma_load_4d_pair(void* dst, const void* tmap, int c0, int c1, int c2, int c3,
                                                 uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %6, 0;\n\t"
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], "
      "[%1, {%2, %3, %4, %5}], [a];\n\t}" ::"r"(smem_u32(dst)),
      "l"(tmap), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
      : "memory");
}
// Tiled TMA store from this CTA, and its end: the source has been read / the bytes are written
__device__ __forceinline__ void tma_store_3d(const void* src, const void* tmap, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(tmap), "r"(c0),
               "r"(c1), "r"(c2), "r"(smem_u32(src))
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// Bounded wait of a whole warp that also gives up as soon as another role of the CTA has given up.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, uint32_t limit) {
  bool here = false;
  for (uint32_t i = 0; i < limit; ++i) {
    here = mbar_try_wait(bar, parity);
    if (here) break;
    if (i > 64) {
      __nanosleep(64);
      if ((i & 127) == 0 && *abort_flag) break;
    }
  }
  if (__all_sync(0xffffffffu, here)) return true;
  *abort_flag = 1;
  return false;
}
// true in exactly one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}" : "=r"(pred));
  return pred != 0;
}

// Shared-memory matrix descriptor (sm_100 format): start address, leading / stride byte
// offsets (all >> 4), version 1, 128-byte swizzle.
__device__ __forceinline__ uint64_t smem_desc(const void* ptr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= uint64_t((smem_u32(ptr) & 0x3FFFFu) >> 4);
  d |= uint64_t(lbo_bytes >> 4) << 16;
  d |= uint64_t(sbo_bytes >> 4) << 32;
  d |= uint64_t(1) << 46;  // descriptor version
  d |= uint64_t(2) << 61;  // SWIZZLE_128B
  return d;
}
// Instruction descriptor, kind::f16: fp32 accumulate, A/B = f16 (0) or bf16 (1), M = 256, N = 128.
__host__ __device__ constexpr uint32_t instr_desc(uint32_t format, uint32_t b_mn_major) {
  return (1u << 4) | (format << 7) | (format << 10) | (b_mn_major << 16) | ((128u >> 3) << 17) | ((256u >> 4) << 24);
}

template <typename T>
struct Fmt;
template <>
struct Fmt<__half> { static constexpr uint32_t kCode = 0; };
template <>
struct Fmt<__nv_bfloat16> { static constexpr uint32_t kCode = 1; };

template <typename T>
__device__ __forceinline__ uint32_t pack2(float a, float b);
template <>
__device__ __forceinline__ uint32_t pack2<__half>(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
template <>
__device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

template <typename T>
__device__ __forceinline__ float unpack_lo(uint32_t w);
template <typename T>
__device__ __forceinline__ float unpack_hi(uint32_t w);
template <>
__device__ __forceinline__ float unpack_lo<__nv_bfloat16>(uint32_t w) { return __uint_as_float(w << 16); }
template <>
__device__ __forceinline__ float unpack_hi<__nv_bfloat16>(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
template <>
__device__ __forceinline__ float unpack_lo<__half>(uint32_t w) {
  return __half2float(__ushort_as_half(static_cast<unsigned short>(w & 0xffffu)));
}
template <>
__device__ __forceinline__ float unpack_hi<__half>(uint32_t w) {
  return __half2float(__ushort_as_half(static_cast<unsigned short>(w >> 16)));
}

// A weight enters P V as two 16-bit terms, P = P_hi + P_lo.  One term was measured for both formats
// and fails the output tolerance on short sequences: bf16 (2^-9 relative rounding) by a few 1e-3
// absolute, fp16 (2^-11) within 2e-3 absolute but up to 2.5e-2 relative on outputs near zero (a
// 37-token sequence, where a few weights carry the row and their rounding errors do not average out),
// against a bound of 1e-2.

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// Largest of 32 scores and mx[0..3]; with kMasked, scores of keys e > limit (newer than the query) do not count.
template <bool kMasked>
__device__ __forceinline__ void max32(const uint32_t* r, int limit, float* mx) {
#pragma unroll
  for (int e = 0; e < 32; e += 2) {
    float a = __uint_as_float(r[e]), b = __uint_as_float(r[e + 1]);
    if (kMasked) {
      if (e > limit) a = -INFINITY;
      if (e + 1 > limit) b = -INFINITY;
    }
    mx[(e >> 1) & 3] = max3(mx[(e >> 1) & 3], a, b);
  }
}
// Largest of a row's 128 scores at tS; unless masked, scores 64..127 are left in r.  (Masked tiles are the
// last one or two of a unit: their code is kept short.)
template <bool kMasked>
__device__ __forceinline__ float row_max(uint32_t tS, uint32_t* r, int limit) {
  float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
  if (kMasked) {
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
      tmem_ld32(tS + c * 32, r);
      tmem_wait_ld();
      max32<true>(r, limit - c * 32, mx);
    }
  } else {
    uint32_t lo[64];
    tmem_ld32(tS, lo);
    tmem_ld32(tS + 32, lo + 32);
    tmem_wait_ld();
    tmem_ld32(tS + 64, r);
    tmem_ld32(tS + 96, r + 32);
    max32<false>(lo, 0, mx);
    max32<false>(lo + 32, 0, mx);
    tmem_wait_ld();
    max32<false>(r, 0, mx);
    max32<false>(r + 32, 0, mx);
  }
  return fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
}

// Weights of 16 keys whose scores are in r: p = exp2(s * qscale - m), stored at taddr as P_hi (8 columns, two
// keys each) and at taddr + 16 as P_lo = p - P_hi; lsum += p.  Keys e > limit are masked.
template <typename T, bool kMasked>
__device__ __forceinline__ void weights16(uint32_t taddr, const uint32_t* r, float qscale, float neg_m, int limit,
                                          float2& lsum) {
  const float2 sc = make_float2(qscale, qscale), nm = make_float2(neg_m, neg_m), m1 = make_float2(-1.f, -1.f);
  uint32_t hi[8], lo[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int e = 2 * i;
    const float2 x = __ffma2_rn(make_float2(__uint_as_float(r[e]), __uint_as_float(r[e + 1])), sc, nm);
    float2 w = make_float2(fast_exp2(x.x), fast_exp2(x.y));
    if (kMasked) {
      if (e > limit) w.x = 0.f;
      if (e + 1 > limit) w.y = 0.f;
    }
    lsum = __fadd2_rn(lsum, w);
    const uint32_t hw = pack2<T>(w.x, w.y);
    hi[i] = hw;
    const float2 d = __ffma2_rn(make_float2(unpack_lo<T>(hw), unpack_hi<T>(hw)), m1, w);
    lo[i] = pack2<T>(d.x, d.y);
  }
  tmem_st8(taddr, hi);
  tmem_st8(taddr + 16, lo);
}
// A row's 128 weights over its 128 columns of scores: per 32 columns, keys 0..15 hi, keys 16..31 hi, then lo.
// announce(0) when keys 64..127 are stored, announce(1) when all are.  Unless masked, scores 64..127 are in r.
template <typename T, bool kMasked, typename F>
__device__ __forceinline__ void weights128(uint32_t tS, uint32_t* r, float qscale, float neg_m, int limit, float2& lsum,
                                           F announce) {
  auto slice = [&](int c, const uint32_t* x) {
    weights16<T, kMasked>(tS + c * 32, x, qscale, neg_m, limit - 32 * c, lsum);
    weights16<T, kMasked>(tS + c * 32 + 8, x + 16, qscale, neg_m, limit - 32 * c - 16, lsum);
  };
  if (kMasked) {
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
      const int c = i ^ 2;
      tmem_ld32(tS + c * 32, r);
      tmem_wait_ld();
      slice(c, r);
      if (i & 1) announce(i >> 1);
    }
  } else {
#pragma unroll 1
    for (int i = 0; i < 2; ++i) {  // slices 2 and 3, then 0 and 1
      slice(2 - 2 * i, r);
      if (i == 0) tmem_ld32(tS, r);
      slice(3 - 2 * i, r + 32);
      if (i == 0) tmem_ld32(tS + 32, r + 32);
      announce(i);
      if (i == 0) tmem_wait_ld();
    }
  }
}

// A running maximum is only moved when the tile's maximum exceeds it by more than this (in
// log2 units): weights stay below 2^8, and O is rescaled in far fewer tiles.
constexpr float kLazyMax = 8.f;

constexpr int kPvWarp = 8, kKeyWarp = 9, kValueWarp = 10, kScoresWarp = 11;
// Launched with 168 registers a thread (12 warps x 32 x 168 = 64512); the softmax groups then take 208 and the
// other four warps keep 88: 256 x 208 + 128 x 88 = 64512.  The compiler allots all roles the 168 of the launch and
// spills 84 bytes in the softmax role, between its masked tiles and the rows' way out (none without that role, 12
// without either of the two).
constexpr int kThreads = 384;
struct Bars {
  uint64_t v_here;           // a last tile of V has landed in this CTA
  uint64_t q_ready[2];       // CTA 0: Q of the unit is there in both CTAs
  uint64_t rows_set[2];      // this CTA's rows of the unit lie in its Q's place, or have been written
  uint64_t scores_go[kBufs]; // CTA 0: K is there in both CTAs, the P V that read this buffer has completed
  uint64_t s_full[kBufs];    // scores complete (K may be overwritten)
  uint64_t pv_go[2][kBufs];  // CTA 0: half of the weights from all eight warps; for the first half, V as well
  uint64_t pv_done[kBufs];   // P V complete (V may be overwritten)
  uint64_t o_free;           // CTA 0: the unit's rows have been taken out of O
  uint64_t l_set[2][4];  // the group without the unit's last tile has left its sums; two units in turn
};
struct Small {
  Bars bars;
  uint32_t tmem;
  int32_t abort;
  // Of each softmax group and row: the running maximum after the group's tile (low word) and that tile's number
  // (high word), in one store, so that the other group needs one look and no barrier.
  volatile unsigned long long m[2][kTile];
  float2 l[2][kTile];  // (sum, the maximum it stands for); two units in turn
};
constexpr int kSmemBytes = 1024 /*align slack*/ + 2 * kQItemB + 2 * kBufs * kHalfB + int(sizeof(Small));
static_assert(kSmemBytes <= 227 * 1024, "shared memory of an SM");

// A ring of kN barriers walked one use at a time: index and phase parity.
template <int kN>
struct Ring {
  int at = 0;
  uint32_t parity = 0;
  __device__ __forceinline__ void next() {
    if (++at == kN) {
      at = 0;
      parity ^= 1u;
    }
  }
};

template <typename T, int kUnits>
__global__ void __launch_bounds__(kThreads, 1)
    prefill_tc_kernel(const PrefillParams p, const __grid_constant__ CUtensorMap map_q,
                      const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                      const __grid_constant__ CUtensorMap map_out,
                      const __grid_constant__ UnitList<kUnits> list) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* sQ = smem;                     // this CTA's item of two units in turn
  uint8_t* sK = sQ + 2 * kQItemB;         // keys 64 r .. 64 r + 63 of a tile: two slabs of 64 elements
  uint8_t* sV = sK + kBufs * kHalfB;    // elements 64 r .. 64 r + 63 of a tile's 128 keys
  Small& sm = *reinterpret_cast<Small*>(sV + kBufs * kHalfB);
  Bars& bars = sm.bars;
  volatile int* abort_flag = &sm.abort;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = int(cluster_rank());
  if (tid == 0) {
    auto init = [](uint64_t* b, int n, uint32_t count) {
      for (int i = 0; i < n; ++i) mbar_init(b + i, count);
    };
    init(&bars.v_here, 1, 1);
    init(bars.q_ready, 2, 1);
    init(bars.rows_set, 2, 4);
    init(bars.scores_go, kBufs, 2);
    init(bars.s_full, kBufs, 1);
    init(bars.pv_go[0], kBufs, 10);
    init(bars.pv_go[1], kBufs, 8);
    init(bars.pv_done, kBufs, 1);
    init(&bars.o_free, 1, 8);
    init(&bars.l_set[0][0], 8, 1);
    for (int i = 0; i < kBufs; ++i) mbar_arrive(&bars.scores_go[i]);  // no P V before the first
    sm.abort = 0;
    mbar_fence_init();
  }
  if (tid < kTile) sm.m[0][tid] = sm.m[1][tid] = ~0ull;  // (the number of no tile)
  if (warp == kPvWarp) tmem_alloc(&sm.tmem, 512);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the other CTA's barriers are there too
  tc_fence_after();
  const uint32_t tmem = sm.tmem;  // columns: three score / weight buffers, then O
  const int64_t after_wait = grid_wait();
  grid_release();

  const int cluster = int(blockIdx.x >> 1);
  const bool inline_list = p.starts == nullptr;
  const int32_t* starts = p.starts + after_wait;
  const Unit* units = p.units + after_wait;
  const int u_first = inline_list ? int(list.start[cluster]) : starts[cluster];
  const int u_end = inline_list ? int(list.start[cluster + 1]) : starts[cluster + 1];
  auto unit_at = [&](int u) {
    if (inline_list) return list.unit[u];
    return units[u];
  };
  // tokens of this CTA's item, and its first token within the unit
  auto my_tokens = [&](const Unit& d, int& first) {
    const bool two = d.ntok > p.item_tokens;
    first = rank == 1 && two ? p.item_tokens : 0;
    if (rank == 0) return two ? p.item_tokens : 0;
    return d.ntok - first;
  };
  auto wait = [&](uint64_t& bar, uint32_t parity) { return warp_wait(&bar, parity, abort_flag, p.wait_limit); };

  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    if (warp == kKeyWarp || warp == kValueWarp) {
      // ===== loaders: TMA boxes of Q and of this CTA's half of K, or of this CTA's half of V, through the block
      // table.  One lane issues, the boxes of a tile unrolled: asked for by a lane each, they took 100 clocks apiece =====
      const bool values = warp == kValueWarp;
      constexpr int kTileBlocks = kTile / kBS;
      Ring<kBufs> buf;
      Ring<2> qs;
      bool ok = true, again = false;  // the buffers have been filled once
      uint32_t last_parity = 0;
      // the rows of unit u, once they lie in place q of Q: an item of all its tokens is stored from here
      auto whole = [&](const Unit& d, int& first) { return d.part < 0 && my_tokens(d, first) == p.item_tokens; };
      auto rows_out = [&](int u, int q, uint32_t parity) {
        if (!wait(bars.rows_set[q], parity)) return false;
        const Unit d = unit_at(u);
        int first;
        if (whole(d, first) && lane == 0) {
          const uint8_t* src = sQ + q * kQItemB;
          tma_store_3d(src, &map_out, 0, d.group * p.group_heads, d.tok0 + first);
          tma_store_3d(src + kQSlabB, &map_out, 64, d.group * p.group_heads, d.tok0 + first);
          tma_store_commit();
          tma_store_wait_read();
        }
        __syncwarp();
        return true;
      };
      for (int u = u_first; u < u_end && ok; ++u) {
        const Unit d = unit_at(u);
        if (!values) {
          if (u - u_first >= 2) ok = rows_out(u - 2, qs.at, qs.parity ^ 1u);
          if (!ok) break;
          int first;
          const int mine = my_tokens(d, first);
          const uint32_t item_bytes = uint32_t(p.item_tokens * p.group_heads) * 256u;
          if (elect_one()) {
            uint64_t* bar = &bars.q_ready[qs.at];
            if (rank == 0) mbar_arrive_expect_tx(bar, mine > 0 ? 2 * item_bytes : item_bytes);
            if (mine > 0) {
              uint8_t* dst = sQ + qs.at * kQItemB;
              tma_load_3d_pair(dst, &map_q, 0, d.group * p.group_heads, d.tok0 + first, bar);
              tma_load_3d_pair(dst + kQSlabB, &map_q, 64, d.group * p.group_heads, d.tok0 + first, bar);
            }
          }
          __syncwarp();
          qs.next();
        }
        const int32_t* table = p.block_table + int64_t(d.seq) * p.max_blocks_per_seq + after_wait;
        const int kvh = d.group / p.head_groups;
        const int kv_len = d.pos0 + d.ntok;
        const int blocks = (kv_len + kBS - 1) / kBS;
        auto load_id = [&](int jt) {  // lanes 0..7: the tile's blocks
          const int i = jt * kTileBlocks + lane;
          return lane < kTileBlocks && i < blocks && jt < d.tile1 ? __ldg(table + i) : 0;
        };
        int next_id = load_id(d.tile0);
        for (int jt = d.tile0; jt < d.tile1; ++jt) {
          int id = next_id;
          next_id = load_id(jt + 1);
          if (id < 0 || (p.num_blocks > 0 && id >= p.num_blocks)) {
            atomicMax(p.status, KPX_ERR_INVALID_ARGUMENT);
            id = 0;
          }
          __syncwarp();
          const int left = kv_len - jt * kTile;  // tokens from the start of this tile
          const int nblk = min(kTileBlocks, blocks - jt * kTileBlocks);
          // test knob: CTA (withhold_cta & 0xffff) never requests one tile that has been announced:
          // (withhold_cta >> 16) = 0: K of its first tile, 1: V of its first tile, 2: K of its second tile
          const int what = p.withhold_cta >> 16;
          const bool fault = p.withhold_cta >= 0 && int(blockIdx.x) == (p.withhold_cta & 0xffff) && u == u_first &&
                             jt == d.tile0 + (what == 2 ? 1 : 0) && values == (what == 1);
          // A barrier is waited for only by a role that its next phase cannot do without: one that it can outrun would
          // find the parity turned twice and wait for ever.  CTA 1 has no keys in a last tile of up to 64, whose
          // scores CTA 0's keys alone let go.  (Without this wait it is never more than a phase ahead: only the last
          // tile of a unit is such a tile, and a unit is begun when the rows of the one before the last have left.)
          const int here = nblk - rank * (kTileBlocks / 2);  // blocks of this CTA's half of K that exist
          if (again && (values || here > 0)) ok = wait(values ? bars.pv_done[buf.at] : bars.s_full[buf.at], buf.parity ^ 1u);
          if (!ok) break;
          if (!values) {
            int blk[kTileBlocks / 2];
#pragma unroll
            for (int i = 0; i < kTileBlocks / 2; ++i) blk[i] = __shfl_sync(0xffffffffu, id, rank * (kTileBlocks / 2) + i);
            if (elect_one()) {
              uint64_t* bar = &bars.scores_go[buf.at];
              if (rank == 0) mbar_arrive_expect_tx(bar, uint32_t(nblk) * (kBS * kD * 2));
              uint8_t* dst = sK + buf.at * kHalfB;
#pragma unroll
              for (int i = 0; i < kTileBlocks / 2; ++i)
                if (i < here && !fault) {
                  tma_load_4d_pair(dst + i * (kBS * 128), &map_k, 0, 0, kvh, blk[i], bar);
                  tma_load_4d_pair(dst + kKSlabB + i * (kBS * 128), &map_k, 64, 0, kvh, blk[i], bar);
                }
            }
          } else {
            int blk[kTileBlocks];
#pragma unroll
            for (int i = 0; i < kTileBlocks; ++i) blk[i] = __shfl_sync(0xffffffffu, id, i);
            uint8_t* dst = sV + buf.at * kHalfB;
            uint64_t* go = &bars.pv_go[0][buf.at];
            if (left >= kTile) {
              if (elect_one()) {
                if (rank == 0) mbar_arrive_expect_tx(go, kTileBlocks * (kBS * kD * 2));
                else arrive_at_cta0(go);
#pragma unroll
                for (int i = 0; i < kTileBlocks; ++i)
                  if (!fault) tma_load_4d_pair(dst + i * (kBS * 128), &map_v, rank * 64, 0, kvh, blk[i], go);
              }
            } else {
              // V rows past the newest token must be zero (a weight of 0 times pool garbage must stay
              // 0); the last box covers some of these rows, so they are zeroed when the boxes have landed
              if (elect_one()) {
                mbar_arrive_expect_tx(&bars.v_here, uint32_t(nblk) * (kBS * 128));
#pragma unroll
                for (int i = 0; i < kTileBlocks; ++i)
                  if (i < nblk && !fault) tma_load_4d(dst + i * (kBS * 128), &map_v, rank * 64, 0, kvh, blk[i], &bars.v_here);
              }
              __syncwarp();
              ok = wait(bars.v_here, last_parity);
              if (!ok) break;
              last_parity ^= 1u;
              for (int i = left * 8 + lane; i < kTile * 8; i += 32)  // 16-byte pieces of rows left..127
                *reinterpret_cast<uint4*>(dst + i * 16) = make_uint4(0, 0, 0, 0);
              fence_async_proxy();
              asm volatile("fence.acq_rel.cluster;" ::: "memory");
              __syncwarp();
              if (lane == 0) arrive_at_cta0(go);
            }
          }
          __syncwarp();
          buf.next();
          again = again || buf.at == 0;
        }
      }
      if (!values) {  // the rows of the last two units
        for (int u = max(u_first, u_end - 2); u < u_end && ok; ++u) {
          const int k = u - u_first;
          ok = rows_out(u, k & 1, uint32_t(k >> 1) & 1u);
        }
        if (lane == 0) tma_store_wait();
        __syncwarp();
      }
    } else if (warp == kScoresWarp && rank == 0) {
      // ===== S = Q K^T of the pair, tile by tile: 8 steps of k = 16 over d = 128.  The whole warp walks the
      // schedule in step and one elected lane issues, so that descriptors and addresses stay in uniform
      // registers =====
      constexpr uint32_t kIdesc = instr_desc(Fmt<T>::kCode, 0);
      const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
      // descriptors of the operand bases; the k steps add to the 16-byte-unit address field
      const uint64_t dq0 = smem_desc(sQ, 0, 1024), dk0 = smem_desc(sK, 0, 1024);
      Ring<kBufs> buf;
      Ring<2> qs;
      bool ok = true;
      for (int u = u_first; u < u_end && ok; ++u) {
        const Unit d = unit_at(u);
        ok = wait(bars.q_ready[qs.at], qs.parity);
        for (int jt = d.tile0; jt < d.tile1 && ok; ++jt) {
          ok = wait(bars.scores_go[buf.at], buf.parity);
          if (!ok) break;
          tc_fence_after();
          const uint64_t a = dq0 + uint64_t(qs.at * (kQItemB >> 4)), b = dk0 + uint64_t(buf.at * (kHalfB >> 4));
          if (elect_one()) {
#pragma unroll
            for (int s = 0; s < 8; ++s)
              umma_ss(tm + buf.at * kTile, a + uint64_t(((s >> 2) * kQSlabB + (s & 3) * 32) >> 4),
                      b + uint64_t(((s >> 2) * kKSlabB + (s & 3) * 32) >> 4), kIdesc, s > 0);
            umma_commit(&bars.s_full[buf.at]);
          }
          __syncwarp();
          buf.next();
        }
        qs.next();
      }
    } else if (warp == kPvWarp && rank == 0) {
      // ===== O += P_hi V + P_lo V of the pair: A = P from tensor memory, B = V: key rows 16 s .., d along MN.
      // The softmax threads are through with keys 64..127 (steps 4..7) first =====
      constexpr uint32_t kIdesc = instr_desc(Fmt<T>::kCode, 1);
      const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0), tO = tm + kBufs * kTile;
      const uint64_t dv0 = smem_desc(sV, kHalfB, 1024);
      Ring<kBufs> buf;
      uint32_t o_parity = 0;
      bool ok = true;
      for (int u = u_first; u < u_end && ok; ++u) {
        const Unit d = unit_at(u);
        // from this tile on, every key is newer than item 0's rows: they are left alone, whatever V holds
        const int tiles0 = d.ntok > p.item_tokens ? (d.pos0 + p.item_tokens - 1) / kTile + 1 : 1 << 30;
        if (u > u_first) {  // the rows of the unit before have been taken out of O
          ok = wait(bars.o_free, o_parity);
          o_parity ^= 1u;
        }
        for (int jt = d.tile0; jt < d.tile1 && ok; ++jt) {
          const uint64_t b = dv0 + uint64_t(buf.at * (kHalfB >> 4));
          const uint32_t tP = tm + buf.at * kTile;
          const bool both = jt < tiles0 || jt == d.tile0;
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            ok = ok && wait(bars.pv_go[half][buf.at], buf.parity);
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
              const int s0 = half == 0 ? 4 : 0;
              if (both) {
#pragma unroll
                for (int s = s0; s < s0 + 4; ++s) {
                  const uint32_t a = tP + (s >> 1) * 32 + (s & 1) * 8;
                  umma_ts(tO, a, b + uint64_t((s * 16 * 128) >> 4), kIdesc, (jt > d.tile0 || half > 0 || s > s0) ? 1u : 0u);
                  umma_ts(tO, a + 16, b + uint64_t((s * 16 * 128) >> 4), kIdesc, 1u);
                }
              } else {
#pragma unroll
                for (int s = s0; s < s0 + 4; ++s) {
                  const uint32_t a = tP + (s >> 1) * 32 + (s & 1) * 8;
                  umma_ts_cta1(tO, a, b + uint64_t((s * 16 * 128) >> 4), kIdesc, 1u);
                  umma_ts_cta1(tO, a + 16, b + uint64_t((s * 16 * 128) >> 4), kIdesc, 1u);
                }
              }
              if (half == 1) {
                umma_commit_here(&bars.scores_go[buf.at]);
                umma_commit(&bars.pv_done[buf.at]);
              }
            }
            __syncwarp();
          }
          buf.next();
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    // ===== softmax: group g takes the tiles whose number in the cluster's sequence is g modulo 2; warp w
    // of either group has query rows (= TMEM lanes) 32 w .. 32 w + 31, a thread one row =====
    const int g = warp >> 2, w = warp & 3, row = w * 32 + lane;
    const uint32_t lane_addr = uint32_t(w * 32) << 16;
    const uint32_t tO = tmem + kBufs * kTile + lane_addr;
    const int row_token = int((uint32_t(row) * p.inv_heads) >> 16);
    int seq0 = 0;            // number of the unit's first tile
    uint32_t l_count = 0;    // units so far in which both groups had tiles
    bool ok = true;
    for (int u = u_first; u < u_end && ok; ++u) {
      const Unit d = unit_at(u);
      const int ntiles = d.tile1 - d.tile0;
      int first;
      const int mine = my_tokens(d, first);
      const int my_pos = d.pos0 + first + row_token;
      float m = -INFINITY;      // running maximum (scaled scores), moved lazily
      float2 l = {0.f, 0.f};    // sum of this group's weights, as an even/odd pair
      for (int j = (seq0 ^ g) & 1; j < ntiles && ok; j += 2) {
        const int n = seq0 + j;  // the tile's number
        const int use = n / kBufs, buf = n - use * kBufs;
        const uint32_t tS = tmem + buf * kTile + lane_addr;
        // the maximum after the tile before, which the other group had: as a rule it is there by now
        unsigned long long before = sm.m[g ^ 1][row];
        ok = wait(bars.s_full[buf], uint32_t(use & 1));
        if (!ok) break;
        tc_fence_after();
        uint32_t r[64];
        const int limit = my_pos - (d.tile0 + j) * kTile;  // keys e > limit are newer than the query
        const bool diag = (d.tile0 + j) * kTile + kTile - 1 > d.pos0 + first;  // some row is masked in this tile
        float m_tile = -INFINITY;
        if (mine > 0) m_tile = (diag ? row_max<true>(tS, r, limit) : row_max<false>(tS, r, 0)) * p.qscale;
        if (n > 0) {
          bool there = int(before >> 32) == n - 1;
          for (uint32_t i = 0; !__all_sync(0xffffffffu, there); ++i) {
            before = sm.m[g ^ 1][row];
            there = int(before >> 32) == n - 1;
            if (i >= p.wait_limit || ((i & 127) == 127 && *abort_flag)) ok = false;
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
          }
          if (!ok) {
            *abort_flag = 1;
            break;
          }
        }
        const float m_before = j > 0 ? __uint_as_float(uint32_t(before)) : -INFINITY;
        float m_now = m_before;
        if (m_tile > m_before + kLazyMax || m_before == -INFINITY)  // (-inf + 8 is -inf: the first tile always moves it)
          m_now = (m_tile == -INFINITY) ? 0.f : m_tile;
        sm.m[g][row] = (static_cast<unsigned long long>(n) << 32) | __float_as_uint(m_now);
        auto announce = [&](int half) {
          tmem_wait_st();  // this warp's weights (and a rescaled O) are in tensor memory
          tc_fence_before();
          __syncwarp();
          if (lane == 0) arrive_at_cta0(&bars.pv_go[half][buf]);
        };
        if (mine > 0) {
          if (m_now != m) {
            const float a = fast_exp2(m - m_now);
            l.x *= a;
            l.y *= a;
            m = m_now;
          }
          if (j > 0 && __any_sync(0xffffffffu, m_now != m_before)) {
            // O stands for the maximum before: rescale it once the P V of the tile before has completed
            // (this tile's is not issued before this warp has announced its weights)
            const int use1 = (n - 1) / kBufs, buf1 = n - 1 - use1 * kBufs;
            ok = wait(bars.pv_done[buf1], uint32_t(use1 & 1));
            if (!ok) break;
            tc_fence_after();
            const float a = fast_exp2(m_before - m_now);
#pragma unroll 1
            for (int c = 0; c < kD / 8; ++c) {
              uint32_t o[8];
              tmem_ld8(tO + c * 8, o);
#pragma unroll
              for (int e = 0; e < 8; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * a);
              tmem_st8(tO + c * 8, o);
            }
          }
          if (diag) weights128<T, true>(tS, r, p.qscale, -m_now, limit, l, announce);
          else weights128<T, false>(tS, r, p.qscale, -m_now, 0, l, announce);
        } else {
          announce(0);
          announce(1);
        }
      }
      if (!ok) break;
      const int last = seq0 + ntiles - 1;
      float2* l_pair = sm.l[l_count & 1];
      uint64_t& l_bar = bars.l_set[l_count & 1][w];
      if ((last & 1) != g) {  // the other group writes the rows
        if (ntiles > 1) {
          l_pair[row] = make_float2(l.x + l.y, m);
          __syncwarp();
          if (lane == 0) mbar_arrive(&l_bar);
        }
      } else {
        float l_row = l.x + l.y;
        if (ntiles > 1) {
          ok = wait(l_bar, (l_count >> 1) & 1);
          if (!ok) break;
          const float2 other = l_pair[row];
          l_row = fmaf(other.x, fast_exp2(other.y - m), l_row);
        }
        const int use = last / kBufs, buf = last - use * kBufs;
        ok = wait(bars.pv_done[buf], uint32_t(use & 1));
        if (!ok) break;
        tc_fence_after();
        // A thread holds a row; stored from here, a warp's stores would touch 32 rows each.  The rows go to the
        // place of the unit's Q (its last scores are complete), laid out as Q was: two slabs of 64 elements, a row
        // 128 bytes, its 16-byte chunks rotated by the row.  The loader stores an item of all its tokens from there;
        // the others are copied here, 16 lanes a row.
        const int slot = (u - u_first) & 1;
        uint8_t* stage = sQ + slot * kQItemB;
        const int rows_here = mine * p.group_heads;
        const int c16 = lane & 15, r2 = lane >> 4;
        auto taken = [&]() {  // O is in registers: the next unit's products may go there
          tc_fence_before();
          __syncwarp();
          if (lane == 0) arrive_at_cta0(&bars.o_free);
        };
        auto chunk = [&](int r, int c) {
          return reinterpret_cast<uint4*>(stage + (c >> 3) * kQSlabB + r * 128 + (((c ^ r) & 7) << 4));
        };
        if (d.part < 0) {
          const float inv = l_row > 0.f ? 1.f / l_row : 0.f;
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            uint32_t r[64];
            tmem_ld32(tO + hf * 64, r);
            tmem_ld32(tO + hf * 64 + 32, r + 32);
            tmem_wait_ld();
            if (hf == 1) taken();
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              auto two = [&](int e) { return pack2<T>(__uint_as_float(r[8 * c + e]) * inv, __uint_as_float(r[8 * c + e + 1]) * inv); };
              *chunk(row, 8 * hf + c) = make_uint4(two(0), two(2), two(4), two(6));
            }
          }
          if (mine == p.item_tokens) {
            fence_async_proxy();
          } else {
            __syncwarp();
            uint8_t* obase = static_cast<uint8_t*>(p.out) +
                             (int64_t(d.tok0 + first) * p.num_q_heads + int64_t(d.group) * p.group_heads) * (kD * 2) + c16 * 16;
#pragma unroll 2
            for (int i = 0; i < 16; ++i) {
              const int rr = w * 32 + 2 * i + r2;
              const int tok = int((uint32_t(rr) * p.inv_heads) >> 16);
              if (rr < rows_here)
                *reinterpret_cast<uint4*>(obase + (int64_t(tok) * p.num_q_heads + (rr - tok * p.group_heads)) * (kD * 2)) = *chunk(rr, c16);
            }
            fence_async_proxy();  // the place is the loader's again
          }
        } else {  // unnormalised, 64 columns at a time
          float* part_rows = p.partials + int64_t(d.part) * kPartSlotFloats + rank * kPartItemFloats;
#pragma unroll 1
          for (int hf = 0; hf < 2; ++hf) {
            uint32_t r[64];
            tmem_ld32(tO + hf * 64, r);
            tmem_ld32(tO + hf * 64 + 32, r + 32);
            tmem_wait_ld();
            if (hf == 1) taken();
#pragma unroll
            for (int c = 0; c < 16; ++c) *chunk(row, c) = make_uint4(r[4 * c], r[4 * c + 1], r[4 * c + 2], r[4 * c + 3]);
            __syncwarp();
#pragma unroll 4
            for (int i = 0; i < 16; ++i) {
              const int rr = w * 32 + 2 * i + r2;
              if (rr < rows_here) *reinterpret_cast<uint4*>(part_rows + rr * kD + hf * 64 + c16 * 4) = *chunk(rr, c16);
            }
            __syncwarp();
          }
          if (row < rows_here) {
            part_rows[kTile * kD + row] = m;
            part_rows[kTile * kD + kTile + row] = l_row;
          }
          fence_async_proxy();
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars.rows_set[slot]);
      }
      if (ntiles > 1) ++l_count;
      seq0 += ntiles;
    }
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {  // let copies and products in flight come to their end
    if (tid == 0) atomicMax(p.status, KPX_ERR_DEVICE_TIMEOUT);
    for (int k = 0; k < 64; ++k) __nanosleep(1000);
  }
  cluster_sync_all();  // nobody leaves while the other CTA's barriers or shared memory are in use
  if (warp == kPvWarp) tmem_dealloc(tmem, 512);
}

// Output rows of a unit whose keys were cut into parts: out = sum_p 2^(m_p - M) O_p / sum_p 2^(m_p - M) l_p.
// blockIdx.x = unit, blockIdx.y = item and group of 8 rows; a warp per row, four elements a lane.  Bound by the
// chain of loads: maxima and sums in one trip, then all parts' rows in one.
constexpr int kMergeWarps = 8;
template <typename T>
__global__ void __launch_bounds__(32 * kMergeWarps)
    prefill_merge_kernel(T* __restrict__ out, const float* __restrict__ partials, int num_q_heads, int group_heads,
                         int item_tokens, const __grid_constant__ MergeList list) {
  const int64_t after_wait = grid_wait();
  grid_release();
  partials += after_wait;
  const Merge md = list.merge[blockIdx.x];
  const int item = int(blockIdx.y) / (kTile / kMergeWarps), lane = threadIdx.x & 31;
  const int row = int(blockIdx.y) % (kTile / kMergeWarps) * kMergeWarps + int(threadIdx.x >> 5);
  const bool two = md.ntok > item_tokens;
  const int first = item == 1 && two ? item_tokens : 0;
  const int tokens = item == 0 ? (two ? item_tokens : 0) : md.ntok - first;
  if (row >= tokens * group_heads) return;
  const float* base = partials + md.slot0 * kPartSlotFloats + item * kPartItemFloats;
  float4 o[kMaxParts];
#pragma unroll
  for (int q = 0; q < kMaxParts; ++q)
    o[q] = *reinterpret_cast<const float4*>(base + (q < md.parts ? q : 0) * kPartSlotFloats + int64_t(row) * kD + 4 * lane);
  // the parts' maxima and sums, one a lane.  A part in which the row saw no key (sum 0) carries a
  // placeholder maximum and does not count.
  float mp = -INFINITY, lp = 0.f;
  if (lane < md.parts) {
    mp = base[lane * kPartSlotFloats + kTile * kD + row];
    lp = base[lane * kPartSlotFloats + kTile * kD + kTile + row];
    if (!(lp > 0.f)) mp = -INFINITY;
  }
  float M = mp;
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, s));
  const float weight = lp > 0.f ? fast_exp2(mp - M) : 0.f;
  float L = 0.f;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int q = 0; q < kMaxParts; ++q) {
    const float w = __shfl_sync(0xffffffffu, weight, q), lq = __shfl_sync(0xffffffffu, lp, q);
    if (lq > 0.f) {  // (a part that does not count may hold anything, NaN included)
      acc.x = fmaf(o[q].x, w, acc.x);
      acc.y = fmaf(o[q].y, w, acc.y);
      acc.z = fmaf(o[q].z, w, acc.z);
      acc.w = fmaf(o[q].w, w, acc.w);
      L = fmaf(lq, w, L);
    }
  }
  const float inv = L > 0.f ? 1.f / L : 0.f;
  const int tok = row / group_heads;
  T* orow = out + (int64_t(md.tok0 + first + tok) * num_q_heads + int64_t(md.group) * group_heads + (row - tok * group_heads)) * kD;
  *reinterpret_cast<uint2*>(orow + 4 * lane) =
      make_uint2(pack2<T>(acc.x * inv, acc.y * inv), pack2<T>(acc.z * inv, acc.w * inv));
}

// A stretch of a work list that is too long for the kernel's own parameters, into the work area.
constexpr int kListThreads = 128;
__global__ void __launch_bounds__(kListThreads)
    list_kernel(uint4* __restrict__ dst, int count, const __grid_constant__ ListPieces list) {
  const int64_t after_wait = grid_wait();
  grid_release();
  const int i = int(blockIdx.x) * kListThreads + int(threadIdx.x);
  if (i < count) dst[i + after_wait] = list.piece[i];
}

struct Ready {};
template <typename K>
int prepare_kernel(K kernel, PerDevice<Ready>& done) {
  int dev = 0;
  KPX_CUDA_TRY(cudaGetDevice(&dev));
  int rc = KPX_OK;
  const Ready* r = done.get(dev, [&](Ready&) {
    rc = cuda_status(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
    return rc == KPX_OK;
  });
  return r ? KPX_OK : (rc != KPX_OK ? rc : KPX_ERR_CUDA);
}

}  // namespace

// -1: cut where it pays (default); 0: never; 2..4: always, into that many parts (tests).
int g_prefill_split = -1;
// Test-only: polls before a bounded wait gives up, and the CTA one of whose tiles never comes.
uint32_t g_prefill_wait_limit = kWaitLimit;
int g_prefill_withhold_cta = -1;

// Host side: work list, tensor maps, launch.  Returns KPX_ERR_UNIMPLEMENTED when the layout, dtype or scale
// is outside this path so that the caller can fall back to the streaming path.
int prefill_tc(void* out, const void* q, const void* k_pool, const void* v_pool, const kpx_kv_layout* layout,
               const int32_t* block_table, int32_t max_blocks_per_seq, const int32_t* cu_q_lens_host,
               const int32_t* start_pos_host, int32_t batch, int32_t num_q_heads, float scale, void* tile_area,
               int64_t tile_area_bytes, int32_t* status, cudaStream_t stream) {
  const int kv_heads = layout->num_kv_heads, kv_mul = num_q_heads / kv_heads;
  if (layout->dtype == KPX_F32 || layout->head_size != kD || layout->block_size != kBS || !block_table ||
      !(scale > 0.f))  // the row maximum is taken before scaling
    return KPX_ERR_UNIMPLEMENTED;
  // TMA: 16-byte aligned bases (strides are multiples of 16 bytes in every valid layout)
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k_pool) | reinterpret_cast<uintptr_t>(v_pool)) & 15)
    return KPX_ERR_UNIMPLEMENTED;
  const int32_t total_q = cu_q_lens_host[batch];
  int group_heads = std::min(kv_mul, kTile);
  while (kv_mul % group_heads) --group_heads;
  const int head_groups = kv_mul / group_heads, groups = kv_heads * head_groups;
  const int item_tokens = kTile / group_heads;
  const int clusters = std::min(std::max(device_info().sm_count / 2, 1), kMaxClusters);
  std::vector<Unit> units = whole_units(cu_q_lens_host, start_pos_host, batch, groups, item_tokens);
  if (units.empty()) return KPX_OK;
  const WorkList work = plan_units(std::move(units), clusters, g_prefill_split);
  // clusters with work
  int used = clusters;
  while (used > 1 && work.start[size_t(used)] == work.start[size_t(used) - 1]) --used;
  // layout of the area: [starts][units] (lists that do not fit a parameter), [part slots]
  const bool inline_list = int(work.units.size()) <= kInlineUnits;
  const int64_t start_bytes = inline_list ? 0 : align256(int64_t(clusters + 1) * 4);
  const int64_t unit_bytes = inline_list ? 0 : align256(int64_t(work.units.size()) * int64_t(sizeof(Unit)));
  const int64_t slot_bytes = work.merges.empty() ? 0 : int64_t(kMaxPartSlots) * kPartSlotFloats * int64_t(sizeof(float));
  if (start_bytes + unit_bytes + slot_bytes > tile_area_bytes) return KPX_ERR_WORKSPACE_TOO_SMALL;

  CUtensorMap map_q, map_k, map_v, map_out;
  {
    // Q and the output [total_q][heads][128]: box = an item's tokens x the group's heads x 64 elements
    const cuuint64_t dims[3] = {cuuint64_t(kD), cuuint64_t(num_q_heads), cuuint64_t(total_q)};
    const cuuint64_t strides[2] = {cuuint64_t(kD) * 2, cuuint64_t(num_q_heads) * kD * 2};
    const cuuint32_t box[3] = {64, cuuint32_t(group_heads), cuuint32_t(item_tokens)};
    if (!make_map(&map_q, layout->dtype, q, 3, dims, strides, box) ||
        !make_map(&map_out, layout->dtype, out, 3, dims, strides, box))
      return KPX_ERR_UNIMPLEMENTED;
  }
  {
    // pool [blocks][kv heads][16 tokens][128] by its strides: box = one (block, head) tile x 64 elements
    const cuuint64_t nblocks = layout->num_blocks > 0 ? cuuint64_t(layout->num_blocks) : (cuuint64_t(1) << 24);
    const cuuint64_t dims[4] = {cuuint64_t(kD), cuuint64_t(kBS), cuuint64_t(kv_heads), nblocks};
    const cuuint64_t strides[3] = {cuuint64_t(layout->token_stride) * 2, cuuint64_t(layout->head_stride) * 2,
                                   cuuint64_t(layout->block_stride) * 2};
    const cuuint32_t box[4] = {64, cuuint32_t(kBS), 1, 1};
    if (!make_map(&map_k, layout->dtype, k_pool, 4, dims, strides, box) ||
        !make_map(&map_v, layout->dtype, v_pool, 4, dims, strides, box))
      return KPX_ERR_UNIMPLEMENTED;
  }
  uint8_t* area = static_cast<uint8_t*>(tile_area);
  PrefillParams p;
  if (inline_list) {
    p.starts = nullptr;
    p.units = nullptr;
  } else {
    std::vector<uint4> image(size_t(start_bytes + unit_bytes) / sizeof(uint4));
    std::memcpy(image.data(), work.start.data(), work.start.size() * 4);
    Unit* units_at = reinterpret_cast<Unit*>(reinterpret_cast<uint8_t*>(image.data()) + start_bytes);
    for (size_t i = 0; i < work.units.size(); ++i) std::memcpy(units_at + i, &work.units[size_t(work.order[i])], sizeof(Unit));
    ListPieces pieces;
    for (size_t at = 0; at < image.size(); at += kListPieces) {
      const size_t count = std::min(image.size() - at, size_t(kListPieces));
      std::memcpy(pieces.piece, image.data() + at, count * sizeof(uint4));
      const int rc = launch_chained(list_kernel, dim3(unsigned((count + kListThreads - 1) / kListThreads)), dim3(kListThreads), 0,
                                    stream, reinterpret_cast<uint4*>(area) + at, int(count), pieces);
      if (rc != KPX_OK) return rc;
    }
    p.starts = reinterpret_cast<const int32_t*>(area);
    p.units = reinterpret_cast<const Unit*>(area + start_bytes);
  }
  p.partials = reinterpret_cast<float*>(area + start_bytes + unit_bytes);
  p.out = out;
  p.block_table = block_table;
  p.status = status;
  p.num_blocks = layout->num_blocks;
  p.max_blocks_per_seq = max_blocks_per_seq;
  p.num_q_heads = num_q_heads;
  p.group_heads = group_heads;
  p.head_groups = head_groups;
  p.item_tokens = item_tokens;
  p.inv_heads = uint32_t(65536 / group_heads + 1);
  p.qscale = scale * kLog2e;
  p.wait_limit = g_prefill_wait_limit;
  p.withhold_cta = g_prefill_withhold_cta;
  auto launch = [&](auto type, auto capacity) -> int {
    constexpr int kUnits = decltype(capacity)::value;
    constexpr auto kernel = prefill_tc_kernel<decltype(type), kUnits>;
    static PerDevice<Ready> ready;
    const int rc = prepare_kernel(kernel, ready);
    if (rc != KPX_OK) return rc;
    UnitList<kUnits> list;
    if (inline_list) {
      for (int c = 0; c <= clusters; ++c) list.start[c] = uint16_t(work.start[size_t(c)]);
      for (size_t i = 0; i < work.units.size(); ++i) list.unit[i] = work.units[size_t(work.order[i])];
    }
    return launch_chained_cluster(kernel, dim3(unsigned(2 * used)), dim3(kThreads), kSmemBytes, 2, stream, p, map_q, map_k,
                                  map_v, map_out, list);
  };
  const bool few = !inline_list || int(work.units.size()) <= kFewUnits;
  auto launch_as = [&](auto type) {
    return few ? launch(type, std::integral_constant<int, kFewUnits>()) : launch(type, std::integral_constant<int, kInlineUnits>());
  };
  const int rc = layout->dtype == KPX_F16 ? launch_as(__half()) : launch_as(__nv_bfloat16());
  if (rc != KPX_OK || work.merges.empty()) return rc;
  MergeList mlist;
  std::copy(work.merges.begin(), work.merges.end(), mlist.merge);
  const dim3 mgrid(unsigned(work.merges.size()), 2 * (kTile / kMergeWarps)), mblock(32 * kMergeWarps);
  return layout->dtype == KPX_F16
             ? launch_chained(prefill_merge_kernel<__half>, mgrid, mblock, 0, stream, static_cast<__half*>(out), p.partials,
                              num_q_heads, group_heads, item_tokens, mlist)
             : launch_chained(prefill_merge_kernel<__nv_bfloat16>, mgrid, mblock, 0, stream, static_cast<__nv_bfloat16*>(out),
                              p.partials, num_q_heads, group_heads, item_tokens, mlist);
}

// Bytes of the work area prefill_tc may need for a call with total_q query tokens.
int64_t prefill_tc_area_bytes(int32_t total_q, int32_t num_q_heads) {
  const int64_t h = num_q_heads > 0 ? num_q_heads : 1;
  // never more units than (token, KV head) pairs, plus the parts of cut ones; the part slots
  return align256(int64_t(kMaxClusters + 1) * 4) +
         align256((int64_t(total_q) + 1) * h * int64_t(sizeof(Unit)) + int64_t(kMaxPartSlots) * int64_t(sizeof(Unit))) +
         int64_t(kMaxPartSlots) * kPartSlotFloats * int64_t(sizeof(float));
}

}  // namespace kpx

// Test knob (not in the public header): makes a bounded wait of the tensor-core kernel run out
// without a faulting or endless kernel: CTA (`withhold_cta` & 0xffff) announces one tile to its
// barrier but never requests it (`withhold_cta` >> 16 = 0: K of its first key tile, 1: V of its
// first key tile, 2: K of its second key tile), and the waits give up after `wait_limit` polls
// (0: the default).
extern "C" __attribute__((visibility("default"))) void kpx_internal_set_prefill_fault(uint32_t wait_limit, int withhold_cta) {
  kpx::g_prefill_wait_limit = wait_limit ? wait_limit : kpx::kWaitLimit;
  kpx::g_prefill_withhold_cta = withhold_cta;
}
// Test knob (not in the public header): see g_prefill_split.
extern "C" __attribute__((visibility("default"))) void kpx_internal_set_prefill_split(int v) { kpx::g_prefill_split = v; }
