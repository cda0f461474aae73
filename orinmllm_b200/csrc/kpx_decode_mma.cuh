// Paged GQA decode attention for 16-bit caches: the split-KV streaming of kpx_decode_impl.cuh (one
// line of blocks cut into equal ranges, one per warp; pieces of cut items assembled by the last
// warp to arrive) with the two contractions on matrix instructions.
//
// Why matrix instructions: with up to eight query heads per KV head a 16-token tile (8 KB of K and
// V) costs about 350 warp instructions here, all of a launch counted (354, fp16), and cost 816 (four
// heads) to 1632 (five to eight heads, in two passes over the tile) as packed fp32 FMAs, so that the
// instruction stream and not HBM set the rate.  One warp owns a tile: S = Q K^T and O += P V are m16n8k16 products whose 16 rows are
//   scores:  rows 0..7 = the eight query heads, rows 8..15 zero;
//   output:  rows 0..7 = P_hi, rows 8..15 = P_lo of the same heads, p = P_hi + P_lo in two 16-bit
//            terms, so that the second term costs no instruction of its own; the two row halves of
//            the fp32 accumulator are added once, when the item ends.  Two bf16 terms hold 16 bits of
//            a weight and not the 24 it has: bf16 caches take a second product with half of P_hi in
//            both and a third term P_lo2 in its rows 8..15 (no row of a product is left at 0, which
//            times an infinity in V would be NaN).
// Thread (g = lane / 4, t = lane % 4) holds head g and tokens 2t, 2t+1, 2t+8, 2t+9 of the scores:
// the layout of the accumulator is that of the A operand of the second product, so weights never
// leave their thread; the row maximum is two shuffles.  Q enters exactly as stored (bf16 rows times a
// power of two, Mma::row_scale); the softmax scale is applied to the fp32 scores.  The weights of fp16
// caches are scaled by 2^12 (the running sum with them), which keeps P_lo of small weights out of
// the subnormals.
//
// Tiles arrive by TMA through 128-byte-swizzled tensor maps of the pools ([half row][16 tokens][64
// elements], one 4 KB box), so that ldmatrix reads them without bank conflicts.  A strided cache
// may end inside a block: the rows of such a block that exist come by one bulk copy each, unswizzled.
// Eight warps per SM.  A launch that has the GPU to itself gives a warp one K and one V slot: 64 KB
// in flight per SM keep HBM busy, and more only lengthens the queues, in which the SMs farther from
// the memory they read fall behind until the last warp ends 25 us after the median one.  us per
// launch with 1 / 2 / 3 slots (alone): 32/8 heads, 64 sequences of 128..4096 tokens 100 / 104 / 110; 16 of
// 8k..32k 215 / 226 / 237; one of 131072 107 / 110 / 113; 28/4 heads bf16, 64 sequences
// 61 / 65 / 66.6.  (Twelve warps of two slots: 134; four warps of six: 126.)
//
// Measured, us per launch in a graph, packed FMAs -> now: 64 sequences of 128..4096 tokens, 28/4 heads
// bf16 93 -> 57 (the third term costs 1 of them), 32/8 fp16 100 -> 94, 32/8 bf16 101 -> 97 (third
// term 3); 16 of 8k..32k, 32/8 fp16 213 -> 201; one of 131072 107 -> 95.  Errors against 64 bits are those
// of the FMAs to five digits (rounding of the output included: fp16 2.1e-4, bf16 1.7e-3).
#pragma once
#include "kpx_decode_impl.cuh"
#include "kpx_tma.cuh"

namespace kpx {
namespace decode {

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldsm4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}

constexpr float kLeastHalf = 5.9604644775390625e-8f;  // 2^-24, the least positive fp16 value

template <typename T>
struct Mma;
template <>
struct Mma<__half> {
  static constexpr int kTerms = 2;            // 16-bit terms that hold a weight: 22 bits, the accuracy of ex2.approx
  static constexpr float kWeightBias = 12.f;  // log2 of the scale the weights carry
  static __device__ __forceinline__ void run(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
  // the part of the softmax scale that the scores take; products of fp16 rows fit fp32 as they are
  static __device__ __forceinline__ float score_scale(float qscale) { return qscale; }
  static __device__ __forceinline__ uint32_t pack(float x, float y) {
    const __half2 h = __floats2half2_rn(x, y);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  static __device__ __forceinline__ float2 unpack(uint32_t w) {
    return __half22float2(*reinterpret_cast<const __half2*>(&w));
  }
};
template <>
struct Mma<__nv_bfloat16> {
  static constexpr int kTerms = 3;  // (two would hold 16 bits)
  static constexpr float kWeightBias = 0.f;
  static __device__ __forceinline__ void run(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
  // bf16 rows reach as far as fp32 does, and their products beyond it although the scaled score need not:
  // the rows take the power of two of the scale, which is exact, the scores its mantissa
  static __device__ __forceinline__ bool normal(float qscale) { return (__float_as_uint(qscale) & 0x7f800000u) != 0; }
  static __device__ __forceinline__ float row_scale(float qscale) {
    return normal(qscale) ? __uint_as_float(__float_as_uint(qscale) & 0x7f800000u) : 1.f;
  }
  static __device__ __forceinline__ float score_scale(float qscale) {
    return normal(qscale) ? __uint_as_float((__float_as_uint(qscale) & 0x807fffffu) | 0x3f800000u) : qscale;
  }
  static __device__ __forceinline__ uint32_t pack(float x, float y) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  static __device__ __forceinline__ float2 unpack(uint32_t w) {
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  }
};

// One warp's part of one item: query rows, running softmax state and accumulator of eight heads, and
// the arithmetic of a 16-token tile.
template <typename T_>
struct MmaTile {
  using T = T_;
  using M = Mma<T>;
  static constexpr int QH = kMmaHeads, kRowB = kD * 2;
  // rows of a staging area in shared memory: the stride spreads the eight rows that a warp reads
  // at a time over the banks
  static constexpr int kRowStride = kRowB + 16;
  static constexpr bool kTensorMaps = true;
  static constexpr int kWidestForm = 8;  // warps of the cluster form that has an SM to itself
  float by;           // what a product with the query rows is multiplied by to be a score (set by scale_q)
  uint32_t qa[8][2];  // A fragments: k step s holds d = 16s + 2t, +1 and 16s + 8 + 2t, +1 of head g
  float acc[16][4];   // d = 8 * tile + 2t, +1 of head g: [0..1] the P_hi part, [2..3] the P_lo part
  float m, l;         // of head g; l: of the thread's own tokens until finish()
  uint32_t hi[2], lo[2], lo2[2];  // weights of the block whose output pass comes next (lo2: kTerms == 3)
  int g, t;               // head; position in the quad
  // ldmatrix addresses: lane 8m + r names row r of matrix m.  K: matrix m = 16-byte chunk m (mod 4)
  // of tokens r; V: matrix m = tokens (m & 1) * 8 + r, chunk m >> 1 (mod 2).
  int lm, lr;
  uint32_t k_off, v_off;

  __device__ __forceinline__ void reset() {
#pragma unroll
    for (int i = 0; i < 16; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;
    m = -INFINITY;
    l = 0.f;
  }
  __device__ __forceinline__ void init(int lane) {
    g = lane >> 2;
    t = lane & 3;
    lm = lane >> 3;
    lr = lane & 7;
    k_off = uint32_t(lr * 128 + ((lm ^ lr) << 4));
    v_off = uint32_t(((lm & 1) * 8 + lr) * 128 + (((lm >> 1) ^ lr) << 4));
    reset();
  }
  // rows of the group's heads, `stride` bytes apart; heads from `heads` on are zero.  Loads only: nothing
  // waits for them before scale_q, so that the requests of the first tiles go out meanwhile.
  __device__ __forceinline__ void load_q(const uint8_t* rows, int stride, int heads) {
    const bool valid = g < heads;
    const uint32_t* qh = reinterpret_cast<const uint32_t*>(rows + (valid ? g : 0) * stride) + t;
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      qa[s][0] = valid ? qh[8 * s] : 0u;
      qa[s][1] = valid ? qh[8 * s + 4] : 0u;
    }
  }
  // after load_q: the softmax scale, shared out between the rows and the scores
  __device__ __forceinline__ void scale_q(float qscale) {
    by = M::score_scale(qscale);
    if constexpr (std::is_same<T, __nv_bfloat16>::value) {
      const float rows_by = M::row_scale(qscale);
#pragma unroll
      for (int s = 0; s < 8; ++s)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float2 f = M::unpack(qa[s][h]);
          qa[s][h] = M::pack(f.x * rows_by, f.y * rows_by);
        }
    }
  }
  __device__ __forceinline__ int token(int e) const { return 2 * t + (e & 1) + (e >> 1) * 8; }
  // Scores and weights of the block whose K tile is at kt; kTail: only nvalid of its tokens exist
  // (linear: its rows lie one after the other, not swizzled).
  template <bool kTail>
  __device__ __forceinline__ void scores_of(uint32_t kt, int nvalid, bool linear) {
    float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};  // tokens 0..7, 8..15
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint32_t a = kt + (k_off ^ ((i & 1) << 6)) + (i >> 1) * 2048, step8 = 1024;
      if (kTail && linear) {
        a = kt + lr * kRowB + (4 * i + lm) * 16;
        step8 = 8 * kRowB;
      }
      uint32_t b0[4], b1[4];
      ldsm4(b0, a);
      ldsm4(b1, a + step8);
      M::run(c0, qa[2 * i][0], 0u, qa[2 * i][1], 0u, b0[0], b0[1]);
      M::run(c1, qa[2 * i][0], 0u, qa[2 * i][1], 0u, b1[0], b1[1]);
      M::run(c0, qa[2 * i + 1][0], 0u, qa[2 * i + 1][1], 0u, b0[2], b0[3]);
      M::run(c1, qa[2 * i + 1][0], 0u, qa[2 * i + 1][1], 0u, b1[2], b1[3]);
    }
    float s[4] = {c0[0] * by, c0[1] * by, c1[0] * by, c1[1] * by};
    if (kTail) {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (token(e) >= nvalid) s[e] = -INFINITY;
    }
    float mx = fmaxf(fmaxf(s[0], s[1]), fmaxf(s[2], s[3]));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float m_new = fmaxf(m, mx);
    const float alpha = fast_exp2(m - m_new);
    const bool changed = m_new != m;
    m = m_new;
    float w[4], first[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      w[e] = fast_exp2(s[e] - m_new + M::kWeightBias);
      if (kTail && token(e) >= nvalid) w[e] = 0.f;
      // 0 only where the weight is (see finish())
      first[e] = M::kTerms == 3 ? 0.5f * w[e] : (w[e] > 0.f ? fmaxf(w[e], kLeastHalf) : 0.f);
    }
    l = l * alpha + ((w[0] + w[1]) + (w[2] + w[3]));
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      hi[h] = M::pack(first[2 * h], first[2 * h + 1]);
      const float2 f = M::unpack(hi[h]);
      float2 r = make_float2(w[2 * h] - f.x, w[2 * h + 1] - f.y);
      if constexpr (M::kTerms == 3) r = make_float2(r.x - f.x, r.y - f.y);
      lo[h] = M::pack(r.x, r.y);
      if constexpr (M::kTerms == 3) {
        const float2 f2 = M::unpack(lo[h]);
        lo2[h] = M::pack(r.x - f2.x, r.y - f2.y);
      }
    }
    if (__any_sync(0xffffffffu, changed)) {
#pragma unroll
      for (int i = 0; i < 16; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][e] *= alpha;
    }
  }
  // Output pass of that block, V tile at vt.
  template <bool kTail>
  __device__ __forceinline__ void output_of(uint32_t vt, int nvalid, bool linear) {
    // rows past the newest token hold anything, NaN included: their halves of the packed pairs are cleared
    uint32_t mask[2] = {0xffffffffu, 0xffffffffu};
    if (kTail) {
#pragma unroll
      for (int h = 0; h < 2; ++h)
        mask[h] = (token(2 * h) < nvalid ? 0xffffu : 0u) | (token(2 * h + 1) < nvalid ? 0xffff0000u : 0u);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      uint32_t a = vt + (v_off ^ ((i & 3) << 5)) + (i >> 2) * 2048;
      if (kTail && linear) a = vt + ((lm & 1) * 8 + lr) * kRowB + (2 * i + (lm >> 1)) * 16;
      uint32_t b[4];
      ldsm4_trans(b, a);
      if (kTail) {
#pragma unroll
        for (int e = 0; e < 4; ++e) b[e] &= mask[e & 1];
      }
      // The products of a tile are summed by themselves and added to the running sums in fp32, rounded
      // to nearest: a matrix instruction cuts its sums off, and over hundreds of tiles that adds up.
      float d[2][4] = {};
#pragma unroll
      for (int u = 0; u < 2; ++u) M::run(d[u], hi[0], lo[0], hi[1], lo[1], b[2 * u], b[2 * u + 1]);
      if (M::kTerms == 3) {
#pragma unroll
        for (int u = 0; u < 2; ++u) M::run(d[u], hi[0], lo2[0], hi[1], lo2[1], b[2 * u], b[2 * u + 1]);
      }
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
          float(&a)[4] = acc[2 * i + u];
          const float2 sum = __fadd2_rn(make_float2(a[e], a[e + 1]), make_float2(d[u][e], d[u][e + 1]));
          a[e] = sum.x;
          a[e + 1] = sum.y;
        }
    }
  }
  __device__ __forceinline__ void scores(const uint8_t* kt, int nvalid, bool linear) {
    if (nvalid < kBS) scores_of<true>(smem_u32(kt), nvalid, linear);
    else scores_of<false>(smem_u32(kt), nvalid, false);
  }
  __device__ __forceinline__ void output(const uint8_t* vt, int nvalid, bool linear) {
    if (nvalid < kBS) output_of<true>(smem_u32(vt), nvalid, linear);
    else output_of<false>(smem_u32(vt), nvalid, false);
  }
  // l over the head's tokens, in all four threads of the quad; acc[i][0..1] = the sum of both parts.
  // Where V holds an infinity (fp16 caches overflow to one) the part of the first terms alone says
  // what becomes of the sum, as no weight but 0 has a first term of 0.  A second term may be 0 or
  // negative, so that its part is then an infinity of either sign or NaN; it is finite otherwise, and
  // counts only if it is.
  __device__ __forceinline__ void finish() {
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
#pragma unroll
    for (int i = 0; i < 16; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (fabsf(acc[i][2 + e]) < INFINITY) acc[i][e] += acc[i][2 + e];
  }
  // after finish(): one more token whose rows are at k_row and v_row
  __device__ __forceinline__ void add_token(const uint8_t* k_row, const uint8_t* v_row) {
    const uint32_t* kr = reinterpret_cast<const uint32_t*>(k_row) + t;
    const uint32_t* vr = reinterpret_cast<const uint32_t*>(v_row) + t;
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float2 a = M::unpack(qa[i][h]), b = M::unpack(kr[8 * i + 4 * h]);
        s = fmaf(a.x, b.x, fmaf(a.y, b.y, s));
      }
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s *= by;
    const float m_new = fmaxf(m, s);
    const float a = fast_exp2(m - m_new), w = fast_exp2(s - m_new + M::kWeightBias);
    m = m_new;
    l = l * a + w;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float2 v = M::unpack(vr[4 * i]);
      acc[i][0] = fmaf(w, v.x, acc[i][0] * a);
      acc[i][1] = fmaf(w, v.y, acc[i][1] * a);
    }
  }
  // after finish(): [heads][128] accumulators, then the maxima, then the sums
  __device__ __forceinline__ void store(float* dst, int heads = kMmaHeads) const {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      *reinterpret_cast<float2*>(dst + g * kD + 8 * i + 2 * t) = make_float2(acc[i][0], acc[i][1]);
    if (t == 0) {
      dst[heads * kD + g] = m;
      dst[heads * kD + heads + g] = l;
    }
  }
  static __device__ __forceinline__ void write4(T* row, int d, float4 v) {
    *reinterpret_cast<uint2*>(row + d) = make_uint2(M::pack(v.x, v.y), M::pack(v.z, v.w));
  }
};

template <int NW, int NS>
struct MmaCfg {
  static constexpr int kTileB = kBS * kD * 2;
  static constexpr int kThreads = 32 * NW;
  static constexpr int kWarpRingB = 2 * NS * kTileB;  // K slots then V slots
  static constexpr int kOffBars = NW * kWarpRingB;
  static constexpr int kOffPrefix = kOffBars + NW * 2 * NS * 8;
  static constexpr int kOffStage = kOffPrefix + (kMaxBatch + 1) * 4 + 12;
  static constexpr int kSmem = 1024 /*align slack*/ + kOffStage;
  // Fused step only: per warp, the rotated query rows of the item's heads, the new token's rotated
  // K row and its V row, and the id of the block the token goes to.  The row stride spreads the
  // eight rows that a warp reads at a time over the banks.
  static constexpr int kRowStride = kD * 2 + 16;
  static constexpr int kStageB = (kMmaHeads + 2) * kRowStride + 16;
  static constexpr int kSmemFused = kSmem + NW * kStageB;
  static_assert(kWarpRingB % 1024 == 0 && kOffStage % 16 == 0, "alignment of the slots and of the staging area");
};

// Adds up the pieces of an item in `cnt` workspace slots of SH heads (the first is slot `first`, the
// i-th one after it slot from + 2 i): into one unnormalised slot at dst, or into the item's output
// rows if dst is nullptr.  32 / SH lanes share a head, so that all lanes have loads in flight however
// few heads there are.  One pass: the maxima, sums and accumulators of kBatch slots are requested
// together and folded into the running ones, so that a batch is one trip to L2.  us per launch in a
// graph, four lanes a head whatever their number and three passes over the slots -> this; fp16:
// 8/8 heads, one sequence of 2000 tokens in the line of blocks 29.0 -> 17.6, 8 of 64..800 28.0 -> 17.0,
// 32/8, one of 2000 23.2 -> 15.9, one of 131072 104.5 -> 96.8 (and 238 registers a thread, not 255).
template <typename T, int SH>
__device__ __forceinline__ void merge_slots(const float* slots, int64_t first, int64_t from, int cnt, int heads,
                                            float* dst, T* rows, int lane) {
  constexpr int kLanes = 32 / SH, kVecs = kD / 4 / kLanes, kBatch = kVecs > 2 ? 16 / kVecs : 8;
  constexpr int64_t kFloats = slot_floats_of(SH);
  const int head = lane / kLanes, t = lane % kLanes;
  if (head >= heads) return;
  const float* row = slots + head * kD + 4 * t;
  const float* stats = slots + SH * kD + head;
  float m = -INFINITY, l = 0.f;
  float4 o[kVecs];
#pragma unroll
  for (int k = 0; k < kVecs; ++k) o[k] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int i0 = 0; i0 < cnt; i0 += kBatch) {
    float mi[kBatch], li[kBatch], m_new = m;
    float4 v[kBatch][kVecs];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int i = min(i0 + u, cnt - 1);
      const int64_t at = (i ? from + 2 * i : first) * kFloats;
      mi[u] = i0 + u < cnt ? __ldcg(stats + at) : -INFINITY;  // (a slot read twice has no weight)
      li[u] = __ldcg(stats + at + SH);
#pragma unroll
      for (int k = 0; k < kVecs; ++k) v[u][k] = __ldcg(reinterpret_cast<const float4*>(row + at + 4 * k * kLanes));
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) m_new = fmaxf(m_new, mi[u]);
    const float a = fast_exp2(m - m_new);
    m = m_new;
    l *= a;
#pragma unroll
    for (int k = 0; k < kVecs; ++k) o[k] = make_float4(o[k].x * a, o[k].y * a, o[k].z * a, o[k].w * a);
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      if (i0 + u >= cnt) break;
      const float w = fast_exp2(mi[u] - m);
      l = fmaf(li[u], w, l);
#pragma unroll
      for (int k = 0; k < kVecs; ++k) {
        o[k].x = fmaf(v[u][k].x, w, o[k].x);
        o[k].y = fmaf(v[u][k].y, w, o[k].y);
        o[k].z = fmaf(v[u][k].z, w, o[k].z);
        o[k].w = fmaf(v[u][k].w, w, o[k].w);
      }
    }
  }
  if (dst) {
#pragma unroll
    for (int k = 0; k < kVecs; ++k) *reinterpret_cast<float4*>(dst + head * kD + 4 * (k * kLanes + t)) = o[k];
    if (t == 0) {
      dst[SH * kD + head] = m;
      dst[SH * kD + SH + head] = l;
    }
  } else {
    const float inv = 1.f / l;
#pragma unroll
    for (int k = 0; k < kVecs; ++k)
      MmaTile<T>::write4(rows + head * kD, 4 * (k * kLanes + t),
                         make_float4(o[k].x * inv, o[k].y * inv, o[k].z * inv, o[k].w * inv));
  }
}

template <typename T, int NW, int NS, int CPS, bool kFused>
__global__ void __launch_bounds__(32 * NW, CPS)
paged_decode_mma_kernel(const DecodeParams p, const __grid_constant__ CUtensorMap map_k,
                        const __grid_constant__ CUtensorMap map_v) {
  using C = MmaCfg<NW, NS>;
  using M = Mma<T>;
  constexpr int kRowB = kD * 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kOffBars) + warp * 2 * NS;  // K slots, V slots
  int* prefix = reinterpret_cast<int*>(smem + C::kOffPrefix);
  uint8_t* ring = smem + warp * C::kWarpRingB;
  const uint32_t ring_u = smem_u32(ring);
  uint8_t* stage = smem + C::kOffStage + warp * C::kStageB;  // fused step only

  // ---- prologue: block prefix over sequences (whole CTA), this warp's barriers ----
  if (lane == 0) {
#pragma unroll
    for (int s = 0; s < 2 * NS; ++s) mbar_init(bars + s, 1);
    mbar_fence_init();
    prefetch_tensormap(&map_k);
    prefetch_tensormap(&map_v);
  }
  const int64_t after_wait = grid_wait();
  // (no grid_release(): kpx_common.cuh)
  // With a plan of the step the prefix and this warp's starting point come from it: one round
  // trip to global memory instead of lengths -> prefix -> search -> first block id.
  bool planned = false;
  int4 plan_entry = make_int4(0, 0, 0, 0);
  if constexpr (!kFused) {
    if (p.plan && !p.small) {
      // header, this warp's entry and the prefix are requested together (a plan buffer always
      // holds kMaxSms x 16 entries and kMaxBatch + 1 prefix words, whatever was planned); what
      // the header says decides afterwards whether they are used
      const int32_t* plan = p.plan + after_wait;
      const int4 h = __ldg(reinterpret_cast<const int4*>(plan));
      const int32_t plan_error = __ldg(plan + 4);
      plan_entry = __ldg(reinterpret_cast<const int4*>(plan + kPlanEntriesAt) + (blockIdx.x * NW + warp));
      for (int b = tid; b <= p.batch; b += C::kThreads) prefix[b] = __ldg(plan + kPlanPrefixAt + b);
      planned = h.x == kPlanMark && h.y == p.batch && h.z == int(gridDim.x) * NW &&
                h.w == p.num_kv_heads * p.head_groups;
      if (planned && blockIdx.x == 0 && tid == 0 && plan_error != 0) atomicMax(p.status, plan_error);
      __syncthreads();
    }
  }
  if (!planned) block_prefix(p, prefix, tid, C::kThreads, warp, lane, blockIdx.x == 0);
  write_empty_rows<T, kFused>(p, prefix, tid, C::kThreads);

  // ---- this warp's range of the line of blocks ----
  const int64_t total = int64_t(prefix[p.batch]) * p.num_kv_heads * p.head_groups;
  int64_t W = int64_t(gridDim.x) * NW;
  int64_t worker = int64_t(blockIdx.x) * NW + warp;
  if (p.small && total < W * p.min_blocks_per_range) {
    // Few blocks per warp: fewer, longer ranges (every piece of a cut item costs a partial and a
    // share of the assembly, and a range of a block or two is all prologue), warps numbered
    // CTA-minor so that the active ones stay spread over all SMs.
    int64_t w = total / p.min_blocks_per_range;
    const int64_t floor_w = int64_t(gridDim.x) * (NW < p.min_warps_per_sm ? NW : p.min_warps_per_sm);
    if (w < floor_w) w = floor_w;
    if (w < 1) w = 1;
    if (w < W) W = w;
    worker = int64_t(warp) * gridDim.x + blockIdx.x;
    if (worker >= W) return;  // nothing below synchronises across warps
  }
  Split split;
  if (total < (int64_t(1) << 31)) {  // (W is at most a few thousand)
    split.quot = int64_t(uint32_t(total) / uint32_t(W));
  } else {
    split.quot = total / W;
  }
  split.rem = total - split.quot * W;
  const int64_t u0 = split.start(worker), u1 = split.start(worker + 1);
  if (u0 >= u1) return;  // nothing below synchronises across warps
  const int n = int(u1 - u0);

  MmaTile<T> tile;
  tile.init(lane);
  const int g = tile.g, t = tile.t;  // head of the group; position in the quad

  // ---- producer side: block ids and tile requests of this warp's own range; one cursor walks
  // the range NS blocks ahead of the consumer ----
  Cursor cur;  // consumer side: first block of the current segment
  if (planned) {
    cur.b = plan_entry.x >> 16;
    cur.sub = plan_entry.x & 0xffff;
    cur.blk = plan_entry.y;
    cur.len = plan_entry.z;
    cur.nblk = prefix[cur.b + 1] - prefix[cur.b];
    cur.refresh(p);
  } else {
    cur.locate(p, prefix, u0);
  }
  auto load_q = [&]() {
    const int h0 = (cur.sub - cur.kvh * p.head_groups) * kMmaHeads;
    tile.load_q(static_cast<const uint8_t*>(p.q) + (int64_t(cur.b) * p.num_q_heads + cur.kvh * p.kv_mul + h0) * kRowB, kRowB,
                p.kv_mul - h0);
  };
  // The first item's rows are requested here, before the first block id and the first tiles, so
  // that their latency (DRAM if nothing brought them to L2) runs under those.
  if constexpr (!kFused) load_q();
  Cursor pc = cur;
  int pc_id;  // block id at pc (loaded one step before it is needed)
  int last_id = 0, last_kvh = 0, last_rows = kBS;  // the block whose K tile was requested last
  int k_issued = 0, v_issued = 0;
  auto checked_id = [&](int id) -> int {
    if (id < 0 || (p.num_blocks > 0 && id >= p.num_blocks)) {
      if (lane == 0) atomicMax(p.status, KPX_ERR_INVALID_ARGUMENT);
      id = 0;
    }
    return id;
  };
  auto load_id = [&]() -> int { return checked_id(pc.row ? __ldg(pc.row + pc.blk) : pc.blk); };
  // request one tile (callers have __syncwarp'ed after the last read of the slot)
  auto copy_tile = [&](const CUtensorMap* map, const uint8_t* pool, int slot_index, bool withhold = false) {
    uint64_t* bar = bars + slot_index;
    uint8_t* dst = ring + slot_index * C::kTileB;
    if (p.tile_contig || last_rows == kBS) {
      if (lane == 0) {
        mbar_arrive_expect_tx(bar, C::kTileB);
        if (!withhold) tma_load_5d(dst, map, 0, 0, 0, last_kvh, last_id, bar);
      }
    } else {
      // the last block of a strided cache: its other rows need not exist
      if (lane == 0) mbar_arrive_expect_tx(bar, uint32_t(last_rows) * kRowB);
      __syncwarp();
      if (lane < last_rows && !withhold)
        bulk_g2s(dst + lane * kRowB, pool + int64_t(last_id) * p.block_stride_b + int64_t(last_kvh) * p.head_stride_b +
                                         int64_t(lane) * p.token_stride_b, kRowB, bar);
    }
  };
  auto issue_k = [&](int slot) {  // K tile of the block at pc; then step pc
    last_id = pc_id;
    last_kvh = pc.kvh;
    last_rows = min(kBS, pc.len - pc.blk * kBS);
    copy_tile(&map_k, p.k_pool, slot, k_issued == 0 && worker == p.withhold_worker);
    ++k_issued;
    pc.advance(p, prefix);
    if (k_issued < n) pc_id = load_id();
  };
  auto issue_v = [&](int slot) {  // V tile of the block whose K tile was requested last
    copy_tile(&map_v, p.v_pool, NS + slot);
    ++v_issued;
  };
  pc_id = planned ? checked_id(plan_entry.w) : load_id();
#pragma unroll
  for (int k = 0; k < NS; ++k) {
    if (k < n) {
      issue_k(k);
      issue_v(k);
    }
  }

  // ---- consumer state ----
  auto begin_item = [&](int blocks_left, bool first) {
    if constexpr (kFused) {
      const int hg = cur.sub - cur.kvh * p.head_groups;
      const int seg = min(blocks_left, cur.nblk - cur.blk);
      const bool ends_item = cur.blk + seg == cur.nblk;
      __syncwarp();  // the previous item's readers of the staging area are done
      stage_new_token<T, kMmaHeads, C::kRowStride>(
          static_cast<const T*>(p.q) + (int64_t(cur.b) * p.num_q_heads + int64_t(cur.kvh) * p.kv_mul) * kD, hg, p.kv_mul,
          static_cast<const T*>(p.k_new) + (int64_t(cur.b) * p.num_kv_heads + cur.kvh) * kD,
          static_cast<const uint8_t*>(p.v_new) + (int64_t(cur.b) * p.num_kv_heads + cur.kvh) * kRowB, ends_item,
          p.sin_cache + int64_t(cur.len) * kD, p.cos_cache + int64_t(cur.len) * kD,
          cur.row ? cur.row + cur.len / kBS : nullptr, cur.len / kBS, stage, lane);
      __syncwarp();
      tile.load_q(stage, C::kRowStride, p.kv_mul - hg * kMmaHeads);
    } else if (!first) {
      load_q();
    }
    tile.scale_q(p.qscale);
    tile.reset();
  };

  auto end_item = [&](const Cursor& item, bool whole_item, int64_t partial_slot, int64_t item_start,
                      bool has_item_end) {
    const int hg = item.sub - item.kvh * p.head_groups;
    const int hq = hg * kMmaHeads + g;  // this thread's head within the KV head
    const bool head_ok = hq < p.kv_mul;
    tile.finish();
    if (kFused && has_item_end) {
      // Fused step: this piece ends the item, so it also carries the new token (position
      // item.len, not in the pool yet), staged when the item began.
      tile.add_token(stage + kMmaHeads * C::kRowStride, stage + (kMmaHeads + 1) * C::kRowStride);
      // append: the first head group's warp stores the rows (lanes 0..15 the K row, 16..31 the V
      // row) into the block that holds position item.len
      if (hg == 0) {
        const int id = *reinterpret_cast<const int32_t*>(stage + (kMmaHeads + 2) * C::kRowStride);
        if (id < 0 || (p.num_blocks > 0 && id >= p.num_blocks)) {
          if (lane == 0) atomicMax(p.status, KPX_ERR_INVALID_ARGUMENT);
        } else {
          const int64_t off = int64_t(id) * p.block_stride_b + int64_t(item.kvh) * p.head_stride_b +
                              int64_t(item.len % kBS) * p.token_stride_b + (lane & 15) * 16;
          *reinterpret_cast<uint4*>((lane < 16 ? p.k_pool_w : p.v_pool_w) + off) =
              *reinterpret_cast<const uint4*>(stage + (kMmaHeads + (lane >> 4)) * C::kRowStride + (lane & 15) * 16);
        }
      }
    }
    T* orow = static_cast<T*>(p.out) + (int64_t(item.b) * p.num_q_heads + item.kvh * p.kv_mul + hq) * kD;
    if (whole_item) {
      if (head_ok) {
        const float inv = 1.f / tile.l;
        uint32_t* o = reinterpret_cast<uint32_t*>(orow) + t;
#pragma unroll
        for (int i = 0; i < 16; ++i) o[4 * i] = M::pack(tile.acc[i][0] * inv, tile.acc[i][1] * inv);
      }
      return;
    }
    // one workspace slot: slot_heads accumulators of 128, then their maxima, then their sums
    const int sh = p.slot_heads;
    const int64_t slot_floats = slot_floats_of(sh);
    if (head_ok) tile.store(p.partials + partial_slot * slot_floats, sh);
    // The item is cut by a range boundary.  Publish this piece, then count it; the warp
    // that brings the count up to the number of pieces assembles the item from all of
    // them (nobody waits: whoever arrives last does the work) and resets the counter.
    __syncwarp();  // every lane's piece is ordered before lane 0's release below
    // every warp between the owners of the item's first and last block holds a piece of it
    const int64_t c_first = split.owner(item_start), c_last = split.owner(item_start + item.nblk - 1);
    const int pieces = int(c_last - c_first) + 1;
    // release our writes, acquire the other arrivals' (device scope, cumulative over the warp);
    // true in the warp that arrives last, which also resets the counter
    auto arrive_last = [&](int* cnt, int expected) -> bool {
      int prev = 0;
      if (lane == 0)
        asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], 1;" : "=r"(prev) : "l"(cnt) : "memory");
      prev = __shfl_sync(0xffffffffu, prev, 0);
      if (prev != expected - 1) return false;
      if (lane == 0) *cnt = 0;
      __syncwarp();
      return true;
    };
    // An item cut into many pieces (one very long sequence) is assembled in two levels so that
    // no single warp reads them all: the pieces of `group` consecutive warps are merged by the
    // last of them to arrive into one slot of a second area, and the last group to finish
    // merges those.  The second area sits at the end of the slot array: [group slots][one
    // slot of group counters]; it is used only if the array has room for it.  A flat item has at
    // most as many pieces as a group has warps: a group then never holds more than two grouped items.
    const int group = sh == 1 ? 32 : 16;  // (one-head slots are short: their last one holds fewer counters)
    const int64_t W_all = int64_t(gridDim.x) * NW;
    const int64_t n_groups = (W_all + group - 1) / group;
    const int64_t group_base = int64_t(p.partial_slots) - 1 - 2 * n_groups;  // first group slot
    const bool flat = pieces <= group || group_base < 2 * W_all || 2 * n_groups > slot_floats_of(sh > 4 ? 4 : sh);
    // what is merged next: cnt slots (only an item's first piece can be a "tail" slot), and where to
    int* counter = p.counters + (item.b * (p.num_kv_heads * p.head_groups) + item.sub);
    int cnt = pieces;
    int64_t first = 2 * c_first + 1, from = 2 * c_first;
    float* dst = nullptr;
    if (!flat) {
      // A group holds pieces of at most two such items: one that entered it from the left (0) and
      // one that starts inside it (1).
      const int64_t gr = worker / group;
      const int in = c_first < gr * group ? 0 : 1;
      const int64_t g_lo = in ? c_first : gr * group;
      const int64_t g_hi = c_last < gr * group + group - 1 ? c_last : gr * group + group - 1;
      counter = p.group_counters + 2 * gr + in;
      cnt = int(g_hi - g_lo) + 1;
      first = 2 * g_lo + in;
      from = 2 * g_lo;
      dst = p.partials + (group_base + 2 * gr + in) * slot_floats;
    }
    T* rows = static_cast<T*>(p.out) + (int64_t(item.b) * p.num_q_heads + item.kvh * p.kv_mul + hg * kMmaHeads) * kD;
    const int heads = min(kMmaHeads, p.kv_mul - hg * kMmaHeads);
    for (;;) {
      if (!arrive_last(counter, cnt)) return;
      switch (sh) {
        case 1: merge_slots<T, 1>(p.partials, first, from, cnt, heads, dst, rows, lane); break;
        case 2: merge_slots<T, 2>(p.partials, first, from, cnt, heads, dst, rows, lane); break;
        case 4: merge_slots<T, 4>(p.partials, first, from, cnt, heads, dst, rows, lane); break;
        default: merge_slots<T, kMmaHeads>(p.partials, first, from, cnt, heads, dst, rows, lane); break;
      }
      if (!dst) return;
      __syncwarp();  // every lane's part of the group slot is ordered before lane 0's release
      const int64_t G0 = c_first / group, G1 = c_last / group;
      counter = p.counters + (item.b * (p.num_kv_heads * p.head_groups) + item.sub);
      cnt = int(G1 - G0) + 1;
      from = group_base + 2 * G0;
      first = from + 1;  // (the item starts inside its first group)
      dst = nullptr;
    }
  };

  auto wait_slot = [&](uint64_t* bar, uint32_t ph) -> bool {
    if (mbar_try_wait(bar, ph)) return true;
    bool ok = mbar_wait_bounded(bar, ph, p.wait_limit);
    if (!__all_sync(0xffffffffu, ok)) {
      // Give up: report, then let the tile copies this warp still has in flight land (a bounded
      // pause far longer than a copy takes) before the warp retires, so that nothing arrives in
      // shared memory that has passed to another CTA.
      if (lane == 0) atomicMax(p.status, KPX_ERR_DEVICE_TIMEOUT);
      for (int k = 0; k < 64; ++k) __nanosleep(1000);
      return false;
    }
    return true;
  };

  begin_item(n, true);
  int64_t item_first = u0 - cur.blk;  // global block index where the current item starts
  int slot = 0;                       // slots of the block to consume, and their phase parity
  uint32_t phase = 0;

  // One block of 16 tokens.  kTail: only nvalid of them exist (the item's last block).  Returns
  // false if a bounded wait gave up.
  auto step = [&](int nvalid, auto tail_tag) -> bool {
    constexpr bool kTail = decltype(tail_tag)::value;
    const bool linear = kTail && !p.tile_contig;  // rows copied one by one, not swizzled
    if (!wait_slot(bars + slot, phase)) return false;
    tile.template scores_of<kTail>(ring_u + slot * C::kTileB, nvalid, linear);
    __syncwarp();  // the K slot is read
    if (k_issued < n) {
      if (lane == 0) fence_proxy_async();
      issue_k(slot);
    }
    if (!wait_slot(bars + NS + slot, phase)) return false;
    tile.template output_of<kTail>(ring_u + (NS + slot) * C::kTileB, nvalid, linear);
    __syncwarp();  // the V slot is read
    if (v_issued < n) {
      if (lane == 0) fence_proxy_async();
      issue_v(slot);
    }
    if (++slot == NS) {
      slot = 0;
      phase ^= 1;
    }
    return true;
  };

  // The range is a sequence of segments, each the part of one item that falls in it.
  int i = 0;
  while (i < n) {
    const int seg = min(n - i, cur.nblk - cur.blk);  // blocks of this item in the range
    if (i + seg < n && lane < (kFused ? 28 : 16)) {
      // the next segment starts a new item: pull its query rows towards L2 now (128-byte lines),
      // and in the fused step the rows it rotates with: the new token's K and V rows and the
      // sin / cos rows of its position
      Cursor nx = cur;
      nx.blk += seg - 1;
      nx.advance(p, prefix);
      const int64_t kv_row = (int64_t(nx.b) * p.num_kv_heads + nx.kvh) * kRowB;
      const int hqn = min((nx.sub - nx.kvh * p.head_groups) * kMmaHeads + (lane >> 1), p.kv_mul - 1);
      const int l = lane - 16;
      const uint8_t* src =
          l < 0   ? static_cast<const uint8_t*>(p.q) +
                      (int64_t(nx.b) * p.num_q_heads + nx.kvh * p.kv_mul + hqn) * kRowB + (lane & 1) * 128
          : l < 2 ? static_cast<const uint8_t*>(p.k_new) + kv_row + l * 128
          : l < 4 ? static_cast<const uint8_t*>(p.v_new) + kv_row + (l - 2) * 128
          : l < 8 ? reinterpret_cast<const uint8_t*>(p.sin_cache + int64_t(nx.len) * kD) + (l - 4) * 128
                  : reinterpret_cast<const uint8_t*>(p.cos_cache + int64_t(nx.len) * kD) + (l - 8) * 128;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(src));
    }
    const bool to_item_end = (cur.blk + seg == cur.nblk);
    const int tail_valid = to_item_end ? cur.len - (cur.nblk - 1) * kBS : kBS;  // tokens in the segment's last block
    const int full = tail_valid < kBS ? seg - 1 : seg;
    for (int b = 0; b < full; ++b)
      if (!step(kBS, std::false_type{})) return;
    if (full < seg && !step(tail_valid, std::true_type{})) return;
    i += seg;
    const int64_t item_end = item_first + cur.nblk;
    const bool whole = (item_first >= u0) && (item_end <= u1);
    const int64_t pslot = (item_first < u0) ? 2 * worker : 2 * worker + 1;
    end_item(cur, whole, pslot, item_first, to_item_end);
    if (i < n) {
      cur.blk += seg - 1;
      cur.advance(p, prefix);
      item_first = item_end;
      begin_item(n - i, false);
    }
  }
}

// Tensor map of a pool: [blocks][kv heads][two halves of a row][16 tokens][64 elements] by the
// layout's strides; one box is a (block, head) tile.
inline bool make_pool_map(CUtensorMap* map, int32_t dtype, const void* pool, const DecodeParams& p) {
  // (a dimension of extent 1 is never stepped over: its stride may be anything valid)
  const cuuint64_t blocks = p.num_blocks > 0 && p.num_blocks < (int64_t(1) << 31) ? cuuint64_t(p.num_blocks) : cuuint64_t(1) << 31;
  const cuuint64_t dims[5] = {64, cuuint64_t(kBS), 2, cuuint64_t(p.num_kv_heads), blocks};
  const cuuint64_t strides[4] = {cuuint64_t(p.token_stride_b), 128, p.num_kv_heads > 1 ? cuuint64_t(p.head_stride_b) : kD * 2,
                                 blocks > 1 ? cuuint64_t(p.block_stride_b) : kBS * kD * 2};
  const cuuint32_t box[5] = {64, cuuint32_t(kBS), 2, 1, 1};
  return make_map(map, dtype, pool, 5, dims, strides, box);
}

template <typename T, int NW, int NS, int CPS, bool kFused>
int launch_mma_form(const DecodeParams& p, cudaStream_t stream) {
  using C = MmaCfg<NW, NS>;
  static_assert(NW * CPS == kMmaWarpsPerSm, "a step's plan fits every form");
  // the shared-memory attribute is set once per device and kernel form; the bit mask makes
  // concurrent first calls and processes that alternate devices safe
  constexpr int smem_bytes = kFused ? C::kSmemFused : C::kSmem;
  static std::atomic<uint64_t> configured{0};
  int dev = 0;
  KPX_CUDA_TRY(cudaGetDevice(&dev));
  auto kern = paged_decode_mma_kernel<T, NW, NS, CPS, kFused>;
  const uint64_t bit = uint64_t(1) << (dev & 63);
  if (dev >= 64 || !(configured.load(std::memory_order_acquire) & bit)) {
    KPX_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes));
    if (dev < 64) configured.fetch_or(bit, std::memory_order_release);
  }
  CUtensorMap map_k, map_v;
  constexpr int32_t dtype = std::is_same<T, __half>::value ? KPX_F16 : KPX_BF16;
  if (!make_pool_map(&map_k, dtype, p.k_pool, p) || !make_pool_map(&map_v, dtype, p.v_pool, p)) return KPX_ERR_CUDA;
  int grid = device_info().sm_count;
  if (grid > kMaxSms) grid = kMaxSms;
  return launch_chained(kern, dim3(grid * CPS), dim3(C::kThreads), smem_bytes, stream, p, map_k, map_v);
}

}  // namespace decode
}  // namespace kpx
