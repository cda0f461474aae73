// Paged GQA decode attention of small launches (a chat, a few short requests): one thread-block
// cluster per item, an item being one (sequence, kv head, query-head group).
//
// What bounds such a launch is not bandwidth but the chain of dependent steps from its first
// instruction to its last store.  Cutting one line of blocks over all warps (kpx_decode_impl.cuh,
// kpx_decode_mma.cuh) costs a prefix over the lengths and a search at the start, and at the end a
// partial in global memory, an atomic, a merge, and for items cut into more than sixteen pieces
// another atomic and merge: six trips to L2 of about a microsecond each.  Here a CTA knows its item
// from its index, reads one length, and its warps take equal shares of the item's blocks; the
// pieces meet in shared memory, first those of a CTA's warps, then those of the cluster's CTAs
// through distributed shared memory.  No workspace slot, no counter, no global round trip.
// Measured when it was built, us per launch in a graph, line of blocks -> cluster form: fp16 32/8 heads, one sequence
// of 512 tokens 20.1 -> 5.5, 2000: 23.0 -> 7.4, 16384: 33.2 -> 22.5, 24000: 38.7 -> 31.2 (23 blocks
// a warp: where the two come together); 8 sequences of 1500: 23.6 -> 13.8; 64 of 200 tokens in CTAs
// of two warps: 13.9; fp32 12/2, 512 tokens: 17.0 -> 6.6, 4096: 22.3 -> 11.4.
//
// Since then a warp asks for the ids of its blocks together with the length (its share is every so-manieth block,
// known without it), and the CTAs send their pieces to the one that assembles a head instead of being asked for
// them one after the other.  Steps of RoPE + append + this, us before -> after: fp32 12/2, 512 tokens, 28 layers
// 276 -> 241; fp16 32/8, 2000 tokens, 36 layers in a graph 361 -> 329 (0.4 a layer of it in the append); fp16 12/2, 8
// sequences, 28 fused launches 274 -> 225 (214 with the new token's rows fetched together, stage_new_token).
//
// The arithmetic of a 16-token tile is a Tile type: MmaTile (16-bit caches, matrix instructions) or
// FmaTile (fp32 caches, packed FMAs).
#pragma once
#include "kpx_decode_mma.cuh"
#include "kpx_once.h"

namespace kpx {
namespace decode {

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// 16 / 8 bytes into the shared memory of CTA `rank` of the cluster, at the address `addr` has here
__device__ __forceinline__ void st_cluster_f4(uint32_t addr, uint32_t rank, float4 v) {
  asm volatile(
      "{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %0, %1;\n\t"
      "st.shared::cluster.v4.f32 [a], {%2,%3,%4,%5};\n\t}" ::"r"(addr),
      "r"(rank), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
      : "memory");
}
__device__ __forceinline__ void st_cluster_f2(uint32_t addr, uint32_t rank, float x, float y) {
  asm volatile(
      "{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %0, %1;\n\t"
      "st.shared::cluster.v2.f32 [a], {%2,%3};\n\t}" ::"r"(addr),
      "r"(rank), "f"(x), "f"(y)
      : "memory");
}

// One warp's tile arithmetic for fp32 caches: eight lanes share a token row (16 dims each), four
// token rows side by side, four passes per block; fp32 throughout.
template <int QH_>
struct FmaTile {
  using T = float;
  static constexpr int QH = QH_, kRowB = kD * 4, kRowStride = kD * 4 + 16;
  static constexpr bool kTensorMaps = false;
  static constexpr int kWidestForm = 6;  // warps of the cluster form that has an SM to itself
  static constexpr float kWeightBias = 0.f;
  float2 q[QH][8], acc[QH][8];
  float m[QH], l[QH];
  int sub, tg;  // lane within the row; row of the four
  __device__ __forceinline__ void init(int lane) {
    sub = lane & 7;
    tg = lane >> 3;
#pragma unroll
    for (int j = 0; j < QH; ++j) {
      m[j] = -INFINITY;
      l[j] = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[j][i] = make_float2(0.f, 0.f);
    }
  }
  // rows of the group's heads, `stride` bytes apart; heads from `heads` on are zero (loads only, as MmaTile)
  __device__ __forceinline__ void load_q(const uint8_t* rows, int stride, int heads) {
#pragma unroll
    for (int j = 0; j < QH; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (j < heads) v = *reinterpret_cast<const float4*>(rows + int64_t(j) * stride + (c * 32 + sub * 4) * 4);
        q[j][2 * c] = make_float2(v.x, v.y);
        q[j][2 * c + 1] = make_float2(v.z, v.w);
      }
  }
  __device__ __forceinline__ void scale_q(float qscale) {
#pragma unroll
    for (int j = 0; j < QH; ++j)
#pragma unroll
      for (int i = 0; i < 8; ++i) q[j][i] = make_float2(q[j][i].x * qscale, q[j][i].y * qscale);
  }
  static __device__ __forceinline__ void row16(const uint8_t* row, int sub, float2 (&f)[8]) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float4 v = *reinterpret_cast<const float4*>(row + (c * 32 + sub * 4) * 4);
      f[2 * c] = make_float2(v.x, v.y);
      f[2 * c + 1] = make_float2(v.z, v.w);
    }
  }
  __device__ __forceinline__ float dot(int j, const float2 (&f)[8]) const {
    float2 s = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 8; ++i) s = __ffma2_rn(q[j][i], f[i], s);
    float r = s.x + s.y;
    r += __shfl_xor_sync(0xffffffffu, r, 1);
    r += __shfl_xor_sync(0xffffffffu, r, 2);
    r += __shfl_xor_sync(0xffffffffu, r, 4);
    return r;
  }
  float w[4][QH];
  __device__ __forceinline__ void scores(const uint8_t* kt, int nvalid, bool) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      float2 f[8];
      row16(kt + (r * 4 + tg) * kRowB, sub, f);
#pragma unroll
      for (int j = 0; j < QH; ++j) {
        const float s = dot(j, f);
        w[r][j] = (r * 4 + tg < nvalid) ? s : -INFINITY;
      }
    }
#pragma unroll
    for (int j = 0; j < QH; ++j) {
      float mx = fmaxf(fmaxf(w[0][j], w[1][j]), fmaxf(w[2][j], w[3][j]));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
      const float m_new = fmaxf(m[j], mx);
      const float a = fast_exp2(m[j] - m_new);
      m[j] = m_new;
      l[j] *= a;
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[j][i] = make_float2(acc[j][i].x * a, acc[j][i].y * a);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        w[r][j] = (r * 4 + tg < nvalid) ? fast_exp2(w[r][j] - m_new) : 0.f;
        l[j] += w[r][j];  // (of the lane's own token rows; the four groups are added at the end)
      }
    }
  }
  __device__ __forceinline__ void output(const uint8_t* vt, int nvalid, bool) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if (r * 4 + tg >= nvalid) continue;  // (such a row may hold anything)
      float2 f[8];
      row16(vt + (r * 4 + tg) * kRowB, sub, f);
#pragma unroll
      for (int j = 0; j < QH; ++j)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[j][i] = __ffma2_rn(make_float2(w[r][j], w[r][j]), f[i], acc[j][i]);
    }
  }
  // everything added up over the warp
  __device__ __forceinline__ void finish() {
#pragma unroll
    for (int j = 0; j < QH; ++j) {
      l[j] += __shfl_xor_sync(0xffffffffu, l[j], 8);
      l[j] += __shfl_xor_sync(0xffffffffu, l[j], 16);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        acc[j][i].x += __shfl_xor_sync(0xffffffffu, acc[j][i].x, 8);
        acc[j][i].y += __shfl_xor_sync(0xffffffffu, acc[j][i].y, 8);
        acc[j][i].x += __shfl_xor_sync(0xffffffffu, acc[j][i].x, 16);
        acc[j][i].y += __shfl_xor_sync(0xffffffffu, acc[j][i].y, 16);
      }
    }
  }
  // after finish(): one more token whose rows are at k_row and v_row
  __device__ __forceinline__ void add_token(const uint8_t* k_row, const uint8_t* v_row) {
    float2 kf[8], vf[8];
    row16(k_row, sub, kf);
    row16(v_row, sub, vf);
#pragma unroll
    for (int j = 0; j < QH; ++j) {
      const float s = dot(j, kf);
      const float m_new = fmaxf(m[j], s);
      const float a = fast_exp2(m[j] - m_new), pw = fast_exp2(s - m_new);
      m[j] = m_new;
      l[j] = l[j] * a + pw;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        acc[j][i] = make_float2(fmaf(pw, vf[i].x, acc[j][i].x * a), fmaf(pw, vf[i].y, acc[j][i].y * a));
    }
  }
  // after finish(): [QH][128] accumulators, QH maxima, QH sums
  __device__ __forceinline__ void store(float* dst) const {
    if (tg != 0) return;
#pragma unroll
    for (int j = 0; j < QH; ++j) {
#pragma unroll
      for (int c = 0; c < 4; ++c)
        *reinterpret_cast<float4*>(dst + j * kD + c * 32 + sub * 4) =
            make_float4(acc[j][2 * c].x, acc[j][2 * c].y, acc[j][2 * c + 1].x, acc[j][2 * c + 1].y);
      if (sub == 0) {
        dst[QH * kD + j] = m[j];
        dst[QH * kD + QH + j] = l[j];
      }
    }
  }
  static __device__ __forceinline__ void write4(float* row, int d, float4 v) {
    *reinterpret_cast<float4*>(row + d) = v;
  }
};

constexpr int kMaxCluster = 16;  // (above 8 only where the device says that such clusters fit)

template <typename Tile, int NW, int NS>
struct ClusterCfg {
  // The largest cluster of this form.  The narrow forms are for launches of more items than SMs (a launch that wants
  // sixteen CTAs an item has gone to the widest form before), and their CTAs share an SM: places for the pieces of
  // sixteen CTAs took the fused form of four warps from two CTAs an SM to one (fp16 32/8 heads, 28 sequences of
  // 100..500 tokens 13.5 -> 18.3 us), and that of three (fp32, 20 of 50..250: 14.2 -> 19.5).
  static constexpr int kPerSm = Tile::kWidestForm / NW, kPerSmFused = NW == 2 ? 3 : kPerSm;
  static constexpr int kCtas = kPerSm > 1 ? 8 : kMaxCluster;
  static constexpr int kTileB = kBS * Tile::kRowB;
  static constexpr int kWarpRingB = 2 * NS * kTileB;  // K slots then V slots; later the warp's piece
  static constexpr int kPieceFloats = Tile::QH * kD + 2 * Tile::QH;
  static constexpr int kOffBars = NW * kWarpRingB;
  // pieces of the heads that this CTA assembles, one from each CTA: 128 floats, maximum, sum
  static constexpr int kGotFloats = kD + 4, kGot = Tile::QH > kCtas ? Tile::QH : kCtas;
  static constexpr int kOffGot = kOffBars + (NW * 2 * NS * 8 + 15) / 16 * 16;
  // Fused step only: as in MmaCfg, for the one warp that adds the new token and, for the query
  // rows, for all.
  static constexpr int kStageB = (Tile::QH + 2) * Tile::kRowStride + 16;
  static constexpr int kOffStage = kOffGot + kGot * kGotFloats * 4;
  static constexpr int kSmem = 1024 /*align slack*/ + kOffStage;
  static constexpr int kSmemFused = kSmem + NW * kStageB;
  static_assert(kWarpRingB % 1024 == 0 && kWarpRingB >= kPieceFloats * 4, "slots are aligned, and hold a piece");
  static constexpr int kSmB = 228 * 1024, kReservedB = 1024;  // shared memory of an SM; the runtime's part of every CTA
  static_assert(kPerSm * (kSmem + kReservedB) <= kSmB && kPerSmFused * (kSmemFused + kReservedB) <= kSmB,
                "the CTAs that are to share an SM fit it");
};

template <typename Tile, int NW, int NS, bool kFused>
__global__ void __launch_bounds__(32 * NW, 1)
decode_cluster_kernel(const DecodeParams p, const __grid_constant__ CUtensorMap map_k,
                      const __grid_constant__ CUtensorMap map_v) {
  using C = ClusterCfg<Tile, NW, NS>;
  using T = typename Tile::T;
  constexpr int QH = Tile::QH, kRowB = Tile::kRowB;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = int(cluster_rank()), ctas = int(cluster_size());
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kOffBars) + warp * 2 * NS;
  uint8_t* ring = smem + warp * C::kWarpRingB;
  uint8_t* stage = smem + C::kOffStage + warp * C::kStageB;  // fused step only
  if (lane == 0) {
#pragma unroll
    for (int s = 0; s < 2 * NS; ++s) mbar_init(bars + s, 1);
    mbar_fence_init();
    if (Tile::kTensorMaps) {
      prefetch_tensormap(&map_k);
      prefetch_tensormap(&map_v);
    }
  }
  __syncwarp();
  if (ctas > 1) cluster_arrive();  // (waited for before this CTA writes to another's shared memory)
  const int64_t after_wait = grid_wait();
  grid_release();

  // the item, and this warp's share of its blocks: every workers-th one, so that the ids of the first 32 can be
  // asked for together with the length (a table row is there up to its width, whatever the length)
  const int item = int(blockIdx.x) / ctas;
  const int per_seq = p.num_kv_heads * p.head_groups;
  const int b = item / per_seq, sub_item = item - b * per_seq;
  const int kvh = sub_item / p.head_groups, hg = sub_item - kvh * p.head_groups;
  const int heads = min(QH, p.kv_mul - hg * QH);
  const int workers = ctas * NW, worker = rank * NW + warp;
  const int32_t* row =
      p.block_table ? p.block_table + int64_t(p.row_index ? p.row_index[b] : b) * p.max_blocks_per_seq + after_wait : nullptr;
  auto id_at = [&](int i) {  // of the i-th block of the share, 0 beyond the table's width
    const int64_t at = worker + int64_t(i) * workers;
    return row ? (at < p.max_blocks_per_seq ? __ldg(row + at) : 0) : int(at);
  };
  int ids = id_at(lane);  // 32 at a time, one per lane
  const int len = seq_len_of(p, b);
  if (p.block_table && p.seq_lens && item % per_seq == 0 && rank == 0 && tid == 0 &&
      p.seq_lens[b] + p.len_bias > p.max_cached_tokens)
    atomicMax(p.status, KPX_ERR_INVALID_ARGUMENT);
  const int nblk = blocks_of(len);
  const int n = worker < nblk ? (nblk - worker + workers - 1) / workers : 0;
  const uint8_t* q_rows = static_cast<const uint8_t*>(p.q) +
                          (int64_t(b) * p.num_q_heads + int64_t(kvh) * p.kv_mul + hg * QH) * kRowB + after_wait;
  Tile tile;
  tile.init(lane);
  if constexpr (!kFused) tile.load_q(q_rows, kRowB, heads);

  auto check_ids = [&](int first) {
    if (first > 0) ids = id_at(first + lane);
    if (first + lane >= n) {
      ids = 0;
    } else if (ids < 0 || (p.num_blocks > 0 && ids >= p.num_blocks)) {
      atomicMax(p.status, KPX_ERR_INVALID_ARGUMENT);
      ids = 0;
    }
    __syncwarp();
  };
  auto issue = [&](int i, bool withhold = false) {  // K and V tiles of block i of the share
    if ((i & 31) == 0) check_ids(i);
    const int id = __shfl_sync(0xffffffffu, ids, i & 31);
    const int rows = min(kBS, len - (worker + i * workers) * kBS);
#pragma unroll
    for (int kv = 0; kv < 2; ++kv) {
      uint64_t* bar = bars + kv * NS + i % NS;
      uint8_t* dst = ring + (kv * NS + i % NS) * C::kTileB;
      const uint8_t* src = (kv ? p.v_pool : p.k_pool) + int64_t(id) * p.block_stride_b + int64_t(kvh) * p.head_stride_b;
      const bool asked = !(withhold && kv == 0);
      if (Tile::kTensorMaps ? (p.tile_contig || rows == kBS) : p.tile_contig) {
        if (lane == 0) {
          mbar_arrive_expect_tx(bar, C::kTileB);
          if (asked) {
            if (Tile::kTensorMaps) tma_load_5d(dst, kv ? &map_v : &map_k, 0, 0, 0, kvh, id, bar);
            else bulk_g2s(dst, src, C::kTileB, bar);
          }
        }
      } else {  // strided rows: those that exist, one bulk copy each
        if (lane == 0) mbar_arrive_expect_tx(bar, uint32_t(rows) * kRowB);
        __syncwarp();
        if (lane < rows && asked) bulk_g2s(dst + lane * kRowB, src + int64_t(lane) * p.token_stride_b, kRowB, bar);
      }
    }
  };
  for (int i = 0; i < NS && i < n; ++i)
    issue(i, i == 0 && int(blockIdx.x) * NW + warp == p.withhold_worker);

  // The fused step's new token is added by the item's last worker, which also stores its rows.
  const bool takes_token = kFused && worker == workers - 1;
  if constexpr (kFused) {
    if (n > 0 || takes_token) {
      stage_new_token<T, QH, Tile::kRowStride>(
          reinterpret_cast<const T*>(q_rows) - int64_t(hg) * QH * kD, hg, p.kv_mul,
          static_cast<const T*>(p.k_new) + (int64_t(b) * p.num_kv_heads + kvh) * kD + after_wait,
          static_cast<const uint8_t*>(p.v_new) + (int64_t(b) * p.num_kv_heads + kvh) * kRowB + after_wait, takes_token,
          p.sin_cache + int64_t(len) * kD + after_wait, p.cos_cache + int64_t(len) * kD + after_wait,
          row ? row + len / kBS : nullptr, len / kBS, stage, lane);
      __syncwarp();
      tile.load_q(stage, Tile::kRowStride, heads);
      tile.scale_q(p.qscale);
    }
  } else {
    tile.scale_q(p.qscale);  // (the tiles have been requested)
  }

  bool ok = true;
  auto wait_tile = [&](uint64_t* bar, uint32_t phase) {
    const bool here = mbar_wait_bounded(bar, phase, p.wait_limit);
    if (__all_sync(0xffffffffu, here)) return true;
    // Give up: report, then let the copies still in flight land (a bounded pause far longer than
    // one takes); the piece is marked, so that the item's rows come out as NaN.
    if (lane == 0) atomicMax(p.status, KPX_ERR_DEVICE_TIMEOUT);
    for (int k = 0; k < 64; ++k) __nanosleep(1000);
    return false;
  };
  for (int i = 0; i < n && ok; ++i) {
    const uint32_t phase = uint32_t(i / NS) & 1u;
    const int rows = min(kBS, len - (worker + i * workers) * kBS);
    const bool linear = rows < kBS && !p.tile_contig;
    ok = wait_tile(bars + i % NS, phase);
    if (!ok) break;
    tile.scores(ring + (i % NS) * C::kTileB, rows, linear);
    ok = wait_tile(bars + NS + i % NS, phase);
    if (!ok) break;
    tile.output(ring + (NS + i % NS) * C::kTileB, rows, linear);
    __syncwarp();  // both slots are read
    if (i + NS < n) {
      if (lane == 0) fence_proxy_async();
      issue(i + NS);
    }
  }
  tile.finish();
  if constexpr (kFused) {
    if (takes_token) {
      const uint8_t* k_row = stage + QH * Tile::kRowStride;
      const uint8_t* v_row = k_row + Tile::kRowStride;
      tile.add_token(k_row, v_row);
      if (hg == 0) {
        const int id = *reinterpret_cast<const int32_t*>(stage + (QH + 2) * Tile::kRowStride);
        if (id < 0 || (p.num_blocks > 0 && id >= p.num_blocks)) {
          if (lane == 0) atomicMax(p.status, KPX_ERR_INVALID_ARGUMENT);
        } else {
          const int64_t off = int64_t(id) * p.block_stride_b + int64_t(kvh) * p.head_stride_b + int64_t(len % kBS) * p.token_stride_b;
          for (int c = lane; c < kRowB / 8; c += 32) {  // 16-byte chunks of the K row, then of the V row
            const bool is_v = c >= kRowB / 16;
            const int at = (is_v ? c - kRowB / 16 : c) * 16;
            *reinterpret_cast<uint4*>((is_v ? p.v_pool_w : p.k_pool_w) + off + at) =
                *reinterpret_cast<const uint4*>((is_v ? v_row : k_row) + at);
          }
        }
      }
    }
  }
  // ---- the pieces of the CTA's warps, then those of the cluster's CTAs.  A piece without tokens
  // has a sum of 0 and does not count. ----
  float* piece = reinterpret_cast<float*>(ring);
  tile.store(piece);
  __syncwarp();
  if (!ok && lane < QH) piece[QH * kD + QH + lane] = NAN;
  __syncthreads();
  float* got = reinterpret_cast<float*>(smem + C::kOffGot);
  auto write_out = [&](int head, float4 o, float L) {
    const float inv = L == 0.f ? 0.f : 1.f / L;
    T* orow = static_cast<T*>(p.out) + (int64_t(b) * p.num_q_heads + int64_t(kvh) * p.kv_mul + hg * QH + head) * kD;
    Tile::write4(orow, 4 * lane, make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv));
  };
  if (ctas > 1) cluster_wait();  // every CTA of the cluster runs
  for (int head = warp; head < heads; head += NW) {  // a warp per head, a lane four dims
    auto at = [&](int i) { return reinterpret_cast<const float*>(smem + i * C::kWarpRingB); };
    float m[NW], l[NW], M = -INFINITY, L = 0.f;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < NW; ++i) {
      m[i] = at(i)[QH * kD + head];
      l[i] = at(i)[QH * kD + QH + head];
      M = fmaxf(M, m[i]);
    }
#pragma unroll
    for (int i = 0; i < NW; ++i) {
      const float w = l[i] == 0.f ? 0.f : fast_exp2(m[i] - M);
      const float4 v = *reinterpret_cast<const float4*>(at(i) + head * kD + 4 * lane);
      L = fmaf(l[i], w, L);
      o.x = fmaf(v.x, w, o.x);
      o.y = fmaf(v.y, w, o.y);
      o.z = fmaf(v.z, w, o.z);
      o.w = fmaf(v.w, w, o.w);
    }
    if (ctas == 1) {
      write_out(head, o, L);
    } else {
      // Head h is assembled by CTA h modulo the cluster's size.  The pieces are sent there: fetched instead, each
      // would be a trip of its own to another SM (and a second barrier keep the CTAs until all had fetched).
      const uint32_t dst = smem_u32(got + ((head / ctas) * ctas + rank) * C::kGotFloats);
      st_cluster_f4(dst + 16 * lane, head % ctas, o);
      if (lane == 0) st_cluster_f2(dst + kD * 4, head % ctas, M, L);
    }
  }
  if (ctas == 1) return;
  __syncwarp();
  cluster_arrive();
  cluster_wait();
  for (int i = warp; i * ctas + rank < heads; i += NW) {
    const float* pieces = got + i * ctas * C::kGotFloats;
    const bool on = lane < ctas;
    const float m = on ? pieces[lane * C::kGotFloats + kD] : -INFINITY, l = on ? pieces[lane * C::kGotFloats + kD + 1] : 0.f;
    float M = m;
#pragma unroll
    for (int k = C::kCtas / 2; k > 0; k >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, k));
    M = __shfl_sync(0xffffffffu, M, 0);
    const float mine = l == 0.f ? 0.f : fast_exp2(m - M);
    float L = 0.f;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < C::kCtas; ++k) {
      if (k >= ctas) break;
      const float w = __shfl_sync(0xffffffffu, mine, k);
      const float4 v = *reinterpret_cast<const float4*>(pieces + k * C::kGotFloats + 4 * lane);
      L = fmaf(__shfl_sync(0xffffffffu, l, k), w, L);
      o.x = fmaf(v.x, w, o.x);
      o.y = fmaf(v.y, w, o.y);
      o.z = fmaf(v.z, w, o.z);
      o.w = fmaf(v.w, w, o.w);
    }
    write_out(i * ctas + rank, o, L);
  }
}

// A kernel form, made ready on the current device: its shared-memory size and cluster size allowed,
// and how many clusters of 1, 2, 4, 8 and 16 CTAs the device holds at a time.
struct ClusterForm {
  int fit[5] = {0, 0, 0, 0, 0};  // index: log2 of the cluster size
};
template <typename Tile, int NW, int NS, bool kFused>
const ClusterForm* cluster_form() {
  using C = ClusterCfg<Tile, NW, NS>;
  constexpr int smem_bytes = kFused ? C::kSmemFused : C::kSmem;
  static PerDevice<ClusterForm> forms;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  return forms.get(dev, [](ClusterForm& f) {
    auto kern = decode_cluster_kernel<Tile, NW, NS, kFused>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes) != cudaSuccess ||
        cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
      (void)cudaGetLastError();
      return false;
    }
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * NW, smem_bytes) != cudaSuccess) {
      (void)cudaGetLastError();
      return false;
    }
    f.fit[0] = per_sm * device_info().sm_count;
    for (int i = 1; i <= 4; ++i) {
      cudaLaunchAttribute attr{};
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim.x = 1u << i;
      attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3(1u << i);
      cfg.blockDim = dim3(32 * NW);
      cfg.dynamicSmemBytes = smem_bytes;
      cfg.attrs = &attr;
      cfg.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&f.fit[i], kern, &cfg) != cudaSuccess) {
        (void)cudaGetLastError();
        f.fit[i] = 0;
      }
    }
    return true;
  });
}

// CTAs per item of a small launch in this form, 0 if it is not for it: all clusters run side by
// side, and a warp's share stays within max_share blocks; beyond that the balance of the line
// of blocks over all SMs is worth more than the short chain.
inline int cluster_ctas(const DecodeParams& p, const ClusterForm& f, int warps, int max_ctas, int max_share) {
  const int64_t items = int64_t(p.batch) * p.num_kv_heads * p.head_groups;
  const int64_t blocks = seq_blocks_bound(p);
  if (blocks < 0 || items > f.fit[0]) return 0;
  int lg = 0;
  while ((1 << lg) < max_ctas && items <= f.fit[lg + 1] && blocks > (int64_t(warps) << lg)) ++lg;  // no more warps than blocks
  return blocks <= (int64_t(warps) << lg) * max_share ? 1 << lg : 0;
}

// Launches p in the cluster form with NW warps a CTA if it is for it; KPX_ERR_UNIMPLEMENTED if not.
template <typename Tile, int NW, int NS, bool kFused>
int try_cluster_form(const DecodeParams& p, int max_share, cudaStream_t stream) {
  using C = ClusterCfg<Tile, NW, NS>;
  const ClusterForm* form = cluster_form<Tile, NW, NS, kFused>();
  const int ctas = form ? cluster_ctas(p, *form, NW, C::kCtas, max_share) : 0;
  if (ctas == 0) return KPX_ERR_UNIMPLEMENTED;
  CUtensorMap map_k{}, map_v{};
  if (Tile::kTensorMaps) {
    constexpr int32_t dtype = std::is_same<typename Tile::T, __half>::value ? KPX_F16 : KPX_BF16;
    if (!make_pool_map(&map_k, dtype, p.k_pool, p) || !make_pool_map(&map_v, dtype, p.v_pool, p)) return KPX_ERR_CUDA;
  }
  const unsigned grid = unsigned(p.batch * p.num_kv_heads * p.head_groups * ctas);
  return launch_chained_cluster(decode_cluster_kernel<Tile, NW, NS, kFused>, dim3(grid), dim3(32 * NW),
                                kFused ? C::kSmemFused : C::kSmem, unsigned(ctas), stream, p, map_k, map_v);
}
template <typename Tile, int NW, int NS>
int try_cluster(const DecodeParams& p, int max_share, cudaStream_t stream) {
  return p.k_new ? try_cluster_form<Tile, NW, NS, true>(p, max_share, stream)
                 : try_cluster_form<Tile, NW, NS, false>(p, max_share, stream);
}

template <typename T>
int dispatch_decode_mma(DecodeParams p, cudaStream_t stream, int flags) {
  p.head_groups = (p.kv_mul + kMmaHeads - 1) / kMmaHeads;
  const bool small = small_launch(p, kMmaHeads, kMmaWarpsPerSm);
  // Fewer, longer ranges only where a launch is so few items that each would be cut into hundreds of
  // pieces.  us per launch, cut so / as ever: one item of 60000 tokens (4/1 heads fp16) 29 / 38, two (16/2)
  // 33 / 34, four of 40000..50000 39 / 36, 640 of 100..350 tokens (28/4 bf16) 27 / 23, 800 of 20..200
  // (8/8 fp16) 23 / 18.
  p.small = small && int64_t(p.batch) * p.num_kv_heads * p.head_groups < g_small_items ? 1 : 0;
  p.slot_heads = p.kv_mul > 4 ? kMmaHeads : heads_per_warp(p.kv_mul);
  // eight-head slots are twice a four-head slot
  if (p.slot_heads == kMmaHeads) p.partial_slots /= 2;
  if (small && g_cluster_share > 0) {
    // eight warps per item and SM, or four or two where there are more items than SMs
    int rc = try_cluster<MmaTile<T>, 8, 3>(p, g_cluster_share, stream);
    if (rc == KPX_ERR_UNIMPLEMENTED) rc = try_cluster<MmaTile<T>, 4, 3>(p, g_cluster_share, stream);
    if (rc == KPX_ERR_UNIMPLEMENTED) rc = try_cluster<MmaTile<T>, 2, 3>(p, g_cluster_share, stream);
    if (rc != KPX_ERR_UNIMPLEMENTED) return rc;
  }
  // Launches that the caller overlaps on the GPU (KPX_DECODE_OVERLAPPED) run as two CTAs of four
  // warps per SM instead of one of eight: an SM then takes up the next launch's work a half
  // at a time while the previous launch's last warps finish.
  const bool overlapped = (g_decode_variant & 3) == 1 ? true : ((g_decode_variant & 3) == 2 ? false : (flags & KPX_DECODE_OVERLAPPED) != 0);
  const bool small_ctas = overlapped && !small;
  if (p.k_new) return small_ctas ? launch_mma_form<T, 4, 3, 2, true>(p, stream) : launch_mma_form<T, 8, 1, 1, true>(p, stream);
  // (slots per warp: kpx_decode_mma.cuh; launches that overlap keep three, 36 layers on three chains:
  // 6667 GB/s, with two 6643, with one 6153)
  return small_ctas ? launch_mma_form<T, 4, 3, 2, false>(p, stream) : launch_mma_form<T, 8, 1, 1, false>(p, stream);
}

}  // namespace decode
}  // namespace kpx
