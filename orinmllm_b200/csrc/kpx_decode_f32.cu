// Decode kernels for float pools: the one place dispatch_decode<float> is defined.
#include "kpx_decode_cluster.cuh"

namespace kpx {
namespace decode {
namespace {
template <int QH>
int launch_shape(DecodeParams p, cudaStream_t stream, int flags) {
  p.head_groups = (p.kv_mul + QH - 1) / QH;
  if (small_launch(p, QH, 6)) {
    if (g_cluster_share > 0) {
      // (half the share of 16-bit caches: a block is twice the bytes)
      int rc = try_cluster<FmaTile<QH>, 6, 2>(p, (g_cluster_share + 1) / 2, stream);
      if (rc == KPX_ERR_UNIMPLEMENTED) rc = try_cluster<FmaTile<QH>, 3, 2>(p, (g_cluster_share + 1) / 2, stream);
      if (rc != KPX_ERR_UNIMPLEMENTED) return rc;
    }
    return launch_decode<float, QH, 6, 2, 8, true>(p, stream);
  }
  // Launches that the caller overlaps on the GPU (KPX_DECODE_OVERLAPPED) run as three small CTAs
  // per SM instead of one large one: an SM then takes up the next launch's work a third at a
  // time while the previous launch's last warps finish.  Alone, the large CTA is faster.
  return (flags & KPX_DECODE_OVERLAPPED) ? launch_decode<float, QH, 2, 2, 8, false, 3>(p, stream)
                                         : launch_decode<float, QH, 6, 2, 8>(p, stream);
}
}  // namespace

template <>
int dispatch_decode<float>(const DecodeParams& p, cudaStream_t stream, int flags) {
  switch (heads_per_warp(p.kv_mul)) {
    case 1: return launch_shape<1>(p, stream, flags);
    case 2: return launch_shape<2>(p, stream, flags);
    default: return launch_shape<4>(p, stream, flags);
  }
}
}  // namespace decode
}  // namespace kpx
