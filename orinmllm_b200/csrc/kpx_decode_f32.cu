// Decode kernels for float pools: the one place dispatch_decode<float> is defined.
#include "kpx_decode_impl.cuh"

namespace kpx {
namespace decode {
template <>
int dispatch_decode<float>(const DecodeParams& p, cudaStream_t stream, int flags) {
  switch (heads_per_warp(p.kv_mul)) {
    case 1: return launch_shape<float, 1>(p, stream, flags);
    case 2: return launch_shape<float, 2>(p, stream, flags);
    default: return launch_shape<float, 4>(p, stream, flags);
  }
}
}  // namespace decode
}  // namespace kpx
