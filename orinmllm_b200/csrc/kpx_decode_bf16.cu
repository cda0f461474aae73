// Decode kernels for __nv_bfloat16 pools: the one place dispatch_decode<__nv_bfloat16> is defined.
#include "kpx_decode_cluster.cuh"

namespace kpx {
namespace decode {
template <>
int dispatch_decode<__nv_bfloat16>(const DecodeParams& p, cudaStream_t stream, int flags) {
  return dispatch_decode_mma<__nv_bfloat16>(p, stream, flags);
}
}  // namespace decode
}  // namespace kpx
