// Decode kernels for __half pools: the one place dispatch_decode<__half> is defined.
#include "kpx_decode_cluster.cuh"

namespace kpx {
namespace decode {
template <>
int dispatch_decode<__half>(const DecodeParams& p, cudaStream_t stream, int flags) {
  return dispatch_decode_mma<__half>(p, stream, flags);
}
}  // namespace decode
}  // namespace kpx
