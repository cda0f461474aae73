// Shared memory of the cluster form's kernels against what an SM has: the narrow forms are there for
// launches of more items than SMs, so their CTAs have to share one.  No GPU is used.
#include <cstdio>

#include "kpx_decode_cluster.cuh"
#include "kpx_decode_mma.cuh"

using namespace kpx::decode;

template <typename Tile, int NW, int NS>
int check(const char* name, int want, int want_fused) {
  using C = ClusterCfg<Tile, NW, NS>;
  const int sm = 228 * 1024, reserved = 1024;  // bytes; the runtime's share of every CTA
  const int plain = sm / (C::kSmem + reserved), fused = sm / (C::kSmemFused + reserved);
  std::printf("%s, %d warps: %d plain, %d fused CTAs of %d and %d bytes\n", name, NW, plain, fused, C::kSmem, C::kSmemFused);
  return plain < want || fused < want_fused;
}

int main() {
  int bad = 0;
  bad |= check<MmaTile<__half>, 8, 3>("fp16", 1, 1) | check<MmaTile<__half>, 4, 3>("fp16", 2, 2) | check<MmaTile<__half>, 2, 3>("fp16", 4, 3);
  bad |= check<MmaTile<__nv_bfloat16>, 4, 3>("bf16", 2, 2) | check<MmaTile<__nv_bfloat16>, 2, 3>("bf16", 4, 3);
  bad |= check<FmaTile<1>, 3, 2>("fp32, 1 head", 2, 2) | check<FmaTile<2>, 3, 2>("fp32, 2 heads", 2, 2) | check<FmaTile<4>, 3, 2>("fp32, 4 heads", 2, 2);
  return bad;
}
