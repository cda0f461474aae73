// A refused launch: its status is returned and nothing stays behind for the next error check of the
// process.  The runtime's two calls are stood in for at link time, so that no GPU is needed.
#include <cstdio>

#include "kpx_common.cuh"

static cudaError_t pending = cudaSuccess;
extern "C" cudaError_t __wrap_cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) {
  return pending = cudaErrorInvalidConfiguration;
}
extern "C" cudaError_t __wrap_cudaGetLastError() {
  const cudaError_t e = pending;
  pending = cudaSuccess;
  return e;
}

static __global__ void kernel(int) {}
static int tried() {
  KPX_CUDA_TRY(__wrap_cudaLaunchKernelExC(nullptr, nullptr, nullptr));
  return KPX_OK;
}

int main() {
  int bad = 0;
  auto check = [&](const char* what, int rc) {
    if (rc != KPX_ERR_CUDA || pending != cudaSuccess) {
      std::printf("%s: status %d, pending error %d\n", what, rc, int(pending));
      bad = 1;
    }
    pending = cudaSuccess;
  };
  check("launch_chained", kpx::launch_chained(kernel, dim3(1), dim3(32), 0, nullptr, 1));
  check("launch_chained_cluster", kpx::launch_chained_cluster(kernel, dim3(8), dim3(32), 0, 8, nullptr, 1));
  check("KPX_CUDA_TRY", tried());
  return bad;
}
