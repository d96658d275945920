// A launch that the runtime refuses must be reported by the call that made it
// and leave nothing behind for the next check of the runtime's last error.
// The two runtime calls involved are replaced at link time (--wrap), so that
// it needs no GPU and launches nothing.
#include <cstdio>

#include "bk_common.cuh"

static cudaError_t g_last = cudaSuccess;

extern "C" cudaError_t __wrap_cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *, void **) {
  return g_last = cudaErrorInvalidConfiguration;
}
extern "C" cudaError_t __wrap_cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}

__global__ void never_runs() {}

int main() {
  using namespace bk::host;
  if (launch_overlapped(never_runs, 1, 32, 0, nullptr, 1) != (int)cudaErrorInvalidConfiguration)
    return std::puts("the launch's error is not reported"), 1;
  if (launch_status() != BK_OK) return std::puts("a later check reports the failed launch"), 1;
  std::puts("ok");
  return 0;
}
