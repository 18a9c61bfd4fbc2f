// launch_after of ptx.jl_b200/csrc/host_common.h on a runtime of its own, for tests/test_launch_after.py:
// prints what it hands to the runtime, and what a failed launch returns and leaves behind.
#include <cstdio>

#include "host_common.h"

static cudaError_t g_next = cudaSuccess, g_last = cudaSuccess;

extern "C" cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* cfg, const void* kernel, void** args) {
  std::printf("launch %u %u %zu %d %d", cfg->gridDim.x, cfg->blockDim.x, cfg->dynamicSmemBytes, **reinterpret_cast<int**>(args),
              kernel != nullptr);
  for (unsigned i = 0; i < cfg->numAttrs; ++i) {
    const cudaLaunchAttribute& a = cfg->attrs[i];
    if (a.id == cudaLaunchAttributeProgrammaticStreamSerialization) std::printf(" after %d", a.val.programmaticStreamSerializationAllowed);
    if (a.id == cudaLaunchAttributeClusterDimension) std::printf(" cluster %u", a.val.clusterDim.x);
  }
  std::printf("\n");
  if (g_next != cudaSuccess) g_last = g_next;
  return g_next;
}

extern "C" cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}

static void kernel(int) {}

int main() {
  ptxb200::launch_after(nullptr, kernel, 3u, 128u, 4096, 1u, 7);
  ptxb200::launch_after(nullptr, kernel, 8u, 64u, 0, 4u, 9);
  for (cudaError_t e : {cudaSuccess, cudaErrorInvalidValue, cudaErrorStreamCaptureInvalidated}) {
    g_next = e;
    const int returned = ptxb200::launch_after(nullptr, kernel, 1u, 32u, 0, 1u, 1);
    std::printf("returned %d expected %d left %d\n", returned, (int)e, (int)cudaGetLastError());
  }
}
