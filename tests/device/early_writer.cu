// A caller's kernel that lets the launch behind it start at once, has every SM read `data` through its
// L1 cache, and only then (`cycles` later) lets one block replace it by `src`. Behind it,
// tests/test_gpu_back_to_back.py calls the library on `data`.
#include <cuda_runtime.h>

__global__ void early_writer(float* data, const float* src, float* sink, int n, long long cycles) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  float sum = 0.0f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    float x;
    asm volatile("ld.global.ca.f32 %0, [%1];" : "=f"(x) : "l"(data + i) : "memory");
    sum += x;
  }
  const long long t0 = clock64();
  while (clock64() - t0 < cycles) {}
  if (blockIdx.x == 0)
    for (int i = threadIdx.x; i < n; i += blockDim.x) data[i] = src[i];
  sink[blockIdx.x * blockDim.x + threadIdx.x] = sum;
}

extern "C" int launch_early_writer(float* data, const float* src, float* sink, int n, long long cycles, int blocks, void* stream) {
  early_writer<<<blocks, 256, 0, (cudaStream_t)stream>>>(data, src, sink, n, cycles);
  return (int)cudaGetLastError();
}
