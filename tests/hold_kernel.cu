// Test infrastructure: a kernel that occupies `blocks` multiprocessors (200 KB of shared memory a block) for `ns`
// nanoseconds and ends by itself (built by tests/test_busy_device.py).
#include <cuda_runtime.h>

__global__ void k_hold(long long ns) {
  long long t0, t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  for (int k = 0; k < 10000000; k++) {
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    if (t - t0 > ns) break;
    __nanosleep(1000);
  }
}

extern "C" int hold(int blocks, long long ns, void* stream) {
  const int smem = 200 * 1024;
  if (cudaFuncSetAttribute(k_hold, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return 1;
  k_hold<<<blocks, 32, smem, (cudaStream_t)stream>>>(ns);
  return cudaGetLastError() != cudaSuccess;
}
