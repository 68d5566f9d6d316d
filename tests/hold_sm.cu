// A kernel that keeps one multiprocessor to itself for a given time (one block
// of 1,024 threads with most of its shared memory).  It waits for nothing but
// the clock.
#include <cuda_runtime.h>
#include <stdint.h>

__global__ void __launch_bounds__(1024) hold_kernel(uint64_t ns) {
  uint64_t t0, t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  do {
    __nanosleep(1000);
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  } while (t - t0 < ns);
}

extern "C" int hold_sm(uint64_t ns, void *stream) {
  constexpr int kBytes = 200 << 10;
  cudaError_t e =
      cudaFuncSetAttribute(hold_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
  if (e != cudaSuccess) return static_cast<int>(e);
  hold_kernel<<<1, 1024, kBytes, static_cast<cudaStream_t>(stream)>>>(ns);
  return static_cast<int>(cudaGetLastError());
}
