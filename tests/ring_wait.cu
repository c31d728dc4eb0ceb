// One warp waits on an mbarrier with a limit of its own per lane, after or
// while another warp completes it, or never: which lanes were told that it
// was done.  For test_gpu_ring_wait.py.
#include "sgpu_persist.cuh"

namespace {
__global__ void k_wait(int mode, const int *limit, int *got) {
  __shared__ unsigned long long bar;
  if (threadIdx.x == 0)
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sgpu::ring_u32(&bar)) : "memory");
  __syncthreads();
  if (mode == 0 && threadIdx.x == 32)  // done before the wait
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sgpu::ring_u32(&bar)) : "memory");
  __syncthreads();
  if (threadIdx.x < 32) {
    got[threadIdx.x] = sgpu::ring_landed(sgpu::ring_wait(&bar, 0, limit[threadIdx.x])) ? 1 : 0;
  } else if (mode == 1 && threadIdx.x == 32) {  // done about 0.2 ms into the wait
    const long long t0 = clock64();
    while (clock64() - t0 < 400000) {
    }
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sgpu::ring_u32(&bar)) : "memory");
  }
  __syncthreads();
}
}  // namespace

extern "C" int ring_wait_answers(int mode, const int *limit, int *got) {
  int *d = nullptr;
  cudaError_t e = cudaMalloc(&d, 64 * sizeof(int));
  if (e == cudaSuccess) e = cudaMemcpy(d, limit, 32 * sizeof(int), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_wait<<<1, 64>>>(mode, d, d + 32);
    e = cudaMemcpy(got, d + 32, 32 * sizeof(int), cudaMemcpyDeviceToHost);
  }
  cudaFree(d);
  return (int)e;
}
