// Holds some SMs for a while: one CTA each with all of the SM's shared memory,
// which ends by itself.  For test_gpu_beside_other_work.py.
#include <cuda_runtime.h>

namespace {
cudaStream_t stream;

__global__ void __launch_bounds__(1024, 1) k_hold(long long ns) {
  extern __shared__ char all[];
  long long t0, t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  do {
    __nanosleep(20000);
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  } while (t - t0 < ns && t >= t0);
  if (ns < 0) all[threadIdx.x] = (char)t;
}
}  // namespace

// ns at most 5 s
extern "C" int hold_sms(int ctas, long long ns) {
  const int bytes = 227 * 1024;
  cudaError_t e = cudaFuncSetAttribute(k_hold, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && !stream) e = cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) {
    k_hold<<<ctas, 1024, bytes, stream>>>(ns < 5000000000ll ? ns : 5000000000ll);
    e = cudaGetLastError();
  }
  return (int)e;
}
extern "C" int release() { return (int)cudaStreamSynchronize(stream); }
