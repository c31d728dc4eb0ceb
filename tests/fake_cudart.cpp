// A stand-in for the CUDA runtime on a machine without a device: "device"
// memory is host memory and every copy is done at once.  It records which
// thread issues a copy on which stream, and can make the n-th call of a
// function fail.  For the tests of the library's host code.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

namespace {
std::mutex mu;
std::map<std::string, int> calls, failing;
thread_local cudaError_t last = cudaSuccess;
std::vector<std::pair<std::thread::id, cudaStream_t>> copies;

cudaError_t call(const char *name) {
  std::lock_guard<std::mutex> lk(mu);
  const int k = ++calls[name];
  const auto f = failing.find(name);
  if (f != failing.end() && (f->second == 0 || f->second == k)) return last = cudaErrorUnknown;
  return cudaSuccess;
}
}  // namespace

extern "C" {
// makes call number n (from 1; 0: every one) of a function fail
void fake_fail(const char *name, int n) { std::lock_guard<std::mutex> lk(mu); calls.clear(); failing[name] = n; }
void fake_reset() { std::lock_guard<std::mutex> lk(mu); calls.clear(); failing.clear(); copies.clear(); last = cudaSuccess; }
int fake_calls(const char *name) { std::lock_guard<std::mutex> lk(mu); return calls[name]; }
int fake_last_error() { return (int)last; }
// copies recorded on the stream by other threads than the caller
int fake_foreign_copies(void *stream) {
  std::lock_guard<std::mutex> lk(mu);
  int k = 0;
  for (auto &c : copies) k += c.second == (cudaStream_t)stream && c.first != std::this_thread::get_id();
  return k;
}

cudaError_t cudaGetLastError() { cudaError_t e = last; last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t) { return "made to fail"; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return call("cudaGetDevice"); }
cudaError_t cudaSetDevice(int) { return call("cudaSetDevice"); }
cudaError_t cudaDeviceSynchronize() { return call("cudaDeviceSynchronize"); }
cudaError_t cudaMalloc(void **p, size_t n) { *p = calloc(1, n); return call("cudaMalloc"); }
cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { *p = malloc(n); return call("cudaHostAlloc"); }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemset(void *p, int v, size_t n) { memset(p, v, n); return call("cudaMemset"); }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { memset(p, v, n); return call("cudaMemsetAsync"); }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return call("cudaMemcpy"); }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  const cudaError_t e = call("cudaMemcpyAsync");
  if (e == cudaSuccess) memcpy(d, s, n);
  std::lock_guard<std::mutex> lk(mu);
  copies.emplace_back(std::this_thread::get_id(), st);
  return e;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  const cudaError_t e = call("cudaStreamCreateWithFlags");
  *s = e == cudaSuccess ? (cudaStream_t)malloc(1) : nullptr;
  return e;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { free((void *)s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return call("cudaStreamSynchronize"); }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *c) { *c = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return call("cudaStreamWaitEvent"); }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)malloc(1); return call("cudaEventCreate"); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = (cudaEvent_t)malloc(1); return call("cudaEventCreateWithFlags"); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free((void *)e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return call("cudaEventRecord"); }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return call("cudaEventSynchronize"); }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return call("cudaEventElapsedTime"); }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
  memset(a, 0, sizeof(*a));
  a->type = cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
}
