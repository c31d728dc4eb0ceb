// Copies between a caller's host arrays and the device.
//
// cudaMemcpyAsync from pageable memory goes through one staging buffer of the
// driver, filled by the calling thread: 11 GB/s on B200's host, a fifth of
// what the link takes from pinned memory.  Large arrays go through pinned
// slots of our own, which a few threads fill (or empty) while the slots
// before are on the link: 28 GB/s (78 MB of a matrix's storage 7.1 -> 2.8 ms).
// Pinning the 8 MB takes 3.7 ms, once in a process.
//
// The slots belong to the process, one set per device, and are given back
// when it ends; a thread that finds them in use copies the plain way.
#include <atomic>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

#include "sgpu_internal.cuh"

namespace sgpu {
namespace {

constexpr int kThreads = 4;             // copying threads, the caller among them
constexpr size_t kSlot = size_t(1) << 20;
constexpr int kSlots = 2;               // per thread: one on the link, one being filled
constexpr int kDevices = 16;
// Smaller copies gain less than the threads cost.
constexpr size_t kLeast = size_t(4) << 20;

struct Stage {
  std::mutex mu;
  bool tried = false;
  char *mem = nullptr;
  cudaEvent_t ev[kThreads][kSlots] = {};
  ~Stage() {
    if (mem) cudaFreeHost(mem);
  }
  bool ready() {
    if (!tried) {
      tried = true;
      bool ok = true;
      for (auto &t : ev)
        for (cudaEvent_t &e : t) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
      void *p = nullptr;
      if (ok && cudaHostAlloc(&p, kThreads * kSlots * kSlot, cudaHostAllocDefault) == cudaSuccess) mem = (char *)p;
      if (!mem) cudaGetLastError();
    }
    return mem != nullptr;
  }
  char *slot(int t, int k) { return mem + ((size_t)t * kSlots + k) * kSlot; }
};

Stage g_stage[kDevices];

bool pageable(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

struct Job {
  char *dst;
  const char *src;
  size_t bytes;
  cudaStream_t s;
  int dev;
  bool in;
  std::atomic<size_t> next{0};
  std::atomic<int> err{0};
};

// One thread's pieces: the next free piece of the array, through its slots in
// turn.  Thread 0 is the caller, in whatever context it has.
void pieces(Stage &st, Job &j, int t) {
  cudaError_t e = t == 0 ? cudaSuccess : cudaSetDevice(j.dev);
  size_t off[kSlots] = {}, len[kSlots] = {};  // download: what a slot holds
  for (int k = 0; e == cudaSuccess && j.err.load(std::memory_order_relaxed) == 0; k ^= 1) {
    const size_t o = j.next.fetch_add(kSlot), n = o < j.bytes ? (j.bytes - o < kSlot ? j.bytes - o : kSlot) : 0;
    if (n != 0) e = cudaEventSynchronize(st.ev[t][k]);  // what an upload left in the slot is on the device
    if (e != cudaSuccess) break;
    if (j.in) {
      if (n == 0) break;
      memcpy(st.slot(t, k), j.src + o, n);
      e = cudaMemcpyAsync(j.dst + o, st.slot(t, k), n, cudaMemcpyHostToDevice, j.s);
      if (e == cudaSuccess) e = cudaEventRecord(st.ev[t][k], j.s);
    } else {
      if (n != 0) {
        e = cudaMemcpyAsync(st.slot(t, k), j.src + o, n, cudaMemcpyDeviceToHost, j.s);
        if (e == cudaSuccess) e = cudaEventRecord(st.ev[t][k], j.s);
      }
      off[k] = o, len[k] = n;
      const int q = k ^ 1;  // the piece before, while this one travels
      if (e == cudaSuccess && len[q] != 0) {
        e = cudaEventSynchronize(st.ev[t][q]);
        if (e == cudaSuccess) memcpy(j.dst + off[q], st.slot(t, q), len[q]);
        len[q] = 0;
      }
      if (n == 0) break;
    }
  }
  if (e != cudaSuccess) j.err.store((int)e);
}

cudaError_t copy(void *dst, const void *src, size_t bytes, cudaStream_t s, bool in) {
  const cudaMemcpyKind kind = in ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
  int dev = 0;
  // the per-thread default stream is another stream in each of the copying threads
  if (bytes < kLeast || s == cudaStreamPerThread || cudaGetDevice(&dev) != cudaSuccess || dev >= kDevices ||
      !pageable(in ? src : dst))
    return cudaMemcpyAsync(dst, src, bytes, kind, s);
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone)
    return cudaMemcpyAsync(dst, src, bytes, kind, s);
  Stage &st = g_stage[dev];
  std::unique_lock<std::mutex> lk(st.mu, std::try_to_lock);
  if (!lk.owns_lock() || !st.ready()) return cudaMemcpyAsync(dst, src, bytes, kind, s);
  Job j;
  j.dst = (char *)dst, j.src = (const char *)src, j.bytes = bytes, j.s = s, j.dev = dev, j.in = in;
  std::vector<std::thread> others;
  try {
    others.reserve(kThreads - 1);
    for (int t = 1; t < kThreads; t++) others.emplace_back([&st, &j, t]() { pieces(st, j, t); });
  } catch (const std::exception &) {
    // fewer threads then
  }
  pieces(st, j, 0);
  for (std::thread &t : others) t.join();
  if (j.err.load() != 0) {  // once more the plain way, which tells what is wrong
    cudaGetLastError();
    cudaStreamSynchronize(s);
    return cudaMemcpyAsync(dst, src, bytes, kind, s);
  }
  return cudaSuccess;
}

}  // namespace

cudaError_t copy_in(void *dst, const void *src, size_t bytes, cudaStream_t s) { return copy(dst, src, bytes, s, true); }
cudaError_t copy_out(void *dst, const void *src, size_t bytes, cudaStream_t s) {
  return copy(dst, src, bytes, s, false);
}

}  // namespace sgpu
