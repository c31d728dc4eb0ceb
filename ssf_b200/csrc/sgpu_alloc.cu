// The device-block cache behind DevBuf.
//
// Handles own large device arrays (the CSR and 3x3-block copies of a
// 1M-equation matrix are about 1.5 GB); building and destroying one per solve
// paid cudaMalloc and cudaFree for each, about 10 ms on B200 for the destroy
// alone.  Released blocks are kept here, per device, and handed out again for
// requests that fit them without wasting more than half; a request that
// cudaMalloc cannot meet returns the cached blocks to the driver first.
//
// Ordering: cudaFree waits for the device's outstanding work, and code that
// releases a buffer may rely on that; devmem_put keeps the guarantee with a
// cudaDeviceSynchronize before the block becomes reusable (a handle's end does
// it once for all its blocks, DevIdle).  Contents: memory fresh from
// cudaMalloc reads as zeros in practice and device flags and counters of this
// library start from that, so a reused block is cleared (and the clear
// finished) before it is handed out: on a stream of the cache's own, so that
// what else the device does is not waited for, and for a handle's small blocks
// when the handle ends.  Solving a system of 1,500 equations on a new handle
// (38 blocks) took 2.36 ms with a clear and two waits of the device for each,
// 1.97 without.
#include <map>
#include <mutex>

#include "sgpu_internal.cuh"

namespace sgpu {
namespace {

struct Block {
  void *p;
  int dev;
  bool cleared;  // its clear is queued on the device's clearing stream
};

std::mutex g_mu;
std::multimap<size_t, Block> g_free;  // bytes -> block
size_t g_cached = 0;
constexpr size_t kCacheCap = size_t(24) << 30;  // bytes kept idle at most
constexpr size_t kSmall = size_t(1) << 20;      // cleared at a handle's end; larger ones only when reused
thread_local int g_idle = 0;                    // within DevIdle, and the device was waited for

// the stream that clears a device's blocks (kept for the process), null on failure
constexpr int kDevices = 16;
cudaStream_t clearing(int dev) {
  static std::mutex mu;
  static cudaStream_t st[kDevices] = {};
  if (dev < 0 || dev >= kDevices) return nullptr;
  std::lock_guard<std::mutex> lk(mu);
  if (!st[dev] && cudaStreamCreateWithFlags(&st[dev], cudaStreamNonBlocking) != cudaSuccess) {
    cudaGetLastError();
    st[dev] = nullptr;
  }
  return st[dev];
}

cudaError_t clear(const Block &b, size_t bytes) {
  cudaStream_t s = clearing(b.dev);
  if (!s) {
    const cudaError_t e = cudaMemset(b.p, 0, bytes);
    return e == cudaSuccess ? cudaDeviceSynchronize() : e;
  }
  const cudaError_t e = b.cleared ? cudaSuccess : cudaMemsetAsync(b.p, 0, bytes, s);
  return e == cudaSuccess ? cudaStreamSynchronize(s) : e;
}

size_t round_bytes(size_t b) {
  if (b <= (size_t(1) << 20)) {  // small: powers of two from 512 B
    size_t r = 512;
    while (r < b) r <<= 1;
    return r;
  }
  const size_t g = size_t(2) << 20;  // large: 2 MiB granules
  return (b + g - 1) / g * g;
}

void flush_locked(int dev) {
  for (auto it = g_free.begin(); it != g_free.end();) {
    if (dev < 0 || it->second.dev == dev) {
      int cur = 0;
      cudaGetDevice(&cur);
      if (it->second.dev != cur) cudaSetDevice(it->second.dev);
      cudaFree(it->second.p);
      if (it->second.dev != cur) cudaSetDevice(cur);
      g_cached -= it->first;
      it = g_free.erase(it);
    } else {
      ++it;
    }
  }
}

}  // namespace

cudaError_t devmem_get(void **p, size_t *bytes) {
  const size_t want = round_bytes(*bytes);
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  Block hit{nullptr, 0, false};
  {
    std::lock_guard<std::mutex> lk(g_mu);
    for (auto it = g_free.lower_bound(want); it != g_free.end() && it->first <= 2 * want; ++it) {
      if (it->second.dev != dev) continue;
      hit = it->second;
      *bytes = it->first;
      g_cached -= it->first;
      g_free.erase(it);
      break;
    }
  }
  if (hit.p) {
    *p = hit.p;
    return clear(hit, *bytes);
  }
  e = cudaMalloc(p, want);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();  // clear the sticky-free allocation error
    std::lock_guard<std::mutex> lk(g_mu);
    flush_locked(dev);
    e = cudaMalloc(p, want);
  }
  if (e == cudaSuccess) *bytes = want;
  return e;
}

void devmem_put(void *p, size_t bytes) {
  if (!p) return;
  int dev = 0;
  cudaGetDevice(&dev);
  if (g_idle <= 0 && cudaDeviceSynchronize() != cudaSuccess) {  // a failed context: give the block back
    cudaFree(p);
    return;
  }
  Block b{p, dev, false};
  if (g_idle > 0 && bytes <= kSmall) {
    cudaStream_t s = clearing(dev);
    b.cleared = s && cudaMemsetAsync(p, 0, bytes, s) == cudaSuccess;
  }
  std::lock_guard<std::mutex> lk(g_mu);
  g_free.emplace(bytes, b);
  g_cached += bytes;
  while (g_cached > kCacheCap && !g_free.empty()) {  // drop the largest idle blocks
    auto it = std::prev(g_free.end());
    cudaFree(it->second.p);
    g_cached -= it->first;
    g_free.erase(it);
  }
}

DevIdle::DevIdle() {
  if (g_idle > 0 || cudaDeviceSynchronize() == cudaSuccess) g_idle++;
  else g_idle--;  // every block finds the failed context itself
}
DevIdle::~DevIdle() { g_idle += g_idle > 0 ? -1 : 1; }

}  // namespace sgpu
