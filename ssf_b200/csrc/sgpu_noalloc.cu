// Jacobi-PCG on a caller-owned device CSR that allocates no device memory.
//
// Some callers of this library cannot allocate GPU memory while they solve:
// a host application that hands the GPU its whole memory pool up front (or
// runs under a custom allocator that owns every device byte), and code that
// must not call cudaMalloc/cudaFree at all because those calls synchronise
// the device and would stall the caller's other streams.  For them this file
// keeps the iteration's work vectors in one file-scope static device array
// of fixed size, created when the library is loaded and held by every GPU
// that loads it until the process exits.  The caller passes the matrix, the
// right-hand side and the solution; nothing else is allocated, by this code
// or by any library it calls (no cudaMalloc, cudaFree, graph, stream or
// event creation).
//
// Limits and sharing:
//  - at most SGPU_NOALLOC_MAX_N equations (131072): the array holds five
//    FP64 vectors of that length plus reduction slots, about 5 MiB;
//  - every call uses the same array, which keeps the last call's contents;
//    the entry point clears what must start at zero (the grid barrier, the
//    reduction tickets, the iteration state) on every call;
//  - calls whose work overlaps on the GPU (two host threads, or two streams
//    of one process, at the same time on the same device) race on the
//    array: serialise them.
//
// Set-up: the array's name in host code is only a host-side stand-in, not a
// device address.  The first call on each device, with that device current,
// asks the runtime for the array's device address (cudaGetSymbolAddress) and
// keeps it; later calls reuse it.
//
// Host waits: every call reads the iteration state back after each chunk of
// iterations (cudaMemcpyAsync + cudaStreamSynchronize), so a call returns
// only when its solve has finished and cannot be recorded into a CUDA graph;
// a call made while its stream is capturing is refused with SGPU_BAD_INPUT
// before anything is enqueued.
//
// Input checks (on the device, before any iteration): every row must satisfy
// 0 <= rowptr[i] <= rowptr[i+1] <= rowptr[n], hold columns in [0, n) and a
// positive diagonal entry; otherwise the call returns SGPU_BAD_INPUT and
// leaves x untouched.  The caller's col/val arrays must hold rowptr[n]
// entries: the checks keep every read inside [0, rowptr[n]).
//
// The iteration (k_pcg_resident, one cooperative launch of a CTA per SM with
// a thread or more per row, hence the largest size; three launches an
// iteration where the device refuses that one or has too few SMs) is the
// reference's symcomprow::cg_prec with the diagonal preconditioner
// (GEFEL/scr.cpp:1093-1205): stop on (r.r)/(f.f) < res, and *ani = i,
// *ares = (r.h)/(f.f) written only on convergence.
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <string>

#include "sgpu_internal.cuh"
#include "sgpu_persist.cuh"

using namespace sgpu;

namespace {

constexpr int kTPB = 256;
constexpr int kMaxN = SGPU_NOALLOC_MAX_N;
constexpr int kBlocks = 148 * 4;  // grid of the input check and of the general form
// iterations of one launch, between two reads of the state: 17 ms on a plate of
// 101,404 equations, 58 ms where three quarters of 8M entries are read from
// global memory each time, longer with more; few enough waits that they cost
// nothing
constexpr long long kChunk = 2048;
constexpr int kGeneralChunk = 16;  // the same of the general form

// byte layout of the scratch array
constexpr size_t kVecBytes = sizeof(double) * (size_t)kMaxN;
constexpr size_t kOffDiag = 0;
constexpr size_t kOffR = kOffDiag + kVecBytes;
constexpr size_t kOffDh = kOffR + kVecBytes;  // pairs {direction, preconditioned residual}
constexpr size_t kOffD = kOffDh + 2 * kVecBytes;
constexpr size_t kOffPart = kOffD + kVecBytes;                          // 2 * kBlocks doubles
constexpr size_t kOffSync = kOffPart + 2 * kBlocks * sizeof(double);
constexpr size_t kOffState = kOffSync + sizeof(GridSync);
constexpr size_t kOffTicket = kOffState + ((sizeof(PcgState) + 255) & ~(size_t)255);  // 4 unsigned
constexpr size_t kScratchBytes = kOffTicket + 256;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

struct Scratch {
  double *diag, *r;
  double2 *dh;  // the general form's product and preconditioned residual
  double *d, *part;
  GridSync *gs;
  PcgState *st;
  unsigned *ticket;
};

Scratch carve(unsigned char *base) {
  Scratch s;
  s.diag = reinterpret_cast<double *>(base + kOffDiag);
  s.r = reinterpret_cast<double *>(base + kOffR);
  s.dh = reinterpret_cast<double2 *>(base + kOffDh);
  s.d = reinterpret_cast<double *>(base + kOffD);
  s.part = reinterpret_cast<double *>(base + kOffPart);
  s.gs = reinterpret_cast<GridSync *>(base + kOffSync);
  s.st = reinterpret_cast<PcgState *>(base + kOffState);
  s.ticket = reinterpret_cast<unsigned *>(base + kOffTicket);
  return s;
}

// device address of the scratch array, per device, found once
std::mutex g_mu;
unsigned char *g_addr[64] = {};

int scratch_address(unsigned char **out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return sgpu::fail(SGPU_CUDA_ERROR, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
  if (dev < 0 || dev >= 64) return sgpu::fail(SGPU_BAD_INPUT, "device ordinal beyond 63");
  std::lock_guard<std::mutex> lk(g_mu);
  if (!g_addr[dev]) {
    void *p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p)
      return sgpu::fail(SGPU_CUDA_ERROR, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
    g_addr[dev] = static_cast<unsigned char *>(p);
  }
  *out = g_addr[dev];
  return SGPU_OK;
}

// clears the state and the reduction tickets (one thread: nothing else of the
// call runs before it)
__global__ void k_na_clear(Scratch s, long long ni, double res, double zero) {
  PcgState z = {};
  z.ni = ni;
  z.res = res;
  z.zero = zero;
  z.crit = SGPU_CRIT_SCR_PREC;
  z.prec = 1;
  z.ani = -1;
  *s.st = z;
  for (int k = 0; k < 4; k++) s.ticket[k] = 0u;
}

// checks every row and extracts the diagonal; a malformed row stops the call
// with SGPU_BAD_INPUT before any product reads the matrix
__global__ void k_na_setup(int n, const int *__restrict__ rowptr, const int *__restrict__ col,
                           const double *__restrict__ val, Scratch s) {
  const int nnz = rowptr[n];
  bool bad = false;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int b = rowptr[i], e = rowptr[i + 1];
    double dv = 0.0;
    if (b < 0 || e < b || e > nnz) {
      bad = true;
    } else {
      bool seen = false;
      for (int k = b; k < e; k++) {
        const int c = col[k];
        if (c < 0 || c >= n) { bad = true; break; }
        if (c == i && !seen) { dv = val[k]; seen = true; }
      }
      if (!(dv > 0.0)) bad = true;  // missing, zero, negative or NaN diagonal
    }
    s.diag[i] = dv;
  }
  if (bad) {  // every writer stores the same values
    s.st->status = SGPU_BAD_INPUT;
    s.st->done = 1;
  }
}

}  // namespace

extern "C" SGPU_API int sgpu_csr_pcg_noalloc_d(int32_t n, const int32_t *rowptr_d, const int32_t *col_d,
                                               const double *val_d, const double *f_d, double *x_d, int64_t ni,
                                               double res, double zero, int64_t iv, void *stream, int64_t *ani,
                                               double *ares, int64_t *iterations) {
  if (n <= 0) return sgpu::fail(SGPU_BAD_INPUT, "n must be positive");
  if (n > kMaxN)
    return sgpu::fail(SGPU_BAD_INPUT, "n = " + std::to_string(n) + " exceeds the no-allocation solver's maximum of " +
                                          std::to_string(kMaxN) + " equations");
  if (!rowptr_d || !col_d || !val_d || !f_d || !x_d) return sgpu::fail(SGPU_BAD_INPUT, "null device pointer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaError_t ce = cudaStreamIsCapturing(st, &cap);
  if (ce != cudaSuccess)
    return sgpu::fail(SGPU_CUDA_ERROR, std::string("cudaStreamIsCapturing: ") + cudaGetErrorString(ce));
  if (cap != cudaStreamCaptureStatusNone)
    return sgpu::fail(SGPU_BAD_INPUT,
                      "the no-allocation solver waits on the host between iterations and cannot run under "
                      "stream capture");
  unsigned char *base = nullptr;
  int rc = scratch_address(&base);
  if (rc != SGPU_OK) return rc;
  const Scratch s = carve(base);
  const int grid = resident_grid();
  bool resident = resident_rows_fit(n, grid);
  k_na_clear<<<1, 1, 0, st>>>(s, (long long)ni, res, zero);
  k_na_setup<<<kBlocks, kTPB, 0, st>>>(n, rowptr_d, col_d, val_d, s);
  sgpu::count_launches(2);
  ResidentArgs a = {};
  a.n = n;
  a.rowptr = rowptr_d;
  a.col = col_d;
  a.val = val_d;
  a.diag = s.diag;
  a.f = f_d;
  a.x = x_d;
  a.r = s.r;
  a.dh = s.dh;
  a.st = s.st;
  a.gs = s.gs;
  a.iv = iv != 0;
  a.most = kChunk;
  const GeneralPcg g = {n,      rowptr_d, col_d, val_d, s.diag, f_d, x_d, s.r, reinterpret_cast<double *>(s.dh) + kMaxN,
                        s.d,    reinterpret_cast<double *>(s.dh), s.st, s.part, s.ticket, kBlocks};
  PcgState h = {};
  auto read = [&](cudaError_t e) {
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, s.st, sizeof(h), cudaMemcpyDeviceToHost, st);
    return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
  };
  cudaError_t e = cudaSuccess;
  for (a.start = 1; resident && e == cudaSuccess && !h.done; a.start = 0) {
    e = cudaMemsetAsync(s.gs, 0, sizeof(GridSync), st);
    if (e == cudaSuccess) e = launch_resident(a, 0, grid, st);
    if (e != cudaSuccess && a.start) {  // refused: fewer SMs for this process than the device has
      cudaGetLastError();
      resident = false;
      e = cudaSuccess;
      break;
    }
    sgpu::count_launches(1);
    e = read(e);
  }
  if (!resident) {
    e = read(e);  // the input check's verdict
    if (e == cudaSuccess && !h.done) general_start(g, iv != 0, st);
    while (e == cudaSuccess && !h.done) {
      general_iterations(g, kGeneralChunk, st);
      e = read(cudaGetLastError());
    }
  }
  if (e != cudaSuccess) return sgpu::fail(SGPU_CUDA_ERROR, std::string("no-allocation PCG: ") + cudaGetErrorString(e));
  if (h.status == SGPU_CUDA_ERROR) return sgpu::fail(SGPU_CUDA_ERROR, "no-allocation PCG: the grid's barrier ran out");
  if (iterations) *iterations = h.it;
  if (h.ani_set) {
    if (ani) *ani = h.ani;
    if (ares) *ares = h.ares;
  }
  return h.status;
}
