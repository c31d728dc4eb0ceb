// Aggregation multilevel preconditioner: the hierarchy shared by the
// single-vector solve (sgpu_amg.cu) and the many-load-case solve
// (sgpu_amg_multi.cu).
#pragma once

#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "sgpu_internal.cuh"

namespace sgpu {

// Device buffers of the hierarchy come from the device's stream-ordered
// memory pool (the pool keeps freed memory, so building a hierarchy for a new
// handle -- a batch solved handle after handle -- does not pay for cudaMalloc
// and cudaFree and their device synchronisation).  The stream is the handle's,
// set by the AMG entry points (amg_stream) before any allocation; a buffer is
// freed on the stream it was allocated on, after the work queued there.
extern thread_local cudaStream_t amg_stream;

template <class T>
struct PBuf {
  T *p = nullptr;
  size_t n = 0;
  cudaStream_t s = nullptr;
  PBuf() = default;
  PBuf(const PBuf &) = delete;
  PBuf &operator=(const PBuf &) = delete;
  ~PBuf() { release(); }
  void release() {
    if (p) cudaFreeAsync(p, s);
    p = nullptr;
    n = 0;
  }
  int alloc(size_t count) {
    if (count <= n && p) return SGPU_OK;
    release();
    if (count == 0) count = 1;
    s = amg_stream;
    cudaError_t e = cudaMallocAsync((void **)&p, count * sizeof(T), s);
    if (e != cudaSuccess) return fail(SGPU_CUDA_ERROR, std::string("cudaMallocAsync: ") + cudaGetErrorString(e));
    n = count;
    return SGPU_OK;
  }
};

template <typename T>
struct LevelVecs {
  PBuf<T> b, x, x2, r, d, d2, res;
  int alloc(size_t n) {
    SGPU_TRY(b.alloc(n));
    SGPU_TRY(x.alloc(n));
    SGPU_TRY(x2.alloc(n));
    SGPU_TRY(r.alloc(n));
    SGPU_TRY(d.alloc(n));
    SGPU_TRY(d2.alloc(n));
    SGPU_TRY(res.alloc(n));
    return SGPU_OK;
  }
};

struct AmgLevel {
  int nb = 0, b = 0, n = 0;
  int64_t nblk = 0;
  int layout = 0;  // 0 owned row-major blocks, 1 handle BSR3, 2 handle CSR
  const int *browptr = nullptr, *bcol = nullptr;
  PBuf<int> own_browptr, own_bcol;
  PBuf<double> val64;  // owned coarse values (FP64), or the level-0 scaled FP64 copy
  PBuf<float> val32;   // owned coarse values (FP32)
  PBuf<double> dinv64;
  PBuf<float> dinv32;
  PBuf<double> dsq64;  // sqrt(dinv): the symmetric scaling of the Lanczos operator
  PBuf<float> dsq32;
  bool unit_diag = false;
  double lmax64 = 0.0, lmax32 = 0.0;
  // transfer to the next level
  int na = 0, k = 0;
  PBuf<int> agg, aggptr, aggnodes;
  PBuf<double> Q64;
  PBuf<float> Q32;
  LevelVecs<double> v64;
  LevelVecs<float> v32;
  // FP32 cycle: values converted, and the slot of this level's smoother
  // bound among the Lanczos runs on the set-up's second stream (-1: none)
  bool val32_ready = false;
  int lz_slot = -1;
};

// The coarse levels of a cycle as a list of steps on the device
// (k_coarse_program), recorded at the start of a solve.
struct CoarseProgram {
  bool current = false;  // recorded for the solve under way (nsteps 0: none)
  int nsteps = 0, block = 0, grid = 0;
  void *result = nullptr;  // level 1's iterate after it
  DevBuf<unsigned char> steps;
};

struct Amg {
  int k0 = 0;             // near-null-space vectors given (0: translations)
  PBuf<double> B0;      // n x k0 as given
  bool built = false;     // hierarchy (FP64 set-up) current
  bool have32 = false;    // FP32 copies current
  bool have64 = false;    // FP64 level-0 scaled copy current
  std::vector<AmgLevel *> lv;
  int nc = 0;             // coarsest (dense) equations
  PBuf<double> M64;
  PBuf<float> M32;
  PBuf<double> cb64, cx64;
  PBuf<float> cb32, cx32;
  // options: Chebyshev degree, coarse-correction weight, smoothing interval
  // [lmax/ratio, 1.1 lmax], largest dense coarsest level, coarse visits per
  // level (1: V-cycle, 2: W-cycle), Lanczos steps of the lmax estimate
  int deg = 1;
  // alpha 1.9: 39 iterations on the 1.01M-DOF cantilever against 41 at 1.7,
  // 33 against 36 on a 362k-DOF plate, 31 against 32 on a 96^3 lognormal
  // conduction cube (all FP32 cycle, true residual 1e-10)
  double ratio = 30.0, alpha = 1.9;
  int coarse_max = 768;
  int dense_max = 4096;  // larger coarsest levels are smoothed, not inverted
  int bottom_deg = 8;    // Chebyshev steps of such a bottom level
  int gamma = 2;       // visits of level 1 per level-0 cycle
  int gamma_deep = 2;  // visits of level l+1 per level-l cycle, l >= 1
  int lanczos_steps = 14;
  // batched independent systems (sgpu_matrix_pcg_batch_agg): the level-0 last
  // smoothing step writes the per-row products z r and z q here
  double *batch_zr = nullptr, *batch_zq = nullptr;
  // level objects by depth, kept when a hierarchy is discarded so that a
  // rebuild of the same matrix reuses their device buffers
  std::vector<AmgLevel *> pool;
  // the level-0 smoother bound of an FP32 cycle, run on a second stream
  // while the aggregation set-up runs on the handle's (amg_build); its
  // workspace stays with the handle
  cudaStream_t side = nullptr;
  cudaEvent_t fork = nullptr;
  bool l0_bound_pending = false;
  bool l0_bound_wanted = false;
  DevBuf<float> lz32;    // 5 vectors of n
  DevBuf<double> lz_ab;  // Lanczos coefficients
  // the coarse smoothing levels' bounds, run on the second stream beside the
  // dense coarsest inverse: 5 vectors of each level, 129 coefficients each
  DevBuf<float> lzc32;
  DevBuf<double> lzc_ab;
  int lzc_levels = 0;
  // Level 0 of the FP32 cycle with half-precision values (3x3 block rows
  // only): every block row padded to a multiple of four blocks (padding:
  // value 0, the row's own column), values component-major per padded row,
  // so that a lane reads one component of four blocks in one 8-byte load.
  // The padded pattern is kept for the handle's life (the pattern of a handle
  // never changes); the values are converted at every FP32 set-up.
  bool want_fp32 = false;  // the set-up under way is for the FP32 cycle
  bool h16_struct = false, h16_vals = false;
  int64_t h16_nblk = 0;     // stored blocks, padding included
  DevBuf<int> h16ptr, h16col;
  DevBuf<uint16_t> h16val;  // IEEE binary16 bit patterns
  CoarseProgram prog32, prog64;
  DevBuf<unsigned char> prog_sync;  // the programs' grid barrier
  ~Amg() {
    for (AmgLevel *l : pool) delete l;
    if (side) {
      cudaStreamSynchronize(side);
      cudaStreamDestroy(side);
    }
    if (fork) cudaEventDestroy(fork);
  }
  void clear() {
    lv.clear();
    built = have32 = have64 = false;
    h16_vals = false;
  }
  AmgLevel *take_level(size_t depth) {
    while (pool.size() <= depth) pool.push_back(new AmgLevel());
    AmgLevel *l = pool[depth];
    l->unit_diag = false;
    l->browptr = l->bcol = nullptr;
    l->val32_ready = false;
    l->lz_slot = -1;
    return l;
  }
};


// Chebyshev smoothing on [lmax/ratio, 1.1 lmax] of D^-1 A: the first step's
// 1/theta and the recurrence coefficients of steps 1..deg-1
struct Cheb {
  double c2_first;             // 1/theta
  double c1[8], c2[8];         // steps 1..deg-1
};

inline Cheb cheb_coeffs(double lmax, double ratio, int deg) {
  Cheb c{};
  const double a = lmax / ratio, b = 1.1 * lmax;
  const double theta = 0.5 * (b + a), delta = 0.5 * (b - a), sigma = theta / delta;
  c.c2_first = 1.0 / theta;
  double rho = 1.0 / sigma;
  for (int k = 1; k < deg && k < 8; k++) {
    const double rn = 1.0 / (2.0 * sigma - rho);
    c.c1[k] = rn * rho;
    c.c2[k] = 2.0 * rn / delta;
    rho = rn;
  }
  return c;
}

template <typename T>
const T *level_vals(const sgpu_matrix m, const AmgLevel &L);
template <>
inline const float *level_vals<float>(const sgpu_matrix m, const AmgLevel &L) {
  if (L.layout == 1) return m->bsr.bval32s.p;
  if (L.layout == 2) return m->csr.val32s.p;
  return L.val32.p;
}
template <>
inline const double *level_vals<double>(const sgpu_matrix m, const AmgLevel &L) {
  return L.val64.p;  // level 0: the scaled FP64 copy; coarse: owned values
}

template <typename T>
const T *level_dinv(const AmgLevel &L);
template <>
inline const float *level_dinv<float>(const AmgLevel &L) { return L.unit_diag ? nullptr : L.dinv32.p; }
template <>
inline const double *level_dinv<double>(const AmgLevel &L) { return L.unit_diag ? nullptr : L.dinv64.p; }

// Builds the hierarchy if the handle has none (set-up in FP64) and the copies
// of the requested cycle precision; set-up device time into *setup_ms.
int amg_ensure(sgpu_matrix m, bool fp32, float *setup_ms);

// A solve's iterations: the first ones launched one kernel after the other,
// the rest as a graph of kChunk of them, launched again while the one before
// it still runs.  The host reads `done` of a finished launch on a second
// stream meanwhile, so the device never waits for it; the kernels of what is
// queued past the end return at once.  A conditional WHILE node around one
// iteration (the form before) puts a gap between iterations, and graphs of 8
// with the host in between (the batches' form before) one between graphs:
// 129,480 equations in FP64 9.05 -> 8.67 ms, 1.01M mixed 24.1 -> 23.7, 64
// load cases 41.0 -> 40.2, 256 plates 63.1 -> 61.4.
class Iterations {
 public:
  Iterations() = default;
  Iterations(const Iterations &) = delete;
  Iterations &operator=(const Iterations &) = delete;
  ~Iterations() {
    for (cudaEvent_t e : mark_)
      if (e) cudaEventSynchronize(e), cudaEventDestroy(e);  // the graph may still run
    if (exec_) cudaGraphExecDestroy(exec_);
    if (own_) cudaStreamDestroy(own_);
  }

  // `iteration` launches one iteration on s; done: the solver state's flag
  // (set by the kernels, never cleared by them), at most max_iters iterations.
  // poll: a stream that is idle now, or null.  s may still have queued kernels
  // on return, all of which see `done`.
  template <class Body>
  int run(cudaStream_t s, cudaStream_t poll, const int *done, int64_t max_iters, Body iteration) {
    const char *lm = getenv("SGPU_FCG_LOOP");
    const bool ahead = !(lm && !strcmp(lm, "chunk"));  // chunk: the host tests before every launch
    if (!poll) {
      if (!own_) SGPU_CUDA(cudaStreamCreateWithFlags(&own_, cudaStreamNonBlocking));
      poll = own_;
    }
    for (cudaEvent_t &e : mark_)
      if (!e) SGPU_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    int64_t queued = 0;
    bool stop = false;
    SGPU_CUDA(cudaEventRecord(mark_[0], s));
    if (!exec_) {
      if (ahead)
        for (; queued < 2; queued++) SGPU_TRY(iteration());
      SGPU_TRY(read(poll, mark_[0], done, &stop));  // converged at the start: no graph
      if (stop || queued >= max_iters) return SGPU_OK;
      SGPU_TRY(capture(s, kChunk, iteration));
    }
    for (int k = 0; !stop && queued < max_iters; k ^= 1) {
      if (!ahead) SGPU_TRY(read(poll, mark_[k ^ 1], done, &stop));
      if (stop) break;
      SGPU_CUDA(cudaGraphLaunch(exec_, s));
      count_launches(nodes_);
      SGPU_CUDA(cudaEventRecord(mark_[k], s));
      queued += kChunk;
      if (ahead && queued > 2 + kChunk) SGPU_TRY(read(poll, mark_[k ^ 1], done, &stop));
    }
    return SGPU_OK;
  }

 private:
  // 1, 2 and 4 take the same time to a percent; a longer graph takes longer to
  // make and leaves more behind the end
  static constexpr int kChunk = 2;

  static int read(cudaStream_t poll, cudaEvent_t mark, const int *done, bool *stop) {
    int flag = 0;
    SGPU_CUDA(cudaStreamWaitEvent(poll, mark, 0));
    SGPU_CUDA(cudaMemcpyAsync(&flag, done, sizeof(int), cudaMemcpyDeviceToHost, poll));
    SGPU_CUDA(cudaStreamSynchronize(poll));
    *stop = flag != 0;
    return SGPU_OK;
  }

  template <class Body>
  int capture(cudaStream_t s, int count, Body iteration) {
    cudaGraph_t g;
    const int64_t before = sgpu_kernel_launches();
    SGPU_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeRelaxed));
    int rc = SGPU_OK;
    for (int it = 0; it < count && rc == SGPU_OK; it++) rc = iteration();
    cudaError_t e = cudaStreamEndCapture(s, &g);
    nodes_ = sgpu_kernel_launches() - before;
    count_launches(-nodes_);  // captured launches run (and are counted) at each replay
    if (e != cudaSuccess)
      return rc != SGPU_OK ? rc : fail(SGPU_CUDA_ERROR, std::string("cudaStreamEndCapture: ") + cudaGetErrorString(e));
    if (rc == SGPU_OK) e = cudaGraphInstantiate(&exec_, g, 0);
    cudaGraphDestroy(g);
    if (rc != SGPU_OK) return rc;
    if (e != cudaSuccess) {
      exec_ = nullptr;
      return fail(SGPU_CUDA_ERROR, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e));
    }
    return SGPU_OK;
  }

  cudaGraphExec_t exec_ = nullptr;
  int64_t nodes_ = 0;
  cudaEvent_t mark_[2] = {nullptr, nullptr};
  cudaStream_t own_ = nullptr;
};

}  // namespace sgpu
