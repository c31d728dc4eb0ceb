// Jacobi-PCG as one resident grid.
//
// A small system's iteration is bound by latency, not by bytes: as three
// launches with a serial sum of the block partials, an iteration of a
// 101,404-equation plate (1.8M entries, 22 MB) took 77 us on B200, of which
// reading its matrix needs 3.  Here the whole iteration runs inside one
// cooperative launch of one CTA per SM and costs one gather and two grid
// barriers: 8.1 us on that plate (162.8 -> 16.9 ms for its 2094 iterations),
// 6.4 to 7 us on systems of 1500 to 24,000 equations.
#pragma once

#include <algorithm>
#include <cstdlib>

#include "sgpu_internal.cuh"

namespace sgpu {

// ---------------------------------------------------------------------------
// grid barrier that also sums
// ---------------------------------------------------------------------------
// Every CTA stores its partial sums, adds to an arrival counter (release) and
// one thread polls the counter (acquire); the first warp then reads all
// partials.  Sums of even and odd barriers have their own slots: a CTA writes
// those of barrier e + 2 only after every CTA has arrived at e + 1, so after
// it has read those of e.  All CTAs add the same values in the same order, so
// every thread of the grid gets the same bits and the control flow that
// follows is uniform.  Measured on 148 CTAs of 1024 threads: 2.3 us, of which
// the CTA's own reduction 0.7; polling 148 flagged partials directly (no
// counter) took 4.1 us, with 148 x 148 polls in flight.
//
// The launch is cooperative: it starts once all its CTAs can run at the same
// time (with 20 SMs held by another kernel for 4.5 s, a solve began after
// those and took as long as ever), so a poll waits for the grid's own CTAs
// only.  It still has a limit, after which the CTA gives up (the others then
// run out too) and the caller reports SGPU_CUDA_ERROR.
constexpr int kPollLimit = 1 << 22;  // about 3 s of polls
constexpr int kMaxGrid = 256;        // CTAs the slots hold

struct GridSync {  // in global memory, zeroed before each launch
  unsigned arrived;
  unsigned pad[31];
  double part[2][2][kMaxGrid];  // parity, sum, CTA
};

__device__ __forceinline__ double persist_warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

struct GridSumShared {
  double part[2][32];  // per warp
  double tot[2];
  int ok;  // written by thread 0 in each barrier
};

// thread 0: arrives and waits until every CTA has; false: gave up
__device__ __forceinline__ bool grid_arrive_wait(GridSync *gs, unsigned target) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&gs->arrived) : "memory");
  unsigned c;
  for (int tries = 0; tries < kPollLimit; tries++) {
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(&gs->arrived) : "memory");
    if (c >= target) return true;
  }
  return false;
}

// v: the thread's partial sums in, the grid's sums out (every thread); e: the
// number of this barrier in the launch, from 1.  Orders every global write
// before it (of all CTAs) before every read after it.  False: gave up.
template <int NV>
__device__ __forceinline__ bool grid_barrier_sum(double (&v)[NV], GridSync *gs, unsigned e, GridSumShared &sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int G = gridDim.x;
#pragma unroll
  for (int q = 0; q < NV; q++) {
    v[q] = persist_warp_sum(v[q]);
    if (lane == 0) sh.part[q][w] = v[q];
  }
  __syncthreads();
  if (w == 0) {
    double t[NV];
#pragma unroll
    for (int q = 0; q < NV; q++) t[q] = persist_warp_sum(lane < nw ? sh.part[q][lane] : 0.0);
    if (lane == 0) {
#pragma unroll
      for (int q = 0; q < NV; q++) __stcg(&gs->part[e & 1][q][blockIdx.x], t[q]);
      sh.ok = grid_arrive_wait(gs, e * (unsigned)G);
    }
    __syncwarp();
    double s[NV];
#pragma unroll
    for (int q = 0; q < NV; q++) s[q] = 0.0;
#pragma unroll
    for (int u = 0; u < kMaxGrid / 32; u++) {
      const int k = lane + 32 * u;
      if (k < G) {
#pragma unroll
        for (int q = 0; q < NV; q++) s[q] += __ldcg(&gs->part[e & 1][q][k]);
      }
    }
#pragma unroll
    for (int q = 0; q < NV; q++) {
      s[q] = persist_warp_sum(s[q]);
      if (lane == 0) sh.tot[q] = s[q];
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NV; q++) v[q] = sh.tot[q];
  return sh.ok != 0;
}

// The barrier alone (same counter, same numbering).
__device__ __forceinline__ bool grid_barrier(GridSync *gs, unsigned e, GridSumShared &sh) {
  __syncthreads();
  if (threadIdx.x == 0) sh.ok = grid_arrive_wait(gs, e * gridDim.x);
  __syncthreads();
  return sh.ok != 0;
}

// ---------------------------------------------------------------------------
// scalars of the iteration
// ---------------------------------------------------------------------------
// The state of the solve, one copy per CTA in shared memory.  Every thread
// evaluates the same tests on the same sums (so no broadcast is needed) and
// thread 0 alone records the outcome; a thread keeps only r.h and beta in
// registers.  What thread 0 writes here is read by the others after the next
// grid barrier at the earliest.
struct CgShared {
  PcgState s;
  __device__ __forceinline__ void load(const PcgState *st) {
    if (threadIdx.x == 0) s = *st;
  }
  // f.f and r.h of the start (scr.cpp:1117-1120: a zero right-hand side is
  // reported and the iteration goes on to the zero denominator;
  // cr.cpp:1160-1164 returns at once); true: stop
  __device__ __forceinline__ bool begin(double ff, double rh) {
    const bool zero_rhs = ff < s.zero;
    const bool stop = (zero_rhs && s.crit == SGPU_CRIT_CR_PREC) || s.ni <= 0;
    if (threadIdx.x == 0) {
      s.nory = ff;
      s.nom = rh;
      s.beta = 0.0;
      s.it = 0;
      if (zero_rhs) {
        s.status = SGPU_ZERO_RHS;
        s.ares = ff;
        s.ani = 0;
        s.ani_set = 1;
      }
      if (stop) s.done = 1;
    }
    return stop;
  }
  // denom = d.p: the breakdown test (scr.cpp:1146-1151, cr.cpp:1177-1181)
  // and alpha; true: stop
  __device__ __forceinline__ bool direction(double dp, double nom, double &alpha) {
    const bool stop = fabs(dp) < s.zero;
    alpha = nom / dp;
    if (threadIdx.x == 0) {
      s.denom = dp;
      if (stop) {
        s.ani = s.it;
        s.ares = nom;
        s.ani_set = 1;
        if (s.status == 0) s.status = SGPU_BREAKDOWN;
        s.done = 1;
      } else {
        s.alpha = alpha;
      }
    }
    return stop;
  }
  // r.r and r.h after the update: beta and the routine's stopping test at
  // iteration it (counted from 0); true: stop (or pause, for SGPU_CRIT_TRUE:
  // the host confirms on the true residual)
  __device__ __forceinline__ bool updated(double rr, double rh, long long it, double &nom, double &beta) {
    beta = rh / nom;
    const int crit = s.crit;
    bool conv;
    if (crit == SGPU_CRIT_SCR_PREC) conv = fabs(rr / s.nory) < s.res;    // scr.cpp:1188
    else if (crit == SGPU_CRIT_CR_PREC) conv = sqrt(rh / s.nory) < s.res;  // cr.cpp:1217
    else conv = rr < s.tol2 * s.nory;
    const bool last = it + 1 >= s.ni;
    if (threadIdx.x == 0) {
      s.rr = rr;
      s.rho_prev = nom;
      s.beta = beta;
      s.nom = rh;
      s.it = it + 1;
      if (conv) {
        s.ani = it;
        s.ares = crit == SGPU_CRIT_CR_PREC ? rh : rh / s.nory;
        s.ani_set = 1;
        if (crit == SGPU_CRIT_TRUE) s.pause = 1;
        else s.done = 1;
      } else if (last) {
        s.done = 1;
        if (s.status == 0) s.status = SGPU_NOT_CONVERGED;
        if (crit == SGPU_CRIT_CR_PREC) {
          s.ani = s.ni;
          s.ares = rh;
          s.ani_set = 1;
        }
      }
    }
    nom = rh;
    return conv || last;
  }
};

// ---------------------------------------------------------------------------
// the resident iteration
// ---------------------------------------------------------------------------
// T lanes own one row for the whole solve: its x, r, h, d and diagonal entry
// stay in their registers and its matrix entries in shared memory (lane s of
// a row has entries s, s + T, ...; a warp's entries are stored slot by slot,
// so a warp reads one contiguous segment per slot).  T is the largest power
// of two that still gives every row of the CTA its lanes, so a small system
// spreads its rows over many lanes and a large one has a thread per row.
//
// Per iteration:
//   gather  y = A d with d = beta d_old + h formed at the gather from the
//           16-byte pairs dh[c] = {d_old, h}: one load per entry instead of
//           a second barrier between the direction update and the product
//   barrier d.y -> alpha
//   update  x, r, h in registers; dh[i] = {d, h} for the next gather
//   barrier r.r, r.h -> beta, stopping test
//
// Warps whose entries do not fit the CTA's shared memory read them from the
// CSR arrays each iteration, eight lanes to a row (105,840 equations with 8M
// entries, where a quarter fits: 28.5 us an iteration).
//
// The kernel starts the solve itself (start != 0: r = f - A x0) and runs at
// most `most` iterations; x and r then go back to memory, so that the next
// launch goes on.  x_in for the start is read when iv != 0.
constexpr int kResidentTPB = 1024;

struct ResidentArgs {
  int n;
  const int *rowptr, *col;
  const double *val, *diag, *f;
  double *x, *r;
  double2 *dh;
  PcgState *st;
  GridSync *gs;
  int rows_per_cta;  // <= kResidentTPB / T
  int cap;           // matrix entries the dynamic shared memory holds
  int start, iv;
  long long most;
};

// what one gather of the iteration reads
struct GatherDir {
  const double2 *dh;
  double beta;
  __device__ __forceinline__ double operator()(int c) const {
    const double2 g = dh[c];
    return fma(beta, g.x, g.y);
  }
};
struct GatherPlain {
  const double *x;
  __device__ __forceinline__ double operator()(int c) const { return x[c]; }
};

// y of the lane's row (valid in all T lanes of the row)
template <int T, class X>
__device__ __forceinline__ double resident_product(const ResidentArgs &a, bool resident, int slots, const double *sv,
                                                   const int *sc, int i, bool active, const X &x) {
  const int lane = threadIdx.x & 31;
  double y = 0.0;
  if (resident) {
#pragma unroll 6
    for (int s = 0; s < slots; s++) y = fma(sv[32 * s], x(sc[32 * s]), y);
#pragma unroll
    for (int o = T / 2; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
    return y;
  }
  // 8 lanes per row (T, where more lanes own a row), 32 / 8 rows of the warp at a time
  constexpr int L = T < 8 ? 8 : T, RPW = 32 / L, ROWS = 32 / T;
  const int sub = lane % L, g = lane / L;
  const int i0 = __shfl_sync(0xffffffffu, i, 0);
  const unsigned act = __ballot_sync(0xffffffffu, active);
#pragma unroll 1
  for (int q = 0; q < ROWS; q += RPW) {
    const int lr = q + g;  // row of the warp, owned by lanes T lr ...
    const int row = i0 + lr;
    double s = 0.0;
    if ((act >> (T * lr)) & 1u) {
      const int b = a.rowptr[row], e = a.rowptr[row + 1];
#pragma unroll 4
      for (int k = b + sub; k < e; k += L) s = fma(a.val[k], x(a.col[k]), s);
    }
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    // the owners of rows q .. q + RPW - 1 take their sums
    const int mine = lane / T;
    const double t = __shfl_sync(0xffffffffu, s, ((mine - q) & (RPW - 1)) * L);
    if (mine >= q && mine < q + RPW) y = t;
  }
  return y;
}

template <int T>
__global__ void __launch_bounds__(kResidentTPB, 1) k_pcg_resident(const ResidentArgs a) {
  extern __shared__ double dyn[];
  __shared__ GridSumShared sums;
  __shared__ CgShared cg;
  __shared__ int woff[kResidentTPB / 32 + 1];
  double *sval = dyn;
  int *scol = reinterpret_cast<int *>(dyn + a.cap);
  if (a.st->done | a.st->pause) return;  // the same in every CTA: this grid writes it after its last barrier
  cg.load(a.st);
  const int prec = a.st->prec;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int lrow = threadIdx.x / T, sub = threadIdx.x % T;
  const int i = blockIdx.x * a.rows_per_cta + lrow;
  const bool active = lrow < a.rows_per_cta && i < a.n;
  const bool owner = active && sub == 0;

  // the rows' entries into shared memory
  int b = 0, len = 0;
  if (active) {
    b = a.rowptr[i];
    len = a.rowptr[i + 1] - b;
  }
  const int slots = len > sub ? (len - sub + T - 1) / T : 0;
  int ws = slots;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ws = max(ws, __shfl_xor_sync(0xffffffffu, ws, o));
  if (lane == 0) woff[w + 1] = 32 * min(ws, a.cap / 32 + 1);
  if (threadIdx.x == 0) woff[0] = 0;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int k = 0; k < kResidentTPB / 32; k++) woff[k + 1] = min(woff[k] + woff[k + 1], a.cap + 32);
  __syncthreads();
  const bool resident = woff[w + 1] <= a.cap;
  const double *sv = sval + woff[w] + lane;
  const int *sc = scol + woff[w] + lane;
  if (resident) {
    double *wv = sval + woff[w] + lane;
    int *wc = scol + woff[w] + lane;
#pragma unroll 4
    for (int s = 0; s < slots; s++) {
      wv[32 * s] = a.val[b + sub + T * s];
      wc[32 * s] = a.col[b + sub + T * s];
    }
  }

  unsigned epoch = 0;
  double xi = 0.0, ri = 0.0, hi = 0.0, di = 0.0, dg = 1.0, nom, beta;
  long long it = a.start ? 0 : a.st->it;
  bool ok = true, stop = false;
  if (active && prec) dg = a.diag[i];
  if (a.start) {
    if (a.iv && active) xi = a.x[i];
    double y = 0.0;
    if (a.iv) y = resident_product<T>(a, resident, slots, sv, sc, i, active, GatherPlain{a.x});
    double v[2] = {0.0, 0.0};
    if (active) {
      const double fi = a.f[i];
      ri = fi - y;
      hi = prec ? ri / dg : ri;
      if (owner) {
        a.dh[i] = make_double2(0.0, hi);
        v[0] = fi * fi;
        v[1] = ri * hi;
      }
    }
    ok = grid_barrier_sum<2>(v, a.gs, ++epoch, sums);
    stop = cg.begin(v[0], v[1]);
    nom = v[1];
    beta = 0.0;
  } else {
    nom = a.st->nom;
    beta = a.st->beta;
    if (active) {
      xi = a.x[i];
      ri = a.r[i];
      const double2 g = a.dh[i];
      di = g.x;
      hi = g.y;
    }
  }

  for (long long k = 0; ok && !stop && k < a.most; k++, it++) {
    // y = A d, d.y
    const double y = resident_product<T>(a, resident, slots, sv, sc, i, active, GatherDir{a.dh, beta});
    di = fma(beta, di, hi);
    double v1[1] = {owner ? di * y : 0.0}, alpha;
    ok = grid_barrier_sum<1>(v1, a.gs, ++epoch, sums);
    if (!ok || cg.direction(v1[0], nom, alpha)) break;
    double v[2] = {0.0, 0.0};
    if (active) {
      xi = fma(alpha, di, xi);
      ri = fma(-alpha, y, ri);
      hi = prec ? ri / dg : ri;
      if (owner) {
        a.dh[i] = make_double2(di, hi);
        v[0] = ri * ri;
        v[1] = ri * hi;
      }
    }
    ok = grid_barrier_sum<2>(v, a.gs, ++epoch, sums);
    if (!ok) break;
    stop = cg.updated(v[0], v[1], it, nom, beta);
  }
  if (owner) {
    a.x[i] = xi;
    a.r[i] = ri;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (!ok) {
      cg.s.status = SGPU_CUDA_ERROR;
      cg.s.done = 1;
    }
    *a.st = cg.s;
  }
}

// CTAs of a resident grid on the current device: one per SM.  SGPU_SMS=<n>
// states how many SMs the process may count on where it has only a share of
// the device's (read at every solve).
inline int resident_grid() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 0;
  if (const char *e = getenv("SGPU_SMS")) sms = std::max(0, atoi(e));
  return sms < kMaxGrid ? sms : kMaxGrid;
}
constexpr int kResidentSmem = 220 * 1024;  // beside about 1.2 KB of static shared memory
constexpr int kResidentCap = kResidentSmem / 12;

template <int T>
inline cudaError_t launch_resident_t(const ResidentArgs &a, int grid, cudaStream_t s) {
  const size_t smem = (size_t)a.cap * 12;
  cudaError_t e = cudaFuncSetAttribute(k_pcg_resident<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kResidentSmem);
  if (e != cudaSuccess) return e;
  ResidentArgs args = a;
  void *p[] = {&args};
  return cudaLaunchCooperativeKernel((const void *)k_pcg_resident<T>, dim3(grid), dim3(kResidentTPB), p, smem, s);
}

// Whether n rows have a thread each in the resident grid.
inline bool resident_rows_fit(int64_t n, int grid) { return grid > 0 && n <= (int64_t)grid * kResidentTPB; }

// Lanes that share a row of the resident grid.
inline int resident_lanes(int n, int grid) {
  const int rows = (n + grid - 1) / grid;  // of a CTA
  int t = 1;
  while (t < 32 && 2 * t * rows <= kResidentTPB) t *= 2;
  return t;
}

// nnz: entries of the matrix where the host knows them (twice a CTA's share
// is asked for, the rest of the SM's memory stays L1), else 0
inline cudaError_t launch_resident(ResidentArgs a, int64_t nnz, int grid, cudaStream_t s) {
  int64_t cap = kResidentCap;
  if (nnz > 0) cap = std::min<int64_t>(cap, 2 * (nnz / grid) + 2048);
  a.cap = (int)cap & ~31;
  a.rows_per_cta = (a.n + grid - 1) / grid;
  const int lanes = resident_lanes(a.n, grid);
  grid = (a.n + a.rows_per_cta - 1) / a.rows_per_cta;  // no CTA without rows
  switch (lanes) {
    case 1: return launch_resident_t<1>(a, grid, s);
    case 2: return launch_resident_t<2>(a, grid, s);
    case 4: return launch_resident_t<4>(a, grid, s);
    case 8: return launch_resident_t<8>(a, grid, s);
    case 16: return launch_resident_t<16>(a, grid, s);
    default: return launch_resident_t<32>(a, grid, s);
  }
}

// ---------------------------------------------------------------------------
// the streaming iteration: matrices that do not fit the SMs
// ---------------------------------------------------------------------------
// One cooperative launch of a CTA per SM; a CTA owns a contiguous range of
// rows.  Per iteration:
//   product  p = A d over the CTA's rows, d.p
//   barrier  alpha
//   update   r, h over the CTA's rows; r.r, r.h
//   barrier  beta, stopping test
//   x += alpha d (the last iteration's too), d = beta d + h
//   barrier
//
// The matrix arrives by bulk copies (cp.async.bulk on an mbarrier) into
// stages that belong to one warp each: a warp multiplies a tile, then its
// lane 0 starts the copy of the tile `depth` ahead into the same stage.  The
// order never ends: behind the last tile of an iteration comes the first of
// the next, so the copies run on through the barriers and the vector phases,
// and HBM works while the three-launch form had ramps, tails and gaps.  The
// gathers of d stay plain loads (d changes between barriers); evict-first
// copies leave L2 to the vectors.
//
// Measured per iteration (B200), against three launches per iteration in a
// graph: 1,008,600 equations in 3x3 blocks (683 MB) 149.7 -> 123 us, of which
// the bytes take 104.5; 132,300 equations (84 MB, in L2) 33.1 -> 21.9 us;
// 481,200 equations of CSR (104 MB) 39.4 -> 27.1 us; 2,130,048 of CSR (640 MB)
// 196 -> 165 us.  x is updated with d, which both read, and not with r, which
// d has to wait for.  Variants that lost: plain loads instead of bulk copies
// (152 us on the first), evict-last copies (157), 12 or 24 warps (133 to 139
// there; on CSR of 2,130,048 equations 12 warps 178, 20 warps 165 to 168), the
// vector phases as functions of their own (CSR of 481,200 equations 31.8).  A
// second stage per warp (LPR 16) lost to wider tiles (139): a tile's gathers,
// not its copy, are what a warp waits for.
__device__ __forceinline__ unsigned ring_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool ring_test(unsigned long long *bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(ring_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait of a thread (a try_wait suspends for up to about a microsecond).
// The lanes of a warp may get different answers, since a copy can land between
// the last polls of two of them: they vote before they part (ring_landed).
__device__ __forceinline__ bool ring_wait(unsigned long long *bar, unsigned parity, int limit = kPollLimit) {
  for (int tries = 0; tries < limit; tries++)
    if (ring_test(bar, parity)) return true;
  return false;
}
// Whether a copy has landed for every lane of the warp.  It stands where the
// lanes meet anyway, behind the work on the copy (that of the lanes that saw it
// land): a vote at the wait itself took 25.8 us an iteration on 262,144 rows of
// 27 entries, this 22.3.
__device__ __forceinline__ bool ring_landed(bool mine) { return __all_sync(0xffffffffu, mine); }

// A matrix as units of rows: block rows of 3 (BSR3, values component-major
// per block row) or single rows (CSR).  The arrays are readable for 16 bytes
// past their last entry.
struct TileMat {
  int units;
  const int *ptr;  // units + 1
  const int *col;
  const double *val;
  int per;    // units of a CTA
  int ent;    // entries a stage holds: the most any tile has
  int depth;  // stages of a warp
};

// ROWS 1: CSR, ROWS 3: BSR3; LPR lanes per unit, tiles of 32 / LPR units.
template <int ROWS, int LPR>
struct TileKind {
  static constexpr int kRows = ROWS;
  static constexpr int kLpr = LPR;
  static constexpr int kUnits = 32 / kLpr;
  static constexpr int kVals = ROWS * ROWS;
  __host__ __device__ static constexpr int val_bytes(int ent) { return (8 * (kVals * ent + 2) + 15) & ~15; }
  __host__ __device__ static constexpr int stage_bytes(int ent) { return val_bytes(ent) + ((4 * (ent + 6) + 15) & ~15); }
};

struct TileArgs {
  int n;
  const double *diag;
  double *x, *r, *h, *d, *p;
  PcgState *st;
  GridSync *gs;
  long long most;
};

// The vector phases over the rows [r0, r1) of the CTA.  A thread's loads of
// two rows are in flight together (its stores may alias its next loads for all
// the compiler knows, so a plain loop has one row's); of four, the registers
// cost the product more than it gives (1,008,600 equations in 3x3 blocks 128
// us an iteration, with one row 126.5, with two 121.5).
constexpr int kRowBatch = 2;
template <int TPBX>
__device__ __forceinline__ double2 tiles_residual(double *r, double *h, const double *p, const double *diag, double alpha,
                                               int r0, int r1) {  // r -= alpha p, h = r / diag; r.r, r.h
  double2 v = {0.0, 0.0};
  for (int i0 = r0 + threadIdx.x; i0 < r1; i0 += kRowBatch * TPBX) {
    double rv[kRowBatch], pv[kRowBatch], g[kRowBatch];
#pragma unroll
    for (int z = 0; z < kRowBatch; z++) {
      const int i = i0 + z * TPBX;
      if (i < r1) rv[z] = r[i], pv[z] = p[i], g[z] = diag ? __ldg(diag + i) : 1.0;
    }
#pragma unroll
    for (int z = 0; z < kRowBatch; z++) {
      const int i = i0 + z * TPBX;
      if (i < r1) {
        const double ri = fma(-alpha, pv[z], rv[z]);
        const double hi = diag ? ri / g[z] : ri;
        r[i] = ri;
        h[i] = hi;
        v.x += ri * ri;
        v.y += ri * hi;
      }
    }
  }
  return v;
}
template <int TPBX>
__device__ __forceinline__ void tiles_direction(double *x, double *d, const double *h, double alpha, double beta,
                                             bool stop, int r0, int r1) {  // x += alpha d, d = beta d + h
  for (int i0 = r0 + threadIdx.x; i0 < r1; i0 += kRowBatch * TPBX) {
    double xv[kRowBatch], dv[kRowBatch], hv[kRowBatch];
#pragma unroll
    for (int z = 0; z < kRowBatch; z++) {
      const int i = i0 + z * TPBX;
      if (i < r1) xv[z] = x[i], dv[z] = d[i], hv[z] = h[i];
    }
#pragma unroll
    for (int z = 0; z < kRowBatch; z++) {
      const int i = i0 + z * TPBX;
      if (i < r1) {
        x[i] = fma(alpha, dv[z], xv[z]);
        if (!stop) d[i] = fma(beta, dv[z], hv[z]);
      }
    }
  }
}

template <int ROWS, int LPR, int TPBX>
__global__ void __launch_bounds__(TPBX, 1) k_pcg_tiles(const TileArgs a, const TileMat m) {
  using K = TileKind<ROWS, LPR>;
  constexpr int kTileWarps = TPBX / 32;
  extern __shared__ __align__(128) unsigned char ring[];
  __shared__ GridSumShared sums;
  __shared__ CgShared cg;
  __shared__ int bad;
  if (a.st->done | a.st->pause) return;  // the same in every CTA: this grid writes it after its last barrier
  const int D = m.depth, vb = K::val_bytes(m.ent), sb = K::stage_bytes(m.ent);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned char *stages = ring + (size_t)w * D * sb;
  unsigned long long *full = reinterpret_cast<unsigned long long *>(ring + (size_t)kTileWarps * D * sb) + w * D;
  int *sp = reinterpret_cast<int *>(ring + (size_t)kTileWarps * D * (sb + 8));
  const int u0 = blockIdx.x * m.per, nu = min(m.per, m.units - u0);  // >= 1: no CTA without units
  const int ntiles = (nu + K::kUnits - 1) / K::kUnits;
  const int mine = ntiles > w ? (ntiles - w + kTileWarps - 1) / kTileWarps : 0;  // the warp's tiles
  cg.load(a.st);
  for (int q = threadIdx.x; q <= nu; q += TPBX) sp[q] = m.ptr[u0 + q];
  if (lane == 0)
    for (int q = 0; q < D; q++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(ring_u32(full + q)) : "memory");
  if (threadIdx.x == 0) bad = 0;
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  const int prec = a.st->prec;
  double nom = a.st->nom, beta = a.st->beta;
  long long it = a.st->it;
  __syncthreads();

  unsigned long long policy;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  // lane 0: copies the warp's tile number j into stage q
  auto issue = [&](int j, int q) {
    const int t = w + kTileWarps * j;
    const int e0 = sp[t * K::kUnits], e1 = sp[min((t + 1) * K::kUnits, nu)];
    const long long v0 = ((long long)K::kVals * e0) & ~1ll, v1 = ((long long)K::kVals * e1 + 1) & ~1ll;
    const int c0 = e0 & ~3, c1 = (e1 + 3) & ~3;
    const unsigned nv = (unsigned)(8 * (v1 - v0)), nc = (unsigned)(4 * (c1 - c0));
    unsigned char *dst = stages + (size_t)q * sb;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(ring_u32(full + q)), "r"(nv + nc)
                 : "memory");
    if (nv)
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
          ::"r"(ring_u32(dst)), "l"(m.val + v0), "r"(nv), "r"(ring_u32(full + q)), "l"(policy)
          : "memory");
    if (nc)
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
          ::"r"(ring_u32(dst + vb)), "l"(m.col + c0), "r"(nc), "r"(ring_u32(full + q)), "l"(policy)
          : "memory");
  };
  int next = 0;       // the warp's next tile to copy (0 .. mine - 1, then the next iteration's first)
  int q = 0;          // stage of the next tile to read
  unsigned ph = 0;    // its phase
  if (mine && lane == 0)
    for (int z = 0; z < D; z++) {
      issue(next, z);
      if (++next == mine) next = 0;
    }

  const int r0 = u0 * K::kRows, r1 = (u0 + nu) * K::kRows;
  unsigned epoch = 0;
  bool ok = true;
  for (long long k = 0; k < a.most; k++, it++) {
    double acc = 0.0;
    for (int j = 0; j < mine; j++) {
      const int t = w + kTileWarps * j;
      const bool landed = ring_wait(full + q, ph);
      const unsigned char *stage = stages + (size_t)q * sb;
      const int t0 = t * K::kUnits, e0 = sp[t0];
      const double *vals = reinterpret_cast<const double *>(stage) + ((K::kVals * e0) & 1);
      const int *cols = reinterpret_cast<const int *>(stage + vb) + (e0 & 3);
      const int sub = lane % LPR, u = t0 + lane / LPR;
      if constexpr (ROWS == 1) {
        double y = 0.0, y2 = 0.0;
        if (landed && u < nu) {
          const int b = sp[u] - e0, len = sp[u + 1] - e0 - b;
          const double *v = vals + b;
          const int *c = cols + b;
          constexpr int U = LPR == 2 ? 9 : 4;
          for (int e = sub; e < len; e += LPR * U) {
            double xx[U];
#pragma unroll
            for (int z = 0; z < U; z++) xx[z] = a.d[c[min(e + LPR * z, len - 1)]];
#pragma unroll
            for (int z = 0; z < U; z++) {
              if (e + LPR * z < len) {
                if (z & 1) y2 = fma(v[e + LPR * z], xx[z], y2);
                else y = fma(v[e + LPR * z], xx[z], y);
              }
            }
          }
          y += y2;
        }
        if (!ring_landed(landed)) {
          bad = 1;
          break;
        }
#pragma unroll
        for (int o = LPR / 2; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o, LPR);
        if (sub == 0 && u < nu) {
          a.p[u0 + u] = y;
          acc += a.d[u0 + u] * y;
        }
      } else {
        double y0 = 0.0, y1 = 0.0, y2 = 0.0;
        if (landed && u < nu) {
          const int s = sp[u] - e0, nbr = sp[u + 1] - e0 - s;
          const double *v = vals + 9 * s;
          const int *c = cols + s;
          constexpr int U = LPR == 8 ? 4 : (LPR == 16 ? 2 : 1);
          for (int e = sub; e < nbr; e += LPR * U) {
            double x0[U], x1[U], x2[U];
#pragma unroll
            for (int z = 0; z < U; z++) {
              const double *xp = a.d + 3 * c[min(e + LPR * z, nbr - 1)];
              x0[z] = xp[0];
              x1[z] = xp[1];
              x2[z] = xp[2];
            }
#pragma unroll
            for (int z = 0; z < U; z++) {
              const int jj = e + LPR * z;
              if (jj < nbr) {
                y0 += v[jj] * x0[z] + v[nbr + jj] * x1[z] + v[2 * nbr + jj] * x2[z];
                y1 += v[3 * nbr + jj] * x0[z] + v[4 * nbr + jj] * x1[z] + v[5 * nbr + jj] * x2[z];
                y2 += v[6 * nbr + jj] * x0[z] + v[7 * nbr + jj] * x1[z] + v[8 * nbr + jj] * x2[z];
              }
            }
          }
        }
        if (!ring_landed(landed)) {
          bad = 1;
          break;
        }
        double y[3] = {y0, y1, y2};
        const double yv = RowSums<3, LPR>::sum(y, sub);
        if (RowSums<3, LPR>::first(sub) && u < nu) {
          const int i = 3 * (u0 + u) + RowSums<3, LPR>::row_of_lane(sub);
          a.p[i] = yv;
          acc += a.d[i] * yv;
        }
      }
      __syncwarp();  // the stage is read: the warp's next copy may overwrite it
      if (lane == 0) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        issue(next, q);
        if (++next == mine) next = 0;
      }
      if (++q == D) {
        q = 0;
        ph ^= 1;
      }
    }
    double dp[1] = {acc}, alpha;
    ok = grid_barrier_sum<1>(dp, a.gs, ++epoch, sums) && !bad;
    if (!ok || cg.direction(dp[0], nom, alpha)) break;
    const double2 t = tiles_residual<TPBX>(a.r, a.h, a.p, prec ? a.diag : nullptr, alpha, r0, r1);
    double v[2] = {t.x, t.y};
    ok = grid_barrier_sum<2>(v, a.gs, ++epoch, sums);
    const bool stop = !ok || cg.updated(v[0], v[1], it, nom, beta);
    tiles_direction<TPBX>(a.x, a.d, a.h, alpha, beta, stop, r0, r1);
    if (stop) break;
    ok = grid_barrier(a.gs, ++epoch, sums);
    if (!ok) break;
  }
  // the copies that nobody reads
  if (mine && lane == 0)
    for (int z = 0; z < D; z++) {
      ring_wait(full + q, ph);
      if (++q == D) {
        q = 0;
        ph ^= 1;
      }
    }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (!ok) {
      cg.s.status = SGPU_CUDA_ERROR;
      cg.s.done = 1;
    }
    *a.st = cg.s;
  }
}

// The rule of the launch: the fewest lanes per unit whose stages (one per
// warp at least) fit.  Fewer lanes mean wider tiles, fewer shuffles and more
// gathers in flight per lane; the longest unit decides whether they fit
// (8 lanes up to 41 blocks a row, 16 up to 82, 32 up to 164 of BSR3; 2 lanes up
// to 66 entries a row, 8 up to 265, 32 up to 704 of CSR).  16 warps of up to 128
// registers; the rows that 32 lanes share, in which every warp has only its
// own row's gathers in flight, run 24 (60,000 rows of 401 entries 89.3 us an
// iteration with 16 warps, 79.4 with 24).  With 24 warps throughout, whose
// stages are shorter, 300,000 rows of 55 entries took 63.2 us (8 lanes)
// against 50.7 (2 lanes), 100,000 of 201 entries 89.8 (32) against 69.7 (8).
constexpr int kTileRing = 200 * 1024;    // stages
constexpr int kTileSmem = 225 * 1024;    // with the unit pointers
template <int ROWS, int LPR>
constexpr int kTileTPB = ROWS == 1 && LPR == 32 ? 768 : 512;

template <int ROWS, int LPR>
inline bool tiles_fit(const TileMat &m, int longest, int sms) {
  using K = TileKind<ROWS, LPR>;
  const int ent = (longest * K::kUnits + 3) & ~3, per = (m.units + sms - 1) / sms;
  const int64_t stage = (int64_t)kTileTPB<ROWS, LPR> / 32 * (K::stage_bytes(ent) + 8);
  return longest > 0 && longest < 4096 && stage <= kTileRing && stage + 4ll * (per + 1) <= kTileSmem;
}

// Stages of a warp, as many as fit beside the unit pointers (and are of use).
template <int ROWS, int LPR>
inline int tile_stages(const TileMat &m, int longest, int sms) {
  using K = TileKind<ROWS, LPR>;
  const int W = kTileTPB<ROWS, LPR> / 32, ent = (longest * K::kUnits + 3) & ~3, per = (m.units + sms - 1) / sms;
  const int ntiles = (per + K::kUnits - 1) / K::kUnits, room = std::min(kTileRing, kTileSmem - 4 * (per + 1));
  return std::min(room / (W * (K::stage_bytes(ent) + 8)), (ntiles + W - 1) / W + 1);
}

template <int ROWS, int LPR>
inline cudaError_t launch_tiles_as(const TileArgs &a, TileMat m, int longest, int sms, cudaStream_t s) {
  using K = TileKind<ROWS, LPR>;
  constexpr int TPBX = kTileTPB<ROWS, LPR>, W = TPBX / 32;
  m.ent = (longest * K::kUnits + 3) & ~3;
  m.per = (m.units + sms - 1) / sms;
  const int grid = (m.units + m.per - 1) / m.per;  // no CTA without units
  const int sb = K::stage_bytes(m.ent) + 8;
  m.depth = tile_stages<ROWS, LPR>(m, longest, sms);
  const size_t smem = (size_t)W * m.depth * sb + 4ull * (m.per + 1);
  auto k = k_pcg_tiles<ROWS, LPR, TPBX>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmem);
  if (e != cudaSuccess) return e;
  TileArgs args = a;
  void *p[] = {&args, &m};
  return cudaLaunchCooperativeKernel((const void *)k, dim3(grid), dim3(TPBX), p, smem, s);
}

// A unit costs its lanes' group a gather's latency however short it is, where
// the general form's kernels have many more warps to hide it.  So the tiles
// are for units of kTileMean entries and more on average, which a long row
// among short ones does not make; kTileSlack allows for the launches that the
// general form pays, i.e. shorter units where there are few of them:
// kTileMean * units - entries <= kTileSlack.  Time of an iteration in tiles
// against the general form, us:
//   CSR, 2 lanes   200,000 rows of 3 13.8 / 22.6; 1M of 3 41.2 / 35.2, of 7 42.0
//                  / 46.3; 2.5M of 7 107 / 95, of 9 110 / 110, of 13 116 / 135
//   CSR, 8 lanes   150,000 rows of 25 (one of 200) 29.4 / 33.4, 600,000 95.0 /
//                  65.0; 300,000 of 101 78.3 / 84.6
//   CSR, 32 lanes  150,000 rows of 89 (one of 600) 68.6 / 59.1; 60,000 of 271
//                  47.9 / 53.3, of 601 81.7 / 85.1
//   BSR3, 8        350,000 rows of 3 57.7 / 49.7, of 13 68.8 / 92.5; 150,000 of
//                  7 30.7 / 36.6
//   BSR3, 16       150,000 of 13 (one of 60) 55.1 / 51.4, of 21 59.2 / 62.0;
//                  50,000 of 45 34.8 / 49.0
//   BSR3, 32       60,000 of 21 (one of 150) 42.6 / 41.6, 150,000 93.3 / 65.5;
//                  50,000 of 101 73.6 / 82.6
template <int ROWS, int LPR>
constexpr int kTileMean = ROWS == 3 ? (LPR == 8 ? 10 : LPR == 16 ? 18 : 45) : (LPR == 2 ? 9 : LPR == 8 ? 55 : 200);
template <int ROWS, int LPR>
constexpr double kTileSlack = ROWS == 3 ? (LPR == 8 ? 1.0e6 : LPR == 16 ? 0.7e6 : 0.8e6)
                                        : (LPR == 2 ? 3.5e6 : LPR == 8 ? 5e6 : 6e6);
// CSR with 2 lanes of which only one stage fits (many rows, whose pointers take
// the shared memory, or a long one): 2M rows of 9 (one of 60) 107 / 95, of 13
// 111 / 127; 4M of 13 (one of 30) 240 / 205, of 17 252 / 240; 3.4M of 27 255 / 285.
template <int ROWS, int LPR>
inline int tiles_pay(const TileMat &m, int longest, int64_t entries, int sms) {
  double mean = kTileMean<ROWS, LPR>, slack = kTileSlack<ROWS, LPR>;
  if (ROWS == 1 && LPR == 2 && tile_stages<ROWS, LPR>(m, longest, sms) < 2) {
    mean = 24;
    slack = 25e6;
  }
  return mean * m.units - (double)entries <= slack ? LPR : 0;
}

// lanes per unit (0: the units are too long, too many or too uneven for tiles)
template <int ROWS>
inline int tile_lanes(const TileMat &m, int longest, int64_t entries, int sms) {
  if (sms <= 0) return 0;
  if constexpr (ROWS == 3) {
    if (tiles_fit<3, 8>(m, longest, sms)) return tiles_pay<3, 8>(m, longest, entries, sms);
    if (tiles_fit<3, 16>(m, longest, sms)) return tiles_pay<3, 16>(m, longest, entries, sms);
    if (tiles_fit<3, 32>(m, longest, sms)) return tiles_pay<3, 32>(m, longest, entries, sms);
  } else {
    if (tiles_fit<1, 2>(m, longest, sms)) return tiles_pay<1, 2>(m, longest, entries, sms);
    if (tiles_fit<1, 8>(m, longest, sms)) return tiles_pay<1, 8>(m, longest, entries, sms);
    if (tiles_fit<1, 32>(m, longest, sms)) return tiles_pay<1, 32>(m, longest, entries, sms);
  }
  return 0;
}
template <int ROWS>
inline cudaError_t launch_tiles(const TileArgs &a, const TileMat &m, int longest, int lanes, int sms, cudaStream_t s) {
  if constexpr (ROWS == 3) {
    if (lanes == 8) return launch_tiles_as<3, 8>(a, m, longest, sms, s);
    if (lanes == 16) return launch_tiles_as<3, 16>(a, m, longest, sms, s);
    return launch_tiles_as<3, 32>(a, m, longest, sms, s);
  } else {
    if (lanes == 2) return launch_tiles_as<1, 2>(a, m, longest, sms, s);
    if (lanes == 8) return launch_tiles_as<1, 8>(a, m, longest, sms, s);
    return launch_tiles_as<1, 32>(a, m, longest, sms, s);
  }
}

// ---------------------------------------------------------------------------
// the general form without a handle (sgpu_pcg.cu)
// ---------------------------------------------------------------------------
// Where the device refuses a resident grid: three launches an iteration on
// plain CSR, with the state's scalars and tests.
struct GeneralPcg {
  int n;
  const int *rowptr, *col;
  const double *val, *diag, *f;
  double *x, *r, *h, *d, *p;
  PcgState *st;
  double *partials;   // 2 * blocks
  unsigned *tickets;  // 3, zero
  int blocks;
};
void general_start(const GeneralPcg &a, bool iv, cudaStream_t s);        // r = f - A x0 and the first direction
void general_iterations(const GeneralPcg &a, int count, cudaStream_t s);

}  // namespace sgpu
