// Many independent systems of uneven size: batched Jacobi-PCG over a
// block-diagonal matrix, as one launch of clusters (the default), as one
// persistent launch of CTAs (many small systems, a system too large for a
// cluster's shared memory, or systems coupled by the matrix), or as a graph of
// segmented launches per iteration.
//
// The uneven batch (hundreds of plane-stress plates of different sizes, each
// its own symcomprow::cg_prec in the reference, GEFEL/scr.cpp:1093) is held
// as ONE block-diagonal CSR whose diagonal blocks are the systems; every
// system keeps its own CG scalars, stopping test and (ani, ares).
//
// Work is cut into segments: a segment is a run of at most S consecutive rows
// of one system.  One CTA handles one segment at a time (grid-stride over the
// segment table); its warps cover the rows.  A segment writes one partial sum;
// the last segment of a system to finish (per-system atomic ticket, no
// waiting) adds the system's partials in segment order (deterministic) and
// updates that system's scalars.  Systems that have converged cost one flag
// read per segment from then on.  S and the lanes per CSR row are picked by a
// short autotuning run on the batch itself.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <vector>

#include "sgpu_internal.cuh"
#include "sgpu_persist.cuh"

using namespace sgpu;

namespace sgpu {
int pcg_prepare(sgpu_matrix m, bool mixed);
}

namespace {

constexpr int TPB = 256;

struct SysState {
  double nory, nom, denom, alpha, beta, rr, ares;
  long long ani, it;
  int done, status, ani_set, pad;
};

struct Seg {
  int sys, row0, row1, idx;  // idx: position of the segment within its system
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV]) {
  __shared__ double sh[NV][TPB / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < NV; q++) v[q] = warp_sum(v[q]);
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NV; q++) sh[q][w] = v[q];
  __syncthreads();
  if (w == 0) {
#pragma unroll
    for (int q = 0; q < NV; q++) v[q] = warp_sum(lane < TPB / 32 ? sh[q][lane] : 0.0);
  }
}

// writes the segment's partials; returns true in thread 0 of the CTA that
// completes the system, with the system totals in tot
template <int NV>
__device__ bool seg_reduce(double (&v)[NV], const Seg &sg, const int *__restrict__ sys_seg0,
                           const int *__restrict__ sys_nseg, double *partials, int nseg_total,
                           unsigned *tickets, double (&tot)[NV]) {
  block_sum<NV>(v);
  __shared__ bool last;
  if (threadIdx.x == 0) {
    const int k = sys_seg0[sg.sys] + sg.idx;
#pragma unroll
    for (int q = 0; q < NV; q++) partials[(size_t)q * nseg_total + k] = v[q];
    __threadfence();
    last = (atomicAdd(tickets + sg.sys, 1u) == (unsigned)sys_nseg[sg.sys] - 1u);
  }
  __syncthreads();
  if (!last || threadIdx.x != 0) return false;
  __threadfence();
  const int k0 = sys_seg0[sg.sys], ns = sys_nseg[sg.sys];
#pragma unroll
  for (int q = 0; q < NV; q++) {
    double s = 0.0;
    for (int k = 0; k < ns; k++) s += __ldcg(partials + (size_t)q * nseg_total + k0 + k);
    tot[q] = s;
  }
  tickets[sg.sys] = 0u;
  return true;
}

// rows of a segment, L lanes per row; returns the row's value in sub-lane 0
template <int L>
__device__ __forceinline__ double row_dot(int i, const int *__restrict__ rowptr, const int *__restrict__ col,
                                          const double *__restrict__ val, const double *__restrict__ x, int sub) {
  double s = 0.0;
  const int b = __ldg(rowptr + i), e = __ldg(rowptr + i + 1);
#pragma unroll 4
  for (int k = b + sub; k < e; k += L) s += __ldcs(val + k) * __ldg(x + __ldcs(col + k));
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, L);
  return s;
}

// p = A v on the rows of every live segment; with DOT, d.p per system -> alpha
template <int L, bool DOT>
__global__ void __launch_bounds__(TPB) k_bspmv(int nsegs, const Seg *__restrict__ segs, const int *__restrict__ rowptr,
                                               const int *__restrict__ col, const double *__restrict__ val,
                                               const double *__restrict__ v, double *__restrict__ y, SysState *st,
                                               const int *__restrict__ sys_seg0, const int *__restrict__ sys_nseg,
                                               double *partials, unsigned *tickets, double zero) {
  constexpr int GPW = 32 / L;
  const int lane = threadIdx.x & 31, g = lane / L, sub = lane % L, w = threadIdx.x >> 5;
  __shared__ int skip;
  for (int si = blockIdx.x; si < nsegs; si += gridDim.x) {
    const Seg sg = segs[si];
    if (DOT) {  // one read of the flag for the whole CTA
      if (threadIdx.x == 0) skip = st[sg.sys].done;
      __syncthreads();
      const int sk = skip;
      __syncthreads();
      if (sk) continue;
    }
    double acc = 0.0;
    for (int base = sg.row0 + w * GPW; base < sg.row1; base += (TPB / 32) * GPW) {
      const int i = base + g;
      const int ii = i < sg.row1 ? i : sg.row1 - 1;  // every lane shuffles
      const double s = row_dot<L>(ii, rowptr, col, val, v, sub);
      if (sub == 0 && i < sg.row1) {
        y[i] = s;
        acc += v[i] * s;
      }
    }
    if (DOT) {
      double vv[1] = {acc}, tot[1];
      if (seg_reduce<1>(vv, sg, sys_seg0, sys_nseg, partials, nsegs, tickets, tot)) {
        SysState &s = st[sg.sys];
        s.denom = tot[0];
        if (fabs(tot[0]) < zero) {  // scr.cpp:1146-1151
          s.ani = s.it;
          s.ares = s.nom;
          s.ani_set = 1;
          if (s.status == 0) s.status = SGPU_BREAKDOWN;
          s.done = 1;
        } else {
          s.alpha = s.nom / tot[0];
        }
      }
      __syncthreads();
    }
  }
}

// r = f - p; h = r/diag; d = h; per system f.f, r.h
__global__ void __launch_bounds__(TPB) k_binit(int nsegs, const Seg *__restrict__ segs, const double *__restrict__ f,
                                               const double *__restrict__ p, const double *__restrict__ diag,
                                               double *__restrict__ r, double *__restrict__ h, double *__restrict__ d,
                                               SysState *st, const int *__restrict__ sys_seg0,
                                               const int *__restrict__ sys_nseg, double *partials, unsigned *tickets,
                                               double zero, long long ni) {
  for (int si = blockIdx.x; si < nsegs; si += gridDim.x) {
    const Seg sg = segs[si];
    double v[2] = {0.0, 0.0};
    for (int i = sg.row0 + threadIdx.x; i < sg.row1; i += TPB) {
      const double fi = f[i], ri = fi - p[i], hi = ri / diag[i];
      r[i] = ri;
      h[i] = hi;
      d[i] = hi;
      v[0] += fi * fi;
      v[1] += ri * hi;
    }
    double tot[2];
    if (seg_reduce<2>(v, sg, sys_seg0, sys_nseg, partials, nsegs, tickets, tot)) {
      SysState s = {};
      s.nory = tot[0];
      s.nom = tot[1];
      s.ani = -1;
      if (tot[0] < zero) {  // scr.cpp:1117-1120
        s.status = SGPU_ZERO_RHS;
        s.ares = tot[0];
        s.ani = 0;
        s.ani_set = 1;
      }
      if (ni <= 0) s.done = 1;
      st[sg.sys] = s;
    }
    __syncthreads();
  }
}

// x += alpha d; r -= alpha p; h = r/diag; per system r.r, r.h -> beta, stop
__global__ void __launch_bounds__(TPB) k_bupdate(int nsegs, const Seg *__restrict__ segs, double *__restrict__ x,
                                                 double *__restrict__ r, double *__restrict__ h,
                                                 const double *__restrict__ d, const double *__restrict__ p,
                                                 const double *__restrict__ diag, SysState *st,
                                                 const int *__restrict__ sys_seg0, const int *__restrict__ sys_nseg,
                                                 double *partials, unsigned *tickets, double res, long long ni,
                                                 int *live_count) {
  __shared__ int skip;
  __shared__ double alpha_s;
  for (int si = blockIdx.x; si < nsegs; si += gridDim.x) {
    const Seg sg = segs[si];
    if (threadIdx.x == 0) {
      skip = st[sg.sys].done;
      alpha_s = st[sg.sys].alpha;
    }
    __syncthreads();
    const int sk = skip;
    const double alpha = alpha_s;
    __syncthreads();
    if (sk) continue;
    double v[2] = {0.0, 0.0};
    for (int i = sg.row0 + threadIdx.x; i < sg.row1; i += TPB) {
      x[i] += alpha * d[i];
      const double ri = r[i] - alpha * p[i], hi = ri / diag[i];
      r[i] = ri;
      h[i] = hi;
      v[0] += ri * ri;
      v[1] += ri * hi;
    }
    double tot[2];
    if (seg_reduce<2>(v, sg, sys_seg0, sys_nseg, partials, nsegs, tickets, tot)) {
      SysState &s = st[sg.sys];
      s.rr = tot[0];
      s.beta = tot[1] / s.nom;
      s.nom = tot[1];
      const long long it = s.it;
      s.it = it + 1;
      if (fabs(tot[0] / s.nory) < res) {  // scr.cpp:1188
        s.ani = it;
        s.ares = tot[1] / s.nory;
        s.ani_set = 1;
        s.done = 1;
      } else if (it + 1 >= ni) {
        s.done = 1;
        if (s.status == 0) s.status = SGPU_NOT_CONVERGED;
      }
      if (s.done) atomicSub(live_count, 1);
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(TPB) k_bdir(int nsegs, const Seg *__restrict__ segs, double *__restrict__ d,
                                              const double *__restrict__ h, const SysState *st) {
  for (int si = blockIdx.x; si < nsegs; si += gridDim.x) {
    const Seg sg = segs[si];
    if (st[sg.sys].done) continue;
    const double beta = st[sg.sys].beta;
    for (int i = sg.row0 + threadIdx.x; i < sg.row1; i += TPB) d[i] = beta * d[i] + h[i];
  }
}

// ---------------------------------------------------------------------------
// the persistent form: one CTA per system at a time
//
// The systems are independent, so a CTA can run a whole system's iteration
// alone -- SpMV, the two reductions, the updates -- separated by CTA
// barriers only: no grid-wide step, no launch per iteration, and a converged
// system costs nothing.  CTAs take systems from a queue (largest first, so
// the longest solves start early) through one atomic counter; the kernel
// ends when the queue is empty.  Nothing waits on another CTA.  Each system's
// sums are formed in a fixed order (thread, then warp, then block), so a
// solve is repeatable bit for bit.
// ---------------------------------------------------------------------------
constexpr int PTPB = 512;

__device__ __forceinline__ void cta_sum2(double &a, double &b, double (*sh)[PTPB / 32]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  a = warp_sum(a);
  b = warp_sum(b);
  __syncthreads();
  if (lane == 0) {
    sh[0][w] = a;
    sh[1][w] = b;
  }
  __syncthreads();
  double ta = 0.0, tb = 0.0;
  for (int k = 0; k < PTPB / 32; k++) {  // every thread sums the warp totals in order
    ta += sh[0][k];
    tb += sh[1][k];
  }
  a = ta;
  b = tb;
}

template <int L>
__global__ void __launch_bounds__(PTPB, 2) k_bpersist(int nsys, const int *__restrict__ order,
                                                      const long long *__restrict__ sysptr, int *next,
                                                      const int *__restrict__ rowptr, const int *__restrict__ col,
                                                      const double *__restrict__ val, const double *__restrict__ diag,
                                                      const double *__restrict__ f, double *__restrict__ x,
                                                      double *__restrict__ r, double *__restrict__ h,
                                                      double *__restrict__ d, double *__restrict__ p, SysState *st,
                                                      long long ni, double res, double zero) {
  __shared__ double sh[2][PTPB / 32];
  __shared__ int q_s;
  constexpr int GPW = 32 / L;
  const int lane = threadIdx.x & 31, g = lane / L, sub = lane % L, w = threadIdx.x >> 5;
  for (;;) {
    if (threadIdx.x == 0) q_s = atomicAdd(next, 1);
    __syncthreads();
    const int q = q_s;
    __syncthreads();
    if (q >= nsys) return;
    const int k = order[q];
    const int r0 = (int)sysptr[k], r1 = (int)sysptr[k + 1];
    // start from x = 0: r = f, h = r/diag, d = h; f.f and r.h
    double a = 0.0, b = 0.0;
    for (int i = r0 + threadIdx.x; i < r1; i += PTPB) {
      const double fi = f[i], hi = fi / diag[i];
      x[i] = 0.0;
      r[i] = fi;
      h[i] = hi;
      d[i] = hi;
      a += fi * fi;
      b += fi * hi;
    }
    cta_sum2(a, b, sh);
    SysState s = {};
    s.nory = a;
    s.nom = b;
    s.ani = -1;
    if (a < zero) {  // scr.cpp:1117-1120: reported, the iteration goes on
      s.status = SGPU_ZERO_RHS;
      s.ares = a;
      s.ani = 0;
      s.ani_set = 1;
    }
    if (ni <= 0) s.done = 1;
    while (!s.done) {
      __syncthreads();  // d complete
      // p = A d and d.p
      double dp = 0.0, unused = 0.0;
      for (int base = r0 + w * GPW; base < r1; base += (PTPB / 32) * GPW) {
        const int i = base + g;
        const int ii = i < r1 ? i : r1 - 1;  // every lane shuffles
        const double y = row_dot<L>(ii, rowptr, col, val, d, sub);
        if (sub == 0 && i < r1) {
          p[i] = y;
          dp += d[i] * y;
        }
      }
      cta_sum2(dp, unused, sh);
      s.denom = dp;
      if (fabs(dp) < zero) {  // scr.cpp:1146-1151
        s.ani = s.it;
        s.ares = s.nom;
        s.ani_set = 1;
        if (s.status == 0) s.status = SGPU_BREAKDOWN;
        s.done = 1;
        break;
      }
      const double alpha = s.nom / dp;
      // x += alpha d; r -= alpha p; h = r/diag; r.r and r.h
      double rr = 0.0, rh = 0.0;
      for (int i = r0 + threadIdx.x; i < r1; i += PTPB) {
        x[i] += alpha * d[i];
        const double ri = r[i] - alpha * p[i], hi = ri / diag[i];
        r[i] = ri;
        h[i] = hi;
        rr += ri * ri;
        rh += ri * hi;
      }
      cta_sum2(rr, rh, sh);
      s.alpha = alpha;
      s.rr = rr;
      s.beta = rh / s.nom;
      s.nom = rh;
      const long long it = s.it;
      s.it = it + 1;
      if (fabs(rr / s.nory) < res) {  // scr.cpp:1188
        s.ani = it;
        s.ares = rh / s.nory;
        s.ani_set = 1;
        s.done = 1;
        break;
      }
      if (it + 1 >= ni) {
        s.done = 1;
        if (s.status == 0) s.status = SGPU_NOT_CONVERGED;
        break;
      }
      const double beta = s.beta;
      for (int i = r0 + threadIdx.x; i < r1; i += PTPB) d[i] = beta * d[i] + h[i];
    }
    if (threadIdx.x == 0) st[k] = s;
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// the cluster form: a system's iteration on the eight SMs of a cluster
// ---------------------------------------------------------------------------
// One CTA per system leaves the largest systems to run alone at the end, one
// SM's bandwidth each, and gathers d through L1.  Here a cluster of eight CTAs
// takes a system (small systems: one CTA each, eight to a cluster), largest
// first, as the block scheduler places the clusters.  A CTA owns a contiguous
// range of the rows: r, p and d stay in its shared memory, and a gather reads
// its own d there and a neighbour's through distributed shared memory.  The
// matrix streams through per-warp stages by bulk copies, as in k_pcg_tiles;
// tiles that fit beside the two streaming stages of a warp are copied once
// and stay.  The sums are exchanged through distributed shared memory and the
// hardware's cluster barrier (0.75 us with the CTA's own reduction, against 2.3
// for a barrier of the whole grid).  Every sum is formed in a fixed order, so
// a solve repeats bit for bit.
//
// Measured on B200: 256 plates of 16 to 128 quadrilaterals a side (2.69M
// equations, 393 iterations on average) 465 -> 68 ms; of the largest system's
// iteration (29,440 equations) the product takes about two thirds.  16 warps:
// 24 leave a warp one stage of the largest systems' matrix.
constexpr int kClu = 8;
constexpr int kCluTPB = 512;
constexpr int kCluWarps = kCluTPB / 32;
constexpr int kCluSmem = 222 * 1024;
constexpr int kCluMaxStages = 24;  // of one warp
constexpr int kCluMine = 8;        // rows of a thread
// rows up to which a CTA runs a system alone: an iteration of 2048 plate rows
// costs one SM about 9 us, eight of them 2.3 us each
constexpr int kCluAlone = 2048;

using CluTile = TileKind<1, 2>;

struct CluArgs {
  const int *items;         // system of each CTA (-1: none)
  const long long *sysptr;
  const int *rowptr, *col;  // col: k_local_cols
  const double *val, *diag, *f;
  double *x;
  SysState *st;
  int ent;                  // entries a stage holds
  long long ni;
  double res, zero;
};

struct CluShared {
  double part[2][kCluWarps];
  double slot[2][3][kClu];  // parity, {sum, sum, gave up}, CTA
  unsigned long long full[kCluWarps][kCluMaxStages];
  int bad;
};

__device__ __forceinline__ unsigned clu_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void clu_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned clu_map(const void *p, unsigned rank) {
  unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
// v = the double at a where p is set (volatile: stays between the barriers)
__device__ __forceinline__ void clu_load_if(double &v, unsigned a, bool p) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q ld.shared::cluster.f64 %0, [%1];\n\t}"
               : "+d"(v)
               : "r"(a), "r"((unsigned)p));
}
// a column entry of k_local_cols below 0: the neighbour's d it names
__device__ __forceinline__ unsigned far_address(const double *ds, int at) {
  return clu_map(ds, ((unsigned)at >> 24) & 7u) + ((unsigned)at & 0xffffffu);
}
__device__ __forceinline__ void clu_store(unsigned a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// sums over the group's CTAs, and a barrier of the group; false: a CTA gave up
template <int NV>
__device__ __forceinline__ bool clu_sum(double (&v)[NV], int C, unsigned rank, unsigned &e, CluShared &sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < NV; q++) {
    v[q] = warp_sum(v[q]);
    if (lane == 0) sh.part[q][w] = v[q];
  }
  __syncthreads();
  e ^= 1u;
  if (w == 0) {
#pragma unroll
    for (int q = 0; q < NV; q++) {
      const double t = warp_sum(lane < kCluWarps ? sh.part[q][lane] : 0.0);
      if (C == 1) sh.slot[e][q][0] = t;
      else if (lane < C) clu_store(clu_map(&sh.slot[e][q][rank], lane), t);
    }
    if (C == 1) sh.slot[e][2][0] = sh.bad ? 1.0 : 0.0;
    else if (lane < C) clu_store(clu_map(&sh.slot[e][2][rank], lane), sh.bad ? 1.0 : 0.0);
  }
  if (C > 1) clu_barrier();
  else __syncthreads();
  if (C == 1) {
#pragma unroll
    for (int q = 0; q < NV; q++) v[q] = sh.slot[e][q][0];
    return sh.slot[e][2][0] == 0.0;
  }
  double gave_up = 0.0;
#pragma unroll
  for (int q = 0; q < NV; q++) {
    double t[kClu];
#pragma unroll
    for (int c = 0; c < kClu; c++) t[c] = sh.slot[e][q][c];
    v[q] = ((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7]));
  }
#pragma unroll
  for (int c = 0; c < kClu; c++) gave_up = fmax(gave_up, sh.slot[e][2][c]);
  return gave_up == 0.0;
}

__global__ void __cluster_dims__(kClu, 1, 1) __launch_bounds__(kCluTPB, 1) k_bcluster(const CluArgs a) {
  extern __shared__ __align__(128) unsigned char dyn[];
  __shared__ CluShared sh;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  // a cluster holds one system (its eight entries equal) or up to eight
  const int *it = a.items + (blockIdx.x / kClu) * kClu;
  const unsigned crank = clu_rank();
  const bool whole = it[0] == it[1];
  const int k = it[crank];
  if (k < 0) return;  // only beside systems of one CTA each
  const int C = whole ? kClu : 1;
  const unsigned rank = whole ? crank : 0u;
  const int r0 = (int)a.sysptr[k], n = (int)(a.sysptr[k + 1] - a.sysptr[k]);
  const int per = (n + C - 1) / C;
  const int g0 = r0 + min((int)rank * per, n), nu = min(per, n - min((int)rank * per, n));
  // shared memory: r, p, d of the CTA's rows, their pointers, the stages
  double *rs = reinterpret_cast<double *>(dyn), *ps = rs + per, *ds = ps + per;
  const unsigned char *dsb = reinterpret_cast<const unsigned char *>(ds);
  int *sp = reinterpret_cast<int *>(ds + per);
  const size_t used = ((size_t)28 * per + 4 + 127) & ~(size_t)127;
  const int vb = CluTile::val_bytes(a.ent), sb = CluTile::stage_bytes(a.ent);
  const int D = min((int)((kCluSmem - used) / ((size_t)kCluWarps * sb)), kCluMaxStages);
  unsigned char *stages = dyn + used + (size_t)w * D * sb;
  unsigned long long *full = sh.full[w];
  const int ntiles = (nu + CluTile::kUnits - 1) / CluTile::kUnits;
  const int mine = ntiles > w ? (ntiles - w + kCluWarps - 1) / kCluWarps : 0;
  const int fixed = mine <= D ? mine : max(0, D - 2), S = D - fixed;  // tiles that stay; streaming stages
  for (int q = threadIdx.x; q <= nu; q += kCluTPB) sp[q] = a.rowptr[g0 + q];
  if (lane == 0)
    for (int q = 0; q < D; q++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(ring_u32(full + q)) : "memory");
  if (threadIdx.x == 0) sh.bad = 0;
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  if (C > 1) clu_barrier();  // the neighbours' shared memory is there from here on
  else __syncthreads();
  auto issue = [&](int j, int q) {
    const int t = w + kCluWarps * j;
    const int e0 = sp[t * CluTile::kUnits], e1 = sp[min((t + 1) * CluTile::kUnits, nu)];
    const long long v0 = (long long)e0 & ~1ll, v1 = ((long long)e1 + 1) & ~1ll;
    const int c0 = e0 & ~3, c1 = (e1 + 3) & ~3;
    const unsigned nv = (unsigned)(8 * (v1 - v0)), nc = (unsigned)(4 * (c1 - c0));
    unsigned char *dst = stages + (size_t)q * sb;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(ring_u32(full + q)), "r"(nv + nc)
                 : "memory");
    if (nv)
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       ring_u32(dst)),
                   "l"(a.val + v0), "r"(nv), "r"(ring_u32(full + q))
                   : "memory");
    if (nc)
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       ring_u32(dst + vb)),
                   "l"(a.col + c0), "r"(nc), "r"(ring_u32(full + q))
                   : "memory");
  };
  int next = fixed;  // the next streamed tile to copy
  if (lane == 0) {
    for (int q = 0; q < fixed; q++) issue(q, q);
    if (fixed < mine)
      for (int z = 0; z < S; z++) {
        issue(next, fixed + z);
        if (++next == mine) next = fixed;
      }
  }
  int q = 0;         // streaming stage of the next tile to read
  unsigned ph = 0;   // its phase

  // start from x = 0: r = f, h = r/diag, d = h; f.f and r.h
  double v2[2] = {0.0, 0.0};
  for (int i = threadIdx.x; i < nu; i += kCluTPB) {
    const double fi = a.f[g0 + i], hi = fi / a.diag[g0 + i];
    a.x[g0 + i] = 0.0;
    rs[i] = fi;
    ds[i] = hi;
    v2[0] += fi * fi;
    v2[1] += fi * hi;
  }
  unsigned e = 0;
  SysState s = {};
  bool ok = clu_sum<2>(v2, C, rank, e, sh);
  s.nory = v2[0];
  s.nom = v2[1];
  s.ani = -1;
  if (v2[0] < a.zero) {  // scr.cpp:1117-1120: reported, the iteration goes on
    s.status = SGPU_ZERO_RHS;
    s.ares = v2[0];
    s.ani = 0;
    s.ani_set = 1;
  }
  if (a.ni <= 0) s.done = 1;
  bool first = true;
  while (ok && !s.done) {
    // p = A d over the CTA's rows, d.p
    double v1[1] = {0.0};
    for (int j = 0; j < mine; j++) {
      const int st = j < fixed ? j : fixed + q;
      const bool landed = (j < fixed && !first) || ring_wait(full + st, j < fixed ? 0u : ph);
      const unsigned char *stage = stages + (size_t)st * sb;
      const int t0 = (w + kCluWarps * j) * CluTile::kUnits, e0 = sp[t0];
      const double *vals = reinterpret_cast<const double *>(stage) + (e0 & 1);
      const int *cols = reinterpret_cast<const int *>(stage + vb) + (e0 & 3);
      const int sub = lane & 1, u = t0 + (lane >> 1);
      double y = 0.0, y2 = 0.0;
      if (landed && u < nu) {
        const int b = sp[u] - e0, len = sp[u + 1] - e0 - b;
        // 9 entries of a lane at a time (a plate's row has 18); the CTA's own
        // d first, then -- few rows, at the range's ends -- the neighbours'
        constexpr int U = 9;
        const int *cl = cols + b + sub;
        const double *vl = vals + b + sub;
        int left = (len - sub + 1) >> 1;  // entries of the lane
        for (; left >= U; left -= U, cl += 2 * U, vl += 2 * U) {
          int at[U], far = 0;
          double xx[U];
#pragma unroll
          for (int z = 0; z < U; z++) {
            at[z] = cl[2 * z];
            far |= at[z];
          }
#pragma unroll
          for (int z = 0; z < U; z++) xx[z] = *reinterpret_cast<const double *>(dsb + max(at[z], 0));
          if (far < 0) {
#pragma unroll
            for (int z = 0; z < U; z++) clu_load_if(xx[z], far_address(ds, at[z]), at[z] < 0);
          }
#pragma unroll
          for (int z = 0; z < U; z++) {
            if (z & 1) y2 = fma(vl[2 * z], xx[z], y2);
            else y = fma(vl[2 * z], xx[z], y);
          }
        }
        for (; left > 0; left--, cl += 2, vl += 2) {
          const int at = cl[0];
          double xx = *reinterpret_cast<const double *>(dsb + max(at, 0));
          if (at < 0) clu_load_if(xx, far_address(ds, at), true);
          y = fma(vl[0], xx, y);
        }
        y += y2;
      }
      if (!ring_landed(landed)) {
        sh.bad = 1;
        break;
      }
      y += __shfl_xor_sync(0xffffffffu, y, 1);
      if (sub == 0 && u < nu) {
        ps[u] = y;
        v1[0] += ds[u] * y;
      }
      __syncwarp();  // the stage is read: the warp's next copy may overwrite it
      if (j >= fixed) {
        if (lane == 0) {
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          issue(next, st);
          if (++next == mine) next = fixed;
        }
        if (++q == S) {
          q = 0;
          ph ^= 1;
        }
      }
    }
    first = false;
    // what the update reads from L2, on its way during the sum (a CTA has at
    // most kCluMine rows a thread: cluster_fits)
    double xg[kCluMine], dg[kCluMine];
#pragma unroll
    for (int z = 0; z < kCluMine; z++) {
      const int i = (int)threadIdx.x + z * kCluTPB;
      if (i < nu) {
        xg[z] = a.x[g0 + i];
        dg[z] = __ldg(a.diag + g0 + i);
      }
    }
    ok = clu_sum<1>(v1, C, rank, e, sh);
    if (!ok) break;
    s.denom = v1[0];
    if (fabs(v1[0]) < a.zero) {  // scr.cpp:1146-1151
      s.ani = s.it;
      s.ares = s.nom;
      s.ani_set = 1;
      if (s.status == 0) s.status = SGPU_BREAKDOWN;
      s.done = 1;
      break;
    }
    const double alpha = s.nom / v1[0];
    // x += alpha d; r -= alpha p; h = r/diag (kept where p was); r.r and r.h
    v2[0] = v2[1] = 0.0;
#pragma unroll
    for (int z = 0; z < kCluMine; z++) {
      const int i = (int)threadIdx.x + z * kCluTPB;
      if (i < nu) {
        a.x[g0 + i] = xg[z] + alpha * ds[i];
        const double ri = rs[i] - alpha * ps[i], hi = ri / dg[z];
        rs[i] = ri;
        ps[i] = hi;
        v2[0] += ri * ri;
        v2[1] += ri * hi;
      }
    }
    ok = clu_sum<2>(v2, C, rank, e, sh);
    if (!ok) break;
    s.alpha = alpha;
    s.rr = v2[0];
    s.beta = v2[1] / s.nom;
    s.nom = v2[1];
    const long long n_it = s.it;
    s.it = n_it + 1;
    if (fabs(v2[0] / s.nory) < a.res) {  // scr.cpp:1188
      s.ani = n_it;
      s.ares = v2[1] / s.nory;
      s.ani_set = 1;
      s.done = 1;
      break;
    }
    if (n_it + 1 >= a.ni) {
      s.done = 1;
      if (s.status == 0) s.status = SGPU_NOT_CONVERGED;
      break;
    }
    for (int i = threadIdx.x; i < nu; i += kCluTPB) ds[i] = s.beta * ds[i] + ps[i];
    if (C > 1) clu_barrier();
    else __syncthreads();
  }
  // the copies that nobody reads (and those of a solve without iterations)
  if (lane == 0) {
    for (int z = 0; z < fixed; z++) ring_wait(full + z, 0u);
    if (fixed < mine)
      for (int z = 0; z < S; z++) {
        ring_wait(full + fixed + q, ph);
        if (++q == S) {
          q = 0;
          ph ^= 1;
        }
      }
  }
  if (rank == 0 && threadIdx.x == 0) {
    if (!ok) {
      s.status = SGPU_CUDA_ERROR;
      s.done = 1;
    }
    a.st[k] = s;
  }
  if (C > 1) clu_barrier();  // no CTA leaves while another may read its d
}

// Where a gather finds its d: for an entry of the CTA's own rows the byte
// offset in its shared d, for a neighbour's the sign bit, the neighbour's rank
// (3 bits at 24) and the offset there (at most 32 KB).  The product then needs
// four instructions per entry instead of fifteen (the compares and clamps of
// the column against the CTA's range were what bound it: 1.28e9 row products
// of 18 entries took 77 ms with them).  flag = 1 where a row of a system has a
// column outside the system: then its entry is not used.
__global__ void k_local_cols(int nsys, const long long *__restrict__ sysptr, const int *__restrict__ rowptr,
                             const int *__restrict__ col, int *__restrict__ lcol, int *flag) {
  const int lane = threadIdx.x & 31;
  for (int k = blockIdx.y; k < nsys; k += gridDim.y) {
    const int r0 = (int)sysptr[k], n = (int)(sysptr[k + 1] - r0);
    const int C = n > kCluAlone ? kClu : 1, per = (n + C - 1) / C;
    for (int i = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); i < n; i += (gridDim.x * blockDim.x) >> 5) {
      const int own = i / per;
      for (int q = rowptr[r0 + i] + lane; q < rowptr[r0 + i + 1]; q += 32) {
        const int rel = col[q] - r0;
        int v = 0;
        if (rel < 0 || rel >= n) {
          *flag = 1;
        } else {
          const int o = rel / per, off = 8 * (rel - o * per);
          v = o == own ? off : (int)(0x80000000u | ((unsigned)o << 24) | (unsigned)off);
        }
        lcol[q] = v;
      }
    }
  }
}

// Whether the cluster form takes the batch: the longest row's stage and the
// largest system's vectors fit a CTA's shared memory with two stages a warp,
// for rows of 18 entries up to 32,768 rows a system, of 27 up to 17,040.  One
// larger system sends the whole batch to CTAs: 256 plates of 16 to 128
// quadrilaterals a side take 71 ms, with one of 128 by 128 among them (33,024
// rows) 471.
bool cluster_fits(int longest, int64_t most_rows) {
  if (longest <= 0 || longest > 2048) return false;
  const int64_t ent = ((int64_t)longest * CluTile::kUnits + 3) & ~3ll;
  const int64_t per = std::max<int64_t>((most_rows + kClu - 1) / kClu, std::min<int64_t>(most_rows, kCluAlone));
  return per <= kCluMine * kCluTPB &&
         28 * per + 256 + 2 * kCluWarps * (int64_t)CluTile::stage_bytes((int)ent) <= kCluSmem;
}

// Whether clusters finish the batch earlier than CTAs with a system each, two
// to an SM: the times of an iteration are summed over the waves of either form
// as if all systems took as many iterations.  A CTA of a cluster has an SM of
// its own, which small systems do not fill.  Measured for 100 iterations (ms,
// clusters / CTAs): 5000 systems of 60 rows of 9 entries 8.09 / 3.54, 2000 of
// 200 4.22 / 2.42, 500 of 1000 2.30 / 1.82; 256 of 2048 rows of 17 3.58 / 4.21,
// 148 of 2000 2.37 / 3.33, 64 of 8000 4.27 / 15.5, 10 of 30,000 2.34 / 57.7.
// mean: entries of a row.
bool cluster_pays(const std::vector<int64_t> &rows, double mean, int sms) {
  // us of an iteration by these measurements
  auto on_cta = [&](int64_t r) { return 2.0 + 1.1e-3 * mean * (double)r; };
  auto on_cluster = [&](int64_t r) {
    return r <= kCluAlone ? 2.7 + 4.5e-4 * mean * (double)r : 3.0 + 5.6e-5 * mean * (double)r;
  };
  std::vector<int64_t> sorted(rows);
  std::sort(sorted.begin(), sorted.end(), std::greater<int64_t>());
  double ctas = 0.0;
  for (int64_t r : sorted) ctas += on_cta(r);
  ctas = std::max(ctas / (2.0 * sms), on_cta(sorted[0]));
  // clusters in launch order, each to the slot that is free first
  std::vector<double> slot((size_t)std::max(1, sms / kClu), 0.0);
  for (size_t k = 0; k < sorted.size(); k += sorted[k] > kCluAlone ? 1 : kClu)
    *std::min_element(slot.begin(), slot.end()) += on_cluster(sorted[k]);
  return *std::max_element(slot.begin(), slot.end()) <= ctas;
}

constexpr int kOther = 1000;  // run_cluster: not for this batch or device

// Whether the device schedules a cluster with a CTA's shared memory each.
bool cluster_runs(int sms) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kClu);
  cfg.blockDim = dim3(kCluTPB);
  cfg.dynamicSmemBytes = kCluSmem;
  int most = 0;
  if (sms >= kClu &&
      cudaFuncSetAttribute(k_bcluster, cudaFuncAttributeMaxDynamicSharedMemorySize, kCluSmem) == cudaSuccess &&
      cudaOccupancyMaxActiveClusters(&most, k_bcluster, &cfg) == cudaSuccess)
    return most > 0;
  cudaGetLastError();
  return false;
}

int run_cluster(sgpu_matrix m, const std::vector<int64_t> &rows, int longest, double *x, const double *f, int64_t ni,
                double res, double zero, std::vector<SysState> &hs, int64_t *iters, float *ms) {
  cudaStream_t s = m->stream;
  const Csr &c = m->csr;
  const int nsys = (int)rows.size();
  std::vector<long long> ptr(nsys + 1, 0);
  for (int k = 0; k < nsys; k++) ptr[k + 1] = ptr[k] + rows[k];
  std::vector<int> order(nsys), items;
  for (int k = 0; k < nsys; k++) order[k] = k;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return rows[a] > rows[b]; });
  int at = 0;
  for (; at < nsys && rows[order[at]] > kCluAlone; at++) items.insert(items.end(), kClu, order[at]);
  for (; at < nsys; at += kClu)
    for (int z = 0; z < kClu; z++) items.push_back(at + z < nsys ? order[at + z] : -1);
  DevBuf<long long> ptr_d;
  DevBuf<int> items_d;
  DevBuf<SysState> st;
  SGPU_TRY(ptr_d.alloc(nsys + 1));
  SGPU_TRY(items_d.alloc(items.size()));
  SGPU_TRY(st.alloc(nsys));
  SGPU_CUDA(cudaMemcpyAsync(ptr_d.p, ptr.data(), (nsys + 1) * sizeof(long long), cudaMemcpyHostToDevice, s));
  SGPU_CUDA(cudaMemcpyAsync(items_d.p, items.data(), items.size() * sizeof(int), cudaMemcpyHostToDevice, s));
  // the neighbours whose d a gather may read are the system's own: where the
  // matrix couples systems, the caller's other form runs
  DevBuf<int> lcol;
  SGPU_TRY(lcol.alloc((size_t)c.nnz + 4));
  int *flag_d = reinterpret_cast<int *>(m->w.counters.p + 8), coupled = 0;
  SGPU_CUDA(cudaMemsetAsync(flag_d, 0, sizeof(int), s));
  const dim3 lg((unsigned)std::max<int64_t>(1, std::min<int64_t>((rows[order[0]] + 63) / 64, 16)),
                (unsigned)std::min(nsys, 2048));
  k_local_cols<<<lg, TPB, 0, s>>>(nsys, ptr_d.p, c.rowptr.p, c.col.p, lcol.p, flag_d);
  count_launches(1);
  SGPU_CUDA(cudaMemcpyAsync(&coupled, flag_d, sizeof(int), cudaMemcpyDeviceToHost, s));
  SGPU_CUDA(cudaStreamSynchronize(s));
  if (coupled) return kOther;
  const int ent = (longest * CluTile::kUnits + 3) & ~3;
  const CluArgs a = {items_d.p, ptr_d.p, c.rowptr.p, lcol.p, c.val.p, c.diag.p, f, x, st.p, ent, (long long)ni, res,
                     zero};
  SGPU_CUDA(cudaEventRecord(m->ev0, s));
  k_bcluster<<<(unsigned)items.size(), kCluTPB, kCluSmem, s>>>(a);
  count_launches(1);
  SGPU_CUDA(cudaGetLastError());
  SGPU_CUDA(cudaEventRecord(m->ev1, s));
  hs.resize(nsys);
  SGPU_CUDA(cudaMemcpyAsync(hs.data(), st.p, nsys * sizeof(SysState), cudaMemcpyDeviceToHost, s));
  SGPU_CUDA(cudaStreamSynchronize(s));
  if (ms) SGPU_CUDA(cudaEventElapsedTime(ms, m->ev0, m->ev1));
  int64_t mx = 0;
  for (const SysState &q : hs) {
    if (q.status == SGPU_CUDA_ERROR) return fail(SGPU_CUDA_ERROR, "batched PCG: a wait inside a cluster ran out");
    mx = std::max<int64_t>(mx, q.it);
  }
  if (iters) *iters = mx;
  return SGPU_OK;
}

// the persistent solve of every system; hs gets the per-system results
int run_persistent(sgpu_matrix m, const std::vector<int64_t> &rows, int L, double *x, const double *f, double *r,
                   double *h, double *d, double *p, int64_t ni, double res, double zero, std::vector<SysState> &hs,
                   int64_t *iters, float *ms) {
  cudaStream_t s = m->stream;
  const Csr &c = m->csr;
  const int nsys = (int)rows.size();
  std::vector<long long> ptr(nsys + 1, 0);
  for (int k = 0; k < nsys; k++) ptr[k + 1] = ptr[k] + rows[k];
  std::vector<int> order(nsys);
  for (int k = 0; k < nsys; k++) order[k] = k;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return rows[a] > rows[b]; });
  DevBuf<long long> ptr_d;
  DevBuf<int> order_d, next_d;
  DevBuf<SysState> st;
  SGPU_TRY(ptr_d.alloc(nsys + 1));
  SGPU_TRY(order_d.alloc(nsys));
  SGPU_TRY(next_d.alloc(1));
  SGPU_TRY(st.alloc(nsys));
  SGPU_CUDA(cudaMemcpyAsync(ptr_d.p, ptr.data(), (nsys + 1) * sizeof(long long), cudaMemcpyHostToDevice, s));
  SGPU_CUDA(cudaMemcpyAsync(order_d.p, order.data(), nsys * sizeof(int), cudaMemcpyHostToDevice, s));
  SGPU_CUDA(cudaMemsetAsync(next_d.p, 0, sizeof(int), s));
  const int grid = std::min(nsys, kNumSMs * 2);
  SGPU_CUDA(cudaEventRecord(m->ev0, s));
  switch (L) {
    case 4:
      k_bpersist<4><<<grid, PTPB, 0, s>>>(nsys, order_d.p, ptr_d.p, next_d.p, c.rowptr.p, c.col.p, c.val.p, c.diag.p,
                                          f, x, r, h, d, p, st.p, (long long)ni, res, zero);
      break;
    case 16:
      k_bpersist<16><<<grid, PTPB, 0, s>>>(nsys, order_d.p, ptr_d.p, next_d.p, c.rowptr.p, c.col.p, c.val.p,
                                           c.diag.p, f, x, r, h, d, p, st.p, (long long)ni, res, zero);
      break;
    default:
      k_bpersist<8><<<grid, PTPB, 0, s>>>(nsys, order_d.p, ptr_d.p, next_d.p, c.rowptr.p, c.col.p, c.val.p, c.diag.p,
                                          f, x, r, h, d, p, st.p, (long long)ni, res, zero);
      break;
  }
  count_launches(1);
  SGPU_CUDA(cudaGetLastError());
  SGPU_CUDA(cudaEventRecord(m->ev1, s));
  hs.resize(nsys);
  SGPU_CUDA(cudaMemcpyAsync(hs.data(), st.p, nsys * sizeof(SysState), cudaMemcpyDeviceToHost, s));
  SGPU_CUDA(cudaStreamSynchronize(s));
  if (ms) SGPU_CUDA(cudaEventElapsedTime(ms, m->ev0, m->ev1));
  int64_t mx = 0;
  for (const SysState &q : hs) mx = std::max<int64_t>(mx, q.it);
  if (iters) *iters = mx;
  return SGPU_OK;
}

struct Plan {
  int S = 1024, L = 8;
};

struct Batch {
  int nsys = 0, nsegs = 0;
  DevBuf<Seg> segs;
  DevBuf<int> seg0, nseg;
  DevBuf<SysState> st;
  DevBuf<unsigned> tickets;
  DevBuf<double> partials;
  DevBuf<int> live;
};

int build_segments(const std::vector<int64_t> &sys_rows, int S, Batch &b, cudaStream_t s) {
  std::vector<Seg> segs;
  std::vector<int> seg0, nseg;
  int64_t row = 0;
  for (size_t k = 0; k < sys_rows.size(); k++) {
    const int64_t r0 = row, r1 = row + sys_rows[k];
    seg0.push_back((int)segs.size());
    int idx = 0;
    for (int64_t a = r0; a < r1; a += S) segs.push_back(Seg{(int)k, (int)a, (int)std::min<int64_t>(a + S, r1), idx++});
    nseg.push_back(idx);
    row = r1;
  }
  b.nsys = (int)sys_rows.size();
  b.nsegs = (int)segs.size();
  SGPU_TRY(b.segs.alloc(segs.size()));
  SGPU_TRY(b.seg0.alloc(seg0.size()));
  SGPU_TRY(b.nseg.alloc(nseg.size()));
  SGPU_TRY(b.st.alloc(b.nsys));
  SGPU_TRY(b.tickets.alloc(b.nsys));
  SGPU_TRY(b.partials.alloc((size_t)2 * b.nsegs));
  SGPU_TRY(b.live.alloc(1));
  SGPU_CUDA(cudaMemcpyAsync(b.segs.p, segs.data(), segs.size() * sizeof(Seg), cudaMemcpyHostToDevice, s));
  SGPU_CUDA(cudaMemcpyAsync(b.seg0.p, seg0.data(), seg0.size() * sizeof(int), cudaMemcpyHostToDevice, s));
  SGPU_CUDA(cudaMemcpyAsync(b.nseg.p, nseg.data(), nseg.size() * sizeof(int), cudaMemcpyHostToDevice, s));
  SGPU_CUDA(cudaMemsetAsync(b.tickets.p, 0, b.nsys * sizeof(unsigned), s));
  SGPU_CUDA(cudaStreamSynchronize(s));
  return SGPU_OK;
}

template <bool DOT>
int launch_bspmv(int L, int grid, Batch &b, const Csr &c, const double *v, double *y, cudaStream_t s, double zero) {
  switch (L) {
    case 4: k_bspmv<4, DOT><<<grid, TPB, 0, s>>>(b.nsegs, b.segs.p, c.rowptr.p, c.col.p, c.val.p, v, y, b.st.p, b.seg0.p,
                                                 b.nseg.p, b.partials.p, b.tickets.p, zero); break;
    case 16: k_bspmv<16, DOT><<<grid, TPB, 0, s>>>(b.nsegs, b.segs.p, c.rowptr.p, c.col.p, c.val.p, v, y, b.st.p,
                                                   b.seg0.p, b.nseg.p, b.partials.p, b.tickets.p, zero); break;
    default: k_bspmv<8, DOT><<<grid, TPB, 0, s>>>(b.nsegs, b.segs.p, c.rowptr.p, c.col.p, c.val.p, v, y, b.st.p, b.seg0.p,
                                                  b.nseg.p, b.partials.p, b.tickets.p, zero); break;
  }
  count_launches(1);
  SGPU_CUDA(cudaGetLastError());
  return SGPU_OK;
}

// one batched solve; x, f device vectors (n); returns per-system results in hs
int run_batch(sgpu_matrix m, Batch &b, const Plan &pl, double *x, const double *f, double *r, double *h, double *d,
              double *p, int64_t ni, double res, double zero, std::vector<SysState> &hs, int64_t *iters,
              float *ms) {
  cudaStream_t s = m->stream;
  const Csr &c = m->csr;
  const int grid = std::min(b.nsegs, kNumSMs * 8);
  SGPU_CUDA(cudaMemsetAsync(b.tickets.p, 0, b.nsys * sizeof(unsigned), s));
  SGPU_CUDA(cudaEventRecord(m->ev0, s));
  SGPU_TRY(launch_bspmv<false>(pl.L, grid, b, c, x, p, s, zero));
  k_binit<<<grid, TPB, 0, s>>>(b.nsegs, b.segs.p, f, p, c.diag.p, r, h, d, b.st.p, b.seg0.p, b.nseg.p, b.partials.p,
                               b.tickets.p, zero, (long long)ni);
  count_launches(1);
  const int nsys = b.nsys;
  SGPU_CUDA(cudaMemcpyAsync(b.live.p, &nsys, sizeof(int), cudaMemcpyHostToDevice, s));
  // a graph of G iterations, relaunched until every system has stopped
  constexpr int G = 16;
  cudaGraph_t gph;
  cudaGraphExec_t exec;
  SGPU_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeRelaxed));
  for (int k = 0; k < G; k++) {
    launch_bspmv<true>(pl.L, grid, b, c, d, p, s, zero);
    k_bupdate<<<grid, TPB, 0, s>>>(b.nsegs, b.segs.p, x, r, h, d, p, c.diag.p, b.st.p, b.seg0.p, b.nseg.p,
                                   b.partials.p, b.tickets.p, res, (long long)ni, b.live.p);
    k_bdir<<<grid, TPB, 0, s>>>(b.nsegs, b.segs.p, d, h, b.st.p);
  }
  SGPU_CUDA(cudaStreamEndCapture(s, &gph));
  cudaError_t e = cudaGraphInstantiate(&exec, gph, 0);
  cudaGraphDestroy(gph);
  if (e != cudaSuccess) return fail(SGPU_CUDA_ERROR, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e));
  int64_t it = 0;
  int live = nsys;
  int rc = SGPU_OK;
  while (live > 0 && it < ni) {
    e = cudaGraphLaunch(exec, s);
    if (e != cudaSuccess) { rc = fail(SGPU_CUDA_ERROR, std::string("cudaGraphLaunch: ") + cudaGetErrorString(e)); break; }
    count_launches(3 * G);
    it += G;
    e = cudaMemcpyAsync(&live, b.live.p, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) { rc = fail(SGPU_CUDA_ERROR, std::string("batch loop: ") + cudaGetErrorString(e)); break; }
  }
  cudaGraphExecDestroy(exec);
  if (rc != SGPU_OK) return rc;
  SGPU_CUDA(cudaEventRecord(m->ev1, s));
  hs.resize(nsys);
  SGPU_CUDA(cudaMemcpyAsync(hs.data(), b.st.p, nsys * sizeof(SysState), cudaMemcpyDeviceToHost, s));
  SGPU_CUDA(cudaStreamSynchronize(s));
  if (ms) SGPU_CUDA(cudaEventElapsedTime(ms, m->ev0, m->ev1));
  if (iters) *iters = it;
  return SGPU_OK;
}

}  // namespace

extern "C" SGPU_API int sgpu_matrix_pcg_batch(sgpu_matrix m, int32_t nsys, const int64_t *sys_rows, double *x,
                                              const double *f, int64_t ni, double res, double zero, int32_t tune,
                                              int64_t *ani, double *ares, int32_t *status, int64_t *iterations,
                                              sgpu_solve_info *info) {
  if (!m || !sys_rows || !x || !f) return fail(SGPU_BAD_INPUT, "null argument");
  if (nsys <= 0) return fail(SGPU_BAD_INPUT, "no systems");
  if (!m->csr.diag_positive) return fail(SGPU_BAD_INPUT, "Jacobi preconditioner needs a positive diagonal");
  std::vector<int64_t> rows(sys_rows, sys_rows + nsys);
  int64_t total = 0;
  for (int64_t v : rows) {
    if (v <= 0) return fail(SGPU_BAD_INPUT, "every system needs at least one equation");
    total += v;
  }
  if (total != m->n) return fail(SGPU_BAD_INPUT, "system sizes do not add up to the matrix size");
  if (info) memset(info, 0, sizeof(*info));
  SGPU_TRY(pcg_prepare(m, false));
  cudaStream_t s = m->stream;
  const size_t n = (size_t)m->n;
  Work &w = m->w;
  SGPU_CUDA(copy_in(w.f.p, f, n * sizeof(double), s));
  // the plan: segment rows S and lanes per row L; tuned on ~32 iterations of
  // this batch when asked (the iterate is reset for the real solve)
  // SGPU_BATCH_FORM=graph: the segmented graph-of-launches form below;
  // otherwise the persistent form (one CTA per system at a time)
  const char *form = getenv("SGPU_BATCH_FORM");
  const bool persistent = !(form && !strcmp(form, "graph"));
  Plan best;
  if (tune && !persistent) {
    float best_ms = 1e30f;
    for (int S : {512, 1024, 2048, 4096})
      for (int L : {4, 8, 16}) {
        Batch b;
        SGPU_TRY(build_segments(rows, S, b, s));
        std::vector<SysState> hs;
        float ms = 0.f;
        int64_t its = 0;
        SGPU_CUDA(cudaMemsetAsync(w.x.p, 0, n * sizeof(double), s));
        SGPU_TRY(run_batch(m, b, Plan{S, L}, w.x.p, w.f.p, w.r.p, w.h.p, w.d.p, w.p.p, 32, res, zero, hs, &its, &ms));
        if (ms < best_ms) { best_ms = ms; best = Plan{S, L}; }
      }
  }
  std::vector<SysState> hs;
  float ms = 0.f;
  int64_t its = 0;
  if (persistent) {
    // lanes per row from the rows' mean length
    const double mean = (double)m->csr.nnz / (double)m->n;
    best.L = mean > 40 ? 16 : (mean > 12 ? 8 : 4);
    best.S = 0;
    const int longest = m->csr.longest;
    const int64_t most = *std::max_element(rows.begin(), rows.end());
    int rc = kOther;
    if (cluster_fits(longest, most) && cluster_pays(rows, mean, kNumSMs) && cluster_runs(resident_grid()))
      rc = run_cluster(m, rows, longest, w.x.p, w.f.p, ni, res, zero, hs, &its, &ms);
    if (rc == SGPU_OK) best.L = CluTile::kLpr;
    if (rc == kOther)
      rc = run_persistent(m, rows, best.L, w.x.p, w.f.p, w.r.p, w.h.p, w.d.p, w.p.p, ni, res, zero, hs, &its, &ms);
    if (rc != SGPU_OK) return rc;
  } else {
    Batch b;
    SGPU_TRY(build_segments(rows, best.S, b, s));
    SGPU_CUDA(cudaMemsetAsync(w.x.p, 0, n * sizeof(double), s));
    SGPU_TRY(run_batch(m, b, best, w.x.p, w.f.p, w.r.p, w.h.p, w.d.p, w.p.p, ni, res, zero, hs, &its, &ms));
  }
  SGPU_CUDA(copy_out(x, w.x.p, n * sizeof(double), s));
  SGPU_CUDA(cudaStreamSynchronize(s));
  int worst = SGPU_OK;
  for (int k = 0; k < nsys; k++) {
    int st = hs[k].status;
    if (!hs[k].done && st == SGPU_OK) st = SGPU_NOT_CONVERGED;
    if (status) status[k] = st;
    if (iterations) iterations[k] = hs[k].it;
    if (hs[k].ani_set) {
      if (ani) ani[k] = hs[k].ani;
      if (ares) ares[k] = hs[k].ares;
    }
    if (st != SGPU_OK && worst == SGPU_OK) worst = st;
  }
  if (info) {
    info->iterations = its;
    info->solve_ms = ms;
    info->spmv_format = 0;
    info->spmv_variant = best.L;
    info->spmv_bytes = (double)m->csr.nnz * 12.0 + (m->n + 1) * 4.0 + 2.0 * m->n * 8.0;
    info->tile_rows = best.S;
  }
  return worst;
}
