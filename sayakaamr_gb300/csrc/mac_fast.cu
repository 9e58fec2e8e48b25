// Device-resident MG-preconditioned BiCGSTAB (the iteration of
// src/SayakaMacSolver.cpp:683-920) for production solves:
//  * scalars (rho, alpha, omega, norms, flags) stay in device memory; the last
//    CTA of every reduction runs the reference's scalar logic (breakdown and
//    convergence tests) in its epilogue, so a solve needs no host round trip;
//  * vector updates are fused with the reductions that follow them;
//  * one iteration is captured in a CUDA graph under a conditional WHILE node
//    that a kernel re-arms until the convergence flag is set;
//  * the V-cycle runs in FP64 or FP32 (residual, transfers, smoother), the
//    bottom level is solved directly with a dense FP64 inverse of the
//    level-1 operator built on the GPU at setup (singular Neumann components
//    are pinned at one cell).
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include <cuda_fp16.h>

#include "dev_alloc.h"
#include "mac_solver.h"
#include "cuda_check.h"
#include "mac_stencil.cuh"
#include "mac_df.cuh"
#include "mac_flow.h"
#include "launch.cuh"
#include "mac_fp.cuh"
#include "tree.h"

namespace sayaka_gb300 {

namespace {

constexpr int kTPB = 256;
constexpr int kMaxRedBlocks = 152 * 4;

// grid of the kernels that end in a grid reduction: every CTA adds one
// same-address atomic to the reduction's tail, so latency-bound sizes (under
// 2M cells) take half the CTAs
inline int red_grid(long work) {
  long g = (work + kTPB - 1) / kTPB;
  const long cap = work < (1l << 21) ? kMaxRedBlocks / 2 : kMaxRedBlocks;
  return (int)std::max<long>(1, std::min<long>(g, cap));
}
inline int ew_grid(long work) {
  long g = (work + kTPB - 1) / kTPB;
  return (int)std::max<long>(1, std::min<long>(g, 152 * 32));
}

__device__ __forceinline__ double wsum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Reduction of NV values (bit i of maxmask: max, else sum) over the `count`
// CTAs whose partial slots are first .. first+count-1 (this CTA's is `slot`):
// each CTA writes its partials; the last of them to arrive combines them in
// slot order (deterministic for a fixed grid) and runs `epi` on thread 0.
// Max values are non-negative (norms): they combine as their bit patterns
// read as unsigned integers, on the integer pipe.  A NaN (all-ones exponent,
// non-zero mantissa) orders above +inf, so a NaN anywhere in a vector reaches
// the convergence test and ends the solve as a breakdown, not as convergence.
__device__ __forceinline__ double bmax(double a, double b) {
  const unsigned long long x = (unsigned long long)__double_as_longlong(a);
  const unsigned long long y = (unsigned long long)__double_as_longlong(b);
  return __longlong_as_double((long long)(x > y ? x : y));
}
__device__ __forceinline__ double wbmax(double v) {
  for (int o = 16; o > 0; o >>= 1) v = bmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

template <int NV, class Epi>
__device__ __forceinline__ void seg_reduce(double (&v)[NV], unsigned maxmask, double *partials, unsigned *counter,
                                           int first, int count, int slot, Epi epi) {
  __shared__ double sh[NV][kTPB / 32];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  // the kTPB / 32 warp results of sh combined by warp 0 (same tree order
  // for every CTA and every launch)
  auto warp0 = [&](double (&r)[NV]) {
#pragma unroll
    for (int i = 0; i < NV; i++) {
      double x = lane < kTPB / 32 ? sh[i][lane] : 0.0;
      for (int o = (kTPB / 64); o > 0; o >>= 1) {
        const double y = __shfl_xor_sync(0xffffffffu, x, o);
        x = ((maxmask >> i) & 1) ? bmax(x, y) : x + y;
      }
      r[i] = x;
    }
  };
#pragma unroll
  for (int i = 0; i < NV; i++) {
    const double r = ((maxmask >> i) & 1) ? wbmax(v[i]) : wsum(v[i]);
    if (lane == 0) sh[i][w] = r;
  }
  __syncthreads();
  if (w == 0) {
    double r[NV];
    warp0(r);
    if (lane == 0) {
#pragma unroll
      for (int i = 0; i < NV; i++) partials[slot * NV + i] = r[i];
      // release the partials, acquire everyone else's if this CTA is last
      unsigned old;
      asm volatile("atom.add.acq_rel.gpu.u32 %0, [%1], 1;" : "=r"(old) : "l"(counter) : "memory");
      last = old == (unsigned)count - 1;
    }
  }
  __syncthreads();
  if (!last) return;
  double acc[NV];
#pragma unroll
  for (int i = 0; i < NV; i++) acc[i] = 0.0;
  for (int b = first + threadIdx.x; b < first + count; b += blockDim.x) {
#pragma unroll
    for (int i = 0; i < NV; i++) {
      const double pv = ((volatile double *)partials)[b * NV + i];
      acc[i] = ((maxmask >> i) & 1) ? bmax(acc[i], pv) : acc[i] + pv;
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < NV; i++) {
    const double r = ((maxmask >> i) & 1) ? wbmax(acc[i]) : wsum(acc[i]);
    if (lane == 0) sh[i][w] = r;
  }
  __syncthreads();
  if (w == 0) {
    double fin[NV];
    warp0(fin);
    if (lane == 0) {
      epi(fin);
      *counter = 0;
    }
  }
}

// the whole grid as one segment
template <int NV, class Epi>
__device__ __forceinline__ void grid_reduce(double (&v)[NV], unsigned maxmask, double *partials, unsigned *counter,
                                            Epi epi) {
  seg_reduce<NV>(v, maxmask, partials, counter, 0, (int)gridDim.x, (int)blockIdx.x, epi);
}

// A forest of independent problems (the connected components of the tree)
// solved with one BiCGSTAB state per problem: the finest tower's blocks are
// listed problem by problem, and the BiCGSTAB kernels run one CTA per chunk
// of at most chunk_cells() consecutive cells of one problem, so that every
// reduction is a segment of whole CTAs (seg_reduce) and every CTA reads one
// state.
// the cells a CTA walks, the state it reads and its reduction segment
struct Work {
  int it0, it1, step;
  FState *st;
  int first, count, slot;
  unsigned *counter;
};
template <bool MULTI>
__device__ __forceinline__ Work work_of(const Chunks &ch, FState *st, int total, unsigned *counters) {
  Work w;
  if constexpr (MULTI) {
    const int k = blockIdx.x, c = ch.comp[k];
    w.it0 = ch.beg[k] + threadIdx.x;
    w.it1 = ch.end[k];
    w.step = blockDim.x;
    w.st = st + c;
    w.first = ch.c0[c];
    w.count = ch.cn[c];
    w.slot = k;
    w.counter = counters ? counters + c : nullptr;
  } else {
    w.it0 = blockIdx.x * blockDim.x + threadIdx.x;
    w.it1 = total;
    w.step = gridDim.x * blockDim.x;
    w.st = st;
    w.first = 0;
    w.count = gridDim.x;
    w.slot = blockIdx.x;
    w.counter = counters;
  }
  return w;
}

// precision conversions of the vector kernels, exact or correctly rounded
// on the integer pipe (mac_fp.cuh)
template <typename T>
__device__ __forceinline__ T narrow_to(double v) {
  if constexpr (sizeof(T) == 4)
    return fpint::narrow(v);
  else
    return v;
}
template <typename T>
__device__ __forceinline__ double widen_from(T v) {
  if constexpr (sizeof(T) == 4)
    return fpint::widen(v);
  else
    return v;
}

__device__ __forceinline__ long cell_of(const BlockList &L, int ncell, int it) {
  const int p = it / ncell;
  return (long)L.blocks[p] * ncell + (it - p * ncell);
}

// ---- epilogues: the reference's scalar logic (src/SayakaMacSolver.cpp:766-904)
struct EpiInit {  // after r0 = b - A x0: |r0|, rho = r0.r0
  FState *st;
  __device__ void operator()(const double *v) const {
    st->rnorm0 = v[0];
    st->rnorm = v[0];
    st->iter = 1;
    if (v[0] == 0) {  // initial convergence: solution untouched
      st->done = 1;
      st->conv = 0;
      st->stat = 0;
      st->trivial = 1;
      return;
    }
    st->rho = v[1];
    if (v[1] == 0) {
      st->stat = 1;
      st->done = 1;
    }
  }
};
struct EpiAlpha {  // rhat.v
  FState *st;
  __device__ void operator()(const double *v) const {
    st->restart = 0;  // the p-update of this iteration has read it
    if (v[0] == 0) {
      st->stat = 1;
      st->done = 1;
      return;
    }
    st->alpha = st->rho / v[0];
  }
};
struct EpiHalf {  // |s|
  FState *st;
  __device__ void operator()(const double *v) const {
    st->rnorm = v[0];
    if (v[0] != v[0]) {  // NaN: breakdown
      st->stat = 1;
      st->done = 1;
      return;
    }
    if (v[0] < st->rnorm0 * st->tol_rel || v[0] < st->tol_abs) {
      st->verify = 1;  // x is final for this pass: check its true residual
      st->done = 1;
    }
  }
};
struct EpiOmega {  // t.s, t.t
  FState *st;
  __device__ void operator()(const double *v) const {
    if (v[1] == 0) {
      st->stat = 1;
      st->done = 1;
      return;
    }
    st->omega = v[0] / v[1];
  }
};
// The recursively updated residual of BiCGSTAB drifts from b - A x by about
// eps |A| |x| per iteration; with small volume fractions (large 1/(dv vf))
// the gap reaches the tolerance.  A converged pass is therefore verified with
// the true residual r = b - A x0 (x folded into x0); if that misses the
// tolerance the solve restarts from x0 with r^ = p = r (at most kMaxRestarts
// times, then it ends as not converged).
constexpr int kMaxRestarts = 5;
struct EpiVerify {  // |b - A x0|, r.r
  FState *st;
  __device__ void operator()(const double *v) const {
    st->verify = 0;
    st->rnorm = v[0];
    if (v[0] != v[0]) {
      st->stat = 1;
      return;
    }
    if (v[0] < st->rnorm0 * st->tol_rel + st->tol_abs) {
      st->conv = 1;
      return;
    }
    if (st->restarts >= kMaxRestarts) return;  // done, not converged
    st->restarts += 1;
    st->rho = v[1];
    if (v[1] == 0) {
      st->stat = 1;
      return;
    }
    st->restart = 1;
    st->done = 0;
  }
};

struct EpiEnd {  // |r|, rhat.r of the next iteration
  FState *st;
  __device__ void operator()(const double *v) const {
    st->rnorm = v[0];
    if (v[0] != v[0]) {  // NaN: breakdown
      st->stat = 1;
      st->done = 1;
      return;
    }
    if (v[0] < st->rnorm0 * st->tol_rel + st->tol_abs) {
      st->verify = 1;  // check the true residual before accepting
      st->done = 1;
      return;
    }
    // learned correction: unless the best residual halves within 2
    // iterations it is switched off and the solve goes on with the plain MG
    // (which reduces it about 5x per iteration on the benchmark workloads)
    if (st->nn_on && !st->nn_off) {
      if (v[0] < 0.5 * st->nn_best) {
        st->nn_best = v[0];
        st->nn_since = 0;
      } else if (++st->nn_since >= 2) {
        // the preconditioner changes from here on: the next iteration
        // restarts the search direction from the residual (p = r)
        st->nn_off = 1;
        st->restart = 1;
      }
    }
    if (st->omega == 0) {
      st->stat = 1;
      st->done = 1;
      return;
    }
    st->rho1 = st->rho;
    st->iter += 1;
    if (st->iter > st->max_iter) {
      st->iter = st->max_iter;
      st->done = 1;
      return;
    }
    st->rho = v[1];
    if (v[1] == 0) {
      st->stat = 1;
      st->done = 1;
      return;
    }
    st->beta = (st->rho / st->rho1) * (st->alpha / st->omega);
  }
};

// ---- kernels -------------------------------------------------------------
// the loop also ends where a bounded wait has run out (err)
__global__ void k_set_cond(cudaGraphConditionalHandle h, const FState *st, const int *err) {
  pdl_enter();
  cudaGraphSetConditional(h, st->done || *err ? 0u : 1u);
}

// x0 = sol, x = 0 on the tower
__global__ void k_pro_copy(BlockList L, int ncell, const double *sol, double *x0, double *x) {
  pdl_enter();
  const int total = L.n * ncell;
  for (int it = blockIdx.x * blockDim.x + threadIdx.x; it < total; it += gridDim.x * blockDim.x) {
    const long q = cell_of(L, ncell, it);
    x0[q] = sol[q];
    x[q] = 0.0;
  }
}

// p = r (first iteration) or p = r + beta*(p - omega*v) in the reference's two
// saxby steps; the V-cycle's residual (rhs - A*0) = masked p in precision T
template <typename T, bool MULTI>
__global__ void k_pupdate(BlockList L, int ncell, Chunks ch, FState *stb, const double *r, double *p, const double *v,
                          const double *vf, T *resid) {
  pdl_enter();
  const Work wk = work_of<MULTI>(ch, stb, list_count(L) * ncell, nullptr);
  const FState *st = wk.st;
  if (st->done) return;
  const bool first = st->iter == 1 || st->restart;
  const double beta = st->beta, om = st->omega;
  for (int it = wk.it0; it < wk.it1; it += wk.step) {
    const long q = cell_of(L, ncell, it);
    double pv;
    if (first) {
      pv = r[q];
    } else {
      pv = __fma_rn(beta, __fma_rn(-om, v[q], p[q]), r[q]);
    }
    p[q] = pv;
    resid[q] = fpint::positive(vf[q]) ? narrow_to<T>(pv) : (T)0;
  }
}

// s = r - alpha v ; x = x + alpha phat ; V-cycle residual = masked s ; |s|
// (phat: the FP64 V-cycle's output itself, or the FP32 one widened to FP64)
template <typename T, typename TP, bool MULTI>
__global__ void __launch_bounds__(kTPB) k_supdate(BlockList L, int ncell, Chunks ch, FState *stb, const double *r,
                                                const double *v, double *s, double *x, const TP *phat,
                                                const double *vf, T *resid, double *partials, unsigned *counter) {
  pdl_enter();
  const Work wk = work_of<MULTI>(ch, stb, list_count(L) * ncell, counter);
  FState *st = wk.st;
  if (st->done) return;
  const double a = st->alpha;
  unsigned long long mu = 0ull;  // max |s| as bit patterns (NaN-propagating)
  for (int it = wk.it0; it < wk.it1; it += wk.step) {
    const long q = cell_of(L, ncell, it);
    const double sv = __fma_rn(-a, v[q], r[q]);
    s[q] = sv;
    x[q] = __fma_rn(a, widen_from<TP>(phat[q]), x[q]);
    resid[q] = fpint::positive(vf[q]) ? narrow_to<T>(sv) : (T)0;
    mu = fpint::max_abs(mu, sv);
  }
  double m[1] = {fpint::from_bits(mu)};
  seg_reduce<1>(m, 1u, partials, wk.counter, wk.first, wk.count, wk.slot, EpiHalf{st});
}

// x = x + omega shat ; r = s - omega t ; |r| ; rhat.r
template <typename T, bool MULTI>
__global__ void __launch_bounds__(kTPB) k_rupdate(BlockList L, int ncell, Chunks ch, FState *stb, double *x,
                                                const T *shat, double *r, const double *s, const double *t,
                                                const double *rhat, double *partials, unsigned *counter) {
  pdl_enter();
  const Work wk = work_of<MULTI>(ch, stb, list_count(L) * ncell, counter);
  FState *st = wk.st;
  if (st->done) return;
  const double om = st->omega;
  unsigned long long mu = 0ull;  // max |r| as bit patterns (NaN-propagating)
  double m[2] = {0.0, 0.0};
  for (int it = wk.it0; it < wk.it1; it += wk.step) {
    const long q = cell_of(L, ncell, it);
    x[q] = __fma_rn(om, widen_from<T>(shat[q]), x[q]);
    const double rv = __fma_rn(-om, t[q], s[q]);
    r[q] = rv;
    mu = fpint::max_abs(mu, rv);
    m[1] = __fma_rn(rhat[q], rv, m[1]);
  }
  m[0] = fpint::from_bits(mu);
  seg_reduce<2>(m, 1u, partials, wk.counter, wk.first, wk.count, wk.slot, EpiEnd{st});
}

// after the loop: x0 += x ; sol = x0 when converged
template <bool MULTI>
__global__ void k_finish(BlockList L, int ncell, Chunks ch, const FState *stb, double *x0, const double *x,
                         double *sol) {
  pdl_enter();
  const Work wk = work_of<MULTI>(ch, const_cast<FState *>(stb), list_count(L) * ncell, nullptr);
  if (!wk.st->conv) return;
  for (int it = wk.it0; it < wk.it1; it += wk.step) {
    const long q = cell_of(L, ncell, it);
    const double v = x0[q] + x[q];
    x0[q] = v;
    sol[q] = v;
  }
}

// phat (FP64) = SOL(=0) + CORR over the tower, from precision T
template <typename T>
__global__ void k_vc_out(BlockList L, int ncell, const FState *st, const T *corr, double *out) {
  pdl_enter();
  if (st->done) return;
  const int total = list_count(L) * ncell;
  for (int it = blockIdx.x * blockDim.x + threadIdx.x; it < total; it += gridDim.x * blockDim.x) {
    const int p = it / ncell;
    if (block_off(L, L.blocks[p])) continue;
    const long q = (long)L.blocks[p] * ncell + (it - p * ncell);
    if constexpr (sizeof(T) == 4)
      out[q] = fpint::widen_plus0(corr[q]);
    else
      out[q] = 0.0 + corr[q];
  }
}

// every problem's state read: the loop goes on while one is not done; the
// shared state's done flag (the guard of the V-cycle kernels) is set once all
// are, or a bounded wait has run out (err)
__global__ void k_set_cond_multi(cudaGraphConditionalHandle h, const FState *stc, int ncomp, FState *st,
                                 const int *err) {
  pdl_enter();
  __shared__ int any;
  if (threadIdx.x == 0) any = 0;
  __syncthreads();
  int a = 0;
  for (int c = threadIdx.x; c < ncomp; c += blockDim.x) a |= !stc[c].done;
  if (a && !*err) atomicOr(&any, 1);
  __syncthreads();
  if (threadIdx.x == 0) {
    st->done = any ? 0 : 1;
    if (h) cudaGraphSetConditional(h, any ? 1u : 0u);
  }
}

// The outer BiCGSTAB's operator on the finest tower.  The reference evaluates
// y = (phi_c * sum T - sum T phi_nb) / dv / vf with two FP64 divisions per
// cell; GB300's FP64 rate is low, so the device solve folds everything that
// depends on the coefficients alone into two per-cell factors built once per
// coefficient set:
//   S = 1/(dv*vf) (0 where vf = 0),  P = D*S,
// D being the diagonal sum T with physical Dirichlet faces counted twice
// (their ghost value is -phi_c).  Then y = phi_c*P - S*sum' T phi_nb over the
// faces that are not physical boundaries, with FMA: 7 FMA + 1 multiply per
// cell instead of about 40 FP64 operations.  The result differs from the
// reference's operator by rounding only (about 1e-16 relative).
// One warp per block divides once for the block's full cells; a solid cell's
// factors are 0, and those of a constant-coefficient block's interior cells
// are its record's (the same values, see k_uniform), so the FP64 pipe sees the
// other cells only.
template <int ND>
__global__ void __launch_bounds__(kTPB) k_op_prep(Topo t, Coef<double> c, BlockList L, double *P, double *S) {
  using namespace stencil;
  const int nb = t.nb, lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
  for (int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < L.n; p += warps) {
    const int b = L.blocks[p];
    const uint16_t ft = L.ftypes[p];
    const double *u = uniform_of(c, b);
    const double dv = geom(c, b, 6), full = 1.0 / (dv * 1.0);
    for (int ci = lane; ci < t.ncell; ci += 32) {
      const long q = (long)b * t.ncell + ci;
      int ijk[3];
      decode_fast<ND>(ci, t, ijk);
      bool inner = true;
      for (int d = 0; d < ND; d++) inner = inner && ijk[d] > 0 && ijk[d] < nb - 1;
      if (u && inner) {
        P[q] = u[4];
        S[q] = u[5];
        continue;
      }
      const double vfv = c.vf[q];
      if (!positive(vfv)) {  // (a NaN is solid too, as everywhere else)
        P[q] = S[q] = 0.0;
        continue;
      }
      double diag = c.alpha * dv;
      for (int f = 0; f < 2 * ND; f++) {
        const int d = f >> 1, s = f & 1;
        const bool bnd = s ? ijk[d] == nb - 1 : ijk[d] == 0;
        const int fx = face_index(d, ijk, s, nb);
        const double tf = c.tff[d][(long)b * t.nfb + fx];
        if (!bnd) {
          diag += tf;
          continue;
        }
        const int ty = face_type_of(ft, f);
        if (ty == 0)
          diag += tf;
        else if (ty == 1)
          diag += t.bc_type[b * 6 + f] == kBCNeumann ? 0.0 : 2.0 * tf;
        else
          diag += cf_face<double, ND>(c, t, b, f, ijk);
      }
      const bool one = __double_as_longlong(vfv) == __double_as_longlong(1.0);
      const double sc = one ? full : 1.0 / (dv * vfv);
      S[q] = sc;
      P[q] = diag * sc;
    }
  }
}

// Factors of the FP64 smoother for every cell of a tower's block list:
// sa = dv*vf/diag, ia = 1/diag (0 where vf = 0), diag = alpha*dv + sum of
// the face coefficients with this tower's face types (physical Dirichlet
// faces twice, Neumann faces not at all), so the sweep needs no FP64 division
// and no diagonal sum.
template <int ND>
__global__ void __launch_bounds__(kTPB) k_smooth_factors(Topo t, Coef<double> c, BlockList L, double *sa,
                                                        double *ia) {
  using namespace stencil;
  const int nb = t.nb, total = L.n * t.ncell;
  for (int it = blockIdx.x * blockDim.x + threadIdx.x; it < total; it += gridDim.x * blockDim.x) {
    int p, ci, ijk[3];
    split_cell<ND>(it, t, p, ci);
    decode_fast<ND>(ci, t, ijk);
    const int b = L.blocks[p];
    const uint16_t ft = L.ftypes[p];
    const double dv = geom(c, b, 6);
    double diag = c.alpha * dv;
    for (int f = 0; f < 2 * ND; f++) {
      const int d = f >> 1, s = f & 1;
      const bool bnd = s ? ijk[d] == nb - 1 : ijk[d] == 0;
      const int fx = face_index(d, ijk, s, nb);
      const double tf = c.tff[d][(long)b * t.nfb + fx];
      if (!bnd) {
        diag += tf;
        continue;
      }
      const int ty = face_type_of(ft, f);
      if (ty == 0)
        diag += tf;
      else if (ty == 1)
        diag += t.bc_type[b * 6 + f] == kBCNeumann ? 0.0 : 2.0 * tf;
      else
        diag += cf_coef(c, t, b, d, fx, ty == 2 ? 1.5 : 0.75);
    }
    const double vfv = c.vf[(long)b * t.ncell + ci];
    const long o = (long)p * t.ncell + ci;
    // a fluid cell whose faces are all closed has no equation (diag 0): it
    // is left at zero instead of dividing by zero
    sa[o] = vfv > 0 && diag > 0 ? dv * vfv / diag : 0.0;
    ia[o] = vfv > 0 && diag > 0 ? 1.0 / diag : 0.0;
  }
}

// Constant-coefficient block records (Coef::ut), one CTA per block: a block
// qualifies when every face of direction d carries the same coefficient T_d
// (boundary faces included) and every cell has vf = 1, compared as bits (off
// the FP64 pipe).  Its interior cells'
// factors are those k_op_prep and k_smooth_factors compute, in the same
// order: diag = alpha*dv + T_0 + T_0 + T_1 + T_1 (+ T_2 + T_2).  The FP32
// record holds the FP32 coefficients, equal throughout the block too.  The FP32
// coefficients of a coarse/fine face (c32.cf) have to be one value as well, as
// the hybrid pass takes them per row: where B and the area fraction vary and
// their product doesn't, these may round apart.
template <int ND>
__global__ void __launch_bounds__(kTPB) k_uniform(Topo t, Coef<double> c, Coef<float> c32, double *u64,
                                                float *u32) {
  __shared__ int ok;
  for (int b = blockIdx.x; b < t.nblocks; b += gridDim.x) {
    if (threadIdx.x == 0) ok = 1;
    __syncthreads();
    const long fb = (long)b * t.nfb, cb = (long)b * t.ncell;
    bool good = true;
    for (int d = 0; d < ND; d++) {
      const double t0 = c.tff[d][fb];
      for (int i = threadIdx.x; i < t.nfb; i += blockDim.x)
        good = good && __double_as_longlong(c.tff[d][fb + i]) == __double_as_longlong(t0);
    }
    for (int i = threadIdx.x; i < t.ncell; i += blockDim.x)
      good = good && __double_as_longlong(c.vf[cb + i]) == __double_as_longlong(1.0);
    const int nface = ND == 3 ? t.nb * t.nb : t.nb;
    for (int f = 0; f < 2 * ND; f++) {
      const int n = t.neighbor[b * 6 + f];
      if (n != -1 && (n < 0 || t.child[n * 8] < 0)) continue;  // coarser, refined
      const float *cf = c32.cf + ((long)b * (2 * ND) + f) * nface;
      for (int i = threadIdx.x; i < nface; i += blockDim.x)
        good = good && __float_as_uint(cf[i]) == __float_as_uint(cf[0]);
    }
    if (!good) ok = 0;
    __syncthreads();
    if (threadIdx.x == 0) {
      double T[3] = {0.0, 0.0, 0.0};
      float T32[3] = {0.f, 0.f, 0.f};
      for (int d = 0; d < ND; d++) {
        T[d] = c.tff[d][fb];
        T32[d] = c32.tff[d][fb];
      }
      const double dv = c.geom[b * 8 + 6];
      double diag = c.alpha * dv;
      for (int f = 0; f < 2 * ND; f++) diag += T[f >> 1];
      const bool on = ok && diag > 0;
      const double sc = 1.0 / (dv * 1.0);
      double *u = u64 + (long)b * kUni;
      float *v = u32 + (long)b * kUni;
      for (int d = 0; d < 3; d++) {
        u[d] = T[d];
        v[d] = T32[d];
      }
      u[3] = on ? 1.0 : 0.0;
      v[3] = on ? 1.f : 0.f;
      u[4] = on ? diag * sc : 0.0;
      u[5] = on ? sc : 0.0;
      u[6] = on ? dv * 1.0 / diag : 0.0;
      u[7] = on ? 1.0 / diag : 0.0;
      for (int k = 4; k < kUni; k++) v[k] = 0.f;
    }
    __syncthreads();
  }
}

// the coefficients of the faces at coarser and at refined neighbours
// (Coef::cf), in the arithmetic of cf_coef
// (the FP32 table from the FP64 arrays, each value rounded to T first)
template <typename T, int ND>
__global__ void __launch_bounds__(kTPB) k_cf_faces(Topo t, Coef<double> c, T *__restrict__ cf) {
  using namespace stencil;
  const int nface = ND == 3 ? t.nb * t.nb : t.nb;
  const long total = (long)t.nblocks * 2 * ND * nface;
  for (long it = blockIdx.x * (long)blockDim.x + threadIdx.x; it < total; it += (long)gridDim.x * blockDim.x) {
    const int m = (int)(it % nface), f = (int)(it / nface % (2 * ND)), b = (int)(it / nface / (2 * ND));
    const int n = t.neighbor[b * 6 + f];
    const bool coarser = n == -1, refined = n >= 0 && t.child[n * 8] >= 0;
    if (!coarser && !refined) continue;
    const int d = f >> 1, s = f & 1, m0 = ND == 3 ? m % t.nb : m, m1 = ND == 3 ? m / t.nb : 0;
    const int ijk[3] = {d == 0 ? (s ? t.nb - 1 : 0) : m0, d == 0 ? m0 : (d == 1 ? (s ? t.nb - 1 : 0) : m1),
                        ND == 3 ? (d == 2 ? (s ? t.nb - 1 : 0) : m1) : 0};
    const long fx = (long)b * t.nfb + face_index(d, ijk, s, t.nb);
    T v = (T)c.beta * (T)geom(c, b, 3 + d) / ((T)geom(c, b, d) * (coarser ? (T)1.5 : (T)0.75));
    v = v * (T)c.bcoef[d][fx];
    cf[it] = v * (T)c.afrac[d][fx];
  }
}

// T S of the blocks whose faces all carry one coefficient (see k_op_rows), else 0
__global__ void k_iso(int nblocks, int nd, double alpha, const double *__restrict__ u64, double *__restrict__ iso) {
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nblocks; b += gridDim.x * blockDim.x) {
    const double *u = u64 + (long)b * kUni;
    const bool on = u[3] != 0.0 && alpha == 0.0 && u[0] == u[1] && (nd == 2 || u[0] == u[2]);
    iso[b] = on ? u[0] * u[5] : 0.0;
  }
}

// sum T * phi_nb over the faces of cell ijk that are not physical boundaries
template <int ND, typename TX>
__device__ __forceinline__ double op_offdiag(const Topo &t, const Coef<double> &c, int b, uint16_t ft,
                                             const int ijk[3], int ci, const TX *__restrict__ x,
                                             const int *__restrict__ hx = nullptr, const double *u = nullptr) {
  using namespace stencil;
  const int nb = t.nb;
  const long cb = (long)b * t.ncell;
  double off = 0.0;
#pragma unroll
  for (int f = 0; f < 2 * ND; f++) {
    const int d = f >> 1, s = f & 1;
    const bool bnd = s ? ijk[d] == nb - 1 : ijk[d] == 0;
    const int fx = face_index(d, ijk, s, nb);
    if (!bnd) {
      const int stride = d == 0 ? 1 : (d == 1 ? nb : nb * nb);
      off = __fma_rn(u ? u[d] : c.tff[d][(long)b * t.nfb + fx], widen_from<TX>(x[cb + ci + (s ? stride : -stride)]),
                     off);
    } else {
      const int ty = face_type_of(ft, f);
      if (ty == 0)
        off = __fma_rn(u ? u[d] : c.tff[d][(long)b * t.nfb + fx],
                       widen_from<TX>(same_level_ghost<TX, false>(t, b, f, ijk, x, hx)), off);
      else if (ty == 2)
        off = __fma_rn(cf_face<double, ND>(c, t, b, f, ijk), widen_from<TX>(fine_crse_ghost<TX, ND, false>(t, b, f, ijk, x, hx)),
                       off);
      else if (ty == 3)
        off += refined_sum<double, ND, false>(t, c, b, f, ijk, x, hx);
    }
  }
  return off;
}

// operator fused with its dot products:
// MODE 0: y = A x, rhat.y (EpiAlpha) ; MODE 1: y = A x, y.w, y.y (EpiOmega) ;
// MODE 2: y = y2 = w - A x (0 where vf = 0), |y|, y.y (EpiInit) ;
// MODE 3: only while verifying: y = y2 = w - A x, |y|, y.y (EpiVerify)
// The operator in double-float (mac_df.cuh) for an FP32 input x: the sum of
// T * x over the faces, then P * x - S * sum, with T, P and S as double-float
// pairs (the records' and the per-cell factors' nearest double-float values,
// T of a block without a record split on the fly); the coarse/fine faces'
// terms are formed in FP64 as in op_offdiag and added in double-float.  The
// result, about 48 significand bits, is rounded to FP64 once.
template <int ND>
__device__ __forceinline__ dfl::df op_offdiag_df(const Topo &t, const Coef<double> &c, int b, uint16_t ft,
                                                 const int ijk[3], int ci, const float *__restrict__ x,
                                                 const int *__restrict__ hx, const float2 *u2) {
  using namespace stencil;
  const int nb = t.nb;
  const long cb = (long)b * t.ncell;
  dfl::df off = {0.f, 0.f};
#pragma unroll
  for (int f = 0; f < 2 * ND; f++) {
    const int d = f >> 1, s = f & 1;
    const bool bnd = s ? ijk[d] == nb - 1 : ijk[d] == 0;
    const int fx = face_index(d, ijk, s, nb);
    if (!bnd) {
      const int stride = d == 0 ? 1 : (d == 1 ? nb : nb * nb);
      const dfl::df T = u2 ? dfl::load(u2 + d) : dfl::from_double(c.tff[d][(long)b * t.nfb + fx]);
      off = dfl::add(off, dfl::mul_f(T, x[cb + ci + (s ? stride : -stride)]));
    } else {
      const int ty = face_type_of(ft, f);
      if (ty == 0) {
        const dfl::df T = u2 ? dfl::load(u2 + d) : dfl::from_double(c.tff[d][(long)b * t.nfb + fx]);
        off = dfl::add(off, dfl::mul_f(T, same_level_ghost<float, false>(t, b, f, ijk, x, hx)));
      } else if (ty == 2) {
        off = dfl::add(off, dfl::mul_f(dfl::from_double(cf_face<double, ND>(c, t, b, f, ijk)),
                                       fine_crse_ghost<float, ND, false>(t, b, f, ijk, x, hx)));
      } else if (ty == 3) {
        off = dfl::add(off, dfl::from_double(refined_sum<double, ND, false>(t, c, b, f, ijk, x, hx)));
      }
    }
  }
  return off;
}

template <int ND, int MODE, typename TX, bool MULTI, bool DFOP = false>
__global__ void __launch_bounds__(kTPB, 4) k_op_red(Topo t, Coef<double> c, BlockList L, Chunks ch,
                                               const TX *__restrict__ x, double *__restrict__ y,
                                               const double *__restrict__ w, const double *__restrict__ P,
                                               const double *__restrict__ S, FState *stb, double *partials,
                                               unsigned *counter, double *__restrict__ y2 = nullptr,
                                               const float2 *__restrict__ P2 = nullptr,
                                               const float2 *__restrict__ S2 = nullptr,
                                               const float2 *__restrict__ U2 = nullptr) {
  using namespace stencil;
  pdl_enter();
  // DFOP: modes 0 and 1 of an FP32 input in double-float
  constexpr bool DF = DFOP && sizeof(TX) == 4 && MODE < 2;
  const Work wk = work_of<MULTI>(ch, stb, list_count(L) * t.ncell, counter);
  FState *st = wk.st;
  if (MODE == 3 && !st->verify) return;
  if (MODE < 2 && st->done) return;
  double acc[2] = {0.0, 0.0};
  unsigned long long mu = 0ull;  // MODE >= 2: max |y| as bit patterns
  for (int it = wk.it0; it < wk.it1; it += wk.step) {
    int p, ci, ijk[3];
    split_cell<ND>(it, t, p, ci);
    decode_fast<ND>(ci, t, ijk);
    const int *e = L.hx ? L.hx + (long)p * kHX : nullptr;
    const int b = e ? e[kHXBlock] : L.blocks[p];
    const uint16_t ft = e ? (uint16_t)(e[kHXInfo] & 0xffff) : L.ftypes[p];
    const long q = (long)b * t.ncell + ci;
    // constant-coefficient block: face coefficients and S from its record,
    // P too for an interior cell (the boundary cells' P depends on the face types)
    const double *u = uniform_of(c, b);
    bool inner = true;
#pragma unroll
    for (int d = 0; d < ND; d++) inner = inner && ijk[d] > 0 && ijk[d] < t.nb - 1;
    double yv;
    if constexpr (DF) {
      const float2 *u2 = u ? U2 + (long)b * kUni : nullptr;
      const dfl::df off = op_offdiag_df<ND>(t, c, b, ft, ijk, ci, x, e, u2);
      const dfl::df pf = (u2 && inner) ? dfl::load(u2 + 4) : dfl::load(P2 + q);
      const dfl::df sf = u2 ? dfl::load(u2 + 5) : dfl::load(S2 + q);
      yv = dfl::to_double(dfl::add(dfl::mul_f(pf, x[q]), dfl::neg(dfl::mul(off, sf))));
    } else {
      const double off = op_offdiag<ND, TX>(t, c, b, ft, ijk, ci, x, e, u);
      const double sc = u ? u[5] : S[q];
      yv = __fma_rn(widen_from<TX>(x[q]), (u && inner) ? u[4] : P[q], -off * sc);
    }
    if constexpr (MODE >= 2) yv = fpint::positive(u ? u[5] : S[q]) ? w[q] - yv : 0.0;
    y[q] = yv;
    if (MODE >= 2) y2[q] = yv;
    if (MODE == 0) acc[0] = __fma_rn(w[q], yv, acc[0]);
    if (MODE == 1) {
      acc[0] = __fma_rn(yv, w[q], acc[0]);
      acc[1] = __fma_rn(yv, yv, acc[1]);
    }
    if (MODE >= 2) {
      mu = fpint::max_abs(mu, yv);
      acc[1] = __fma_rn(yv, yv, acc[1]);
    }
  }
  if (MODE >= 2) acc[0] = fpint::from_bits(mu);
  if (MODE == 0) seg_reduce<2>(acc, 0u, partials, wk.counter, wk.first, wk.count, wk.slot, EpiAlpha{st});
  if (MODE == 1) seg_reduce<2>(acc, 0u, partials, wk.counter, wk.first, wk.count, wk.slot, EpiOmega{st});
  if (MODE == 2) seg_reduce<2>(acc, 1u, partials, wk.counter, wk.first, wk.count, wk.slot, EpiInit{st});
  if (MODE == 3) seg_reduce<2>(acc, 1u, partials, wk.counter, wk.first, wk.count, wk.slot, EpiVerify{st});
}

// N cells of k_op_rows at face f toward a coarser or refined neighbour, with
// transverse indices (i0 .. i0+N-1, i1): off += factor * value per cell (e: the
// block's halo descriptor).  A call keeps the kernel small; its N cells' loads
// are in flight together (cell by cell, a small problem's launch waited four
// times over: 15 us for 27 thousand cells).
template <int ND, int N>
static __device__ __noinline__ double4 op_cross(const double *__restrict__ cf, const float *__restrict__ x,
                                                const int *__restrict__ e, int nb, int nc, int f, int i0, int i1,
                                                double4 off) {
  const int d = f >> 1, half = nb >> 1, nface = ND == 3 ? nb * nb : nb, across = (f & 1) ? 0 : nb - 1;
  const int su = d == 0 ? nb : 1, sv = d == 2 ? nb : nb * nb, sd = d == 0 ? 1 : (d == 1 ? nb : nb * nb);
  const int info = e[kHXInfo];
  double k[N], v[N];
  if (((info >> (2 * f)) & 3) == 2) {
    const int wc = info >> 16, q0 = d == 0 ? 1 : 0, q1 = d == 2 ? 1 : 2;
    const int t0 = ((wc >> q0) & 1) * half, t1 = ND == 3 ? ((wc >> q1) & 1) * half + (i1 >> 1) : 0;
    const double *row = cf + ((long)e[kHXBlock] * (2 * ND) + f) * nface + i0 + nb * i1;
    const float *xc = x + (long)e[f] * nc + across * sd + t1 * sv;
#pragma unroll
    for (int n = 0; n < N; n++) {
      k[n] = row[n];
      v[n] = fpint::widen(xc[(t0 + ((i0 + n) >> 1)) * su]);
    }
  } else {
    // (four cells never straddle the halves of a face: nb / 2 is even, and
    // where it is not a multiple of 4 each cell finds its own fine block)
    const int h1 = ND == 3 && i1 >= half ? 1 : 0;
#pragma unroll
    for (int n = 0; n < N; n++) {
      const int h0 = i0 + n >= half ? 1 : 0;
      const long F = e[kHXKids + f * 4 + h0 + 2 * h1];
      const int t0 = 2 * (i0 + n - h0 * half), t1 = 2 * (i1 - h1 * half);
      const double *row = cf + (F * (2 * ND) + (f ^ 1)) * nface;
      const float *xf = x + F * nc + across * sd;
      double val = 0.0;
#pragma unroll
      for (int a1 = 0; a1 < (ND == 3 ? 2 : 1); a1++)
#pragma unroll
        for (int a0 = 0; a0 < 2; a0++)
          val += row[t0 + a0 + nb * (t1 + a1)] * fpint::widen(xf[(t0 + a0) * su + (t1 + a1) * sv]);
      k[n] = 1.0;
      v[n] = val;
    }
  }
  off.x = __fma_rn(k[0], v[0], off.x);
  if (N > 1) {
    off.y = __fma_rn(k[N > 1 ? 1 : 0], v[N > 1 ? 1 : 0], off.y);
    off.z = __fma_rn(k[N > 2 ? 2 : 0], v[N > 2 ? 2 : 0], off.z);
    off.w = __fma_rn(k[N > 3 ? 3 : 0], v[N > 3 ? 3 : 0], off.w);
  }
  return off;
}

// The operator with its dot products (modes 0 and 1 of k_op_red) on an FP32
// input, blocks whose edge is a multiple of 4 cells: a thread takes four cells
// of a row, whose neighbours along y and z are four cells of another row (of
// the block, or of the neighbour behind a same-level face) and lie in the
// thread's own 16 bytes along x, so the loads are 16 bytes wide and no cell
// inside a warp takes another path than the next one.
//
// In a block whose faces all carry one coefficient T and whose cells are
// fluid (iso: T S, alpha 0), y = T S (n x_c - sum x_nb), n counting same-level
// faces once, Dirichlet faces twice (their ghost is -x_c), Neumann faces not
// at all.  The difference is formed exactly on the FP32 pipe
// (dfl::exact_delta): a cell then takes an addition and a product of FP64
// instead of 2 ND + 2 multiply-adds, which is what bounds this kernel (GB300:
// two FP64 lanes per SM and clock).  Other blocks take the general form of
// k_op_red on the same loads, the coarse/fine faces among them from their
// table (Coef::cf: without it each costs a division on the FP64 pipe).
template <int ND, int MODE, bool MULTI>
__global__ void __launch_bounds__(kTPB, 4) k_op_rows(Topo t, Coef<double> c, BlockList L, Chunks ch,
                                                   const float *__restrict__ x, double *__restrict__ y,
                                                   const double *__restrict__ w, const double *__restrict__ P,
                                                   const double *__restrict__ S, FState *stb, double *partials,
                                                   unsigned *counter, const double *__restrict__ iso, int per) {
  using namespace stencil;
  pdl_enter();
  Work wk = work_of<MULTI>(ch, stb, list_count(L) * t.ncell, counter);
  FState *st = wk.st;
  if (st->done) return;
  const int nb = t.nb, nc = t.ncell;
  double acc[2] = {0.0, 0.0};
  // MULTI: the CTA's chunk; else `per` threads of every CTA work, so that a
  // small problem reaches as many SMs, each with its own FP64 pipe, as it can
  const int tid = threadIdx.x;
  const int first = MULTI ? wk.it0 + 3 * tid : 4 * ((int)blockIdx.x * per + tid);
  const int step = 4 * (MULTI ? (int)blockDim.x : (int)gridDim.x * per);
  for (int it = MULTI || tid < per ? first : wk.it1; it < wk.it1; it += step) {
    int p, ci, ijk[3];
    split_cell<ND>(it, t, p, ci);
    decode_fast<ND>(ci, t, ijk);
    const int *e = L.hx + (long)p * kHX;
    const int2 ib = *reinterpret_cast<const int2 *>(e + kHXInfo);
    const int b = ib.y;
    const uint16_t ft = (uint16_t)(ib.x & 0xffff);
    const long cb = (long)b * nc;
    const float *xb = x + cb + ci;
    const double K = iso[b];
    // the six (four) neighbour rows: v[0], v[1] the cells left and right of
    // the four, r[] the four cells below and above them per direction
    float4 r[2 * (ND - 1)];
    float vx[2] = {0.f, 0.f};
    float nrow = 2.f * ND, nl = 0.f, nr = 0.f;  // multiplicity of x_c, and of the first and last cell
    bool cf = false;
    const float4 xc = *reinterpret_cast<const float4 *>(xb);
#pragma unroll
    for (int f = 0; f < 2 * ND; f++) {
      const int d = f >> 1, s = f & 1, stride = d == 0 ? 1 : (d == 1 ? nb : nb * nb);
      const bool bnd = d == 0 ? (s ? ijk[0] + 4 == nb : ijk[0] == 0) : (s ? ijk[d] == nb - 1 : ijk[d] == 0);
      const float *q = xb + (d == 0 ? (s ? 4 : -1) : (s ? stride : -stride));
      bool there = true;
      if (bnd) {
        const int ty = face_type_of(ft, f);
        there = ty == 0;
        cf = cf || ty > 1;
        if (ty == 0) {
          q = x + (long)e[f] * nc + ci + (d == 0 ? (s ? 4 - nb : nb - 1) : (s ? (1 - nb) * stride : (nb - 1) * stride));
        } else if (ty == 1) {
          const float n = t.bc_type[b * 6 + f] == kBCNeumann ? -1.f : 1.f;
          if (d > 0)
            nrow += n;
          else if (s)
            nr = n;
          else
            nl = n;
        }
      }
      if (d == 0)
        vx[s] = there ? *q : 0.f;
      else
        r[f >= 2 ? f - 2 : 0] = there ? *reinterpret_cast<const float4 *>(q) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const double2 wa = *reinterpret_cast<const double2 *>(w + cb + ci);
    const double2 wb = *reinterpret_cast<const double2 *>(w + cb + ci + 2);
    const float xv[6] = {vx[0], xc.x, xc.y, xc.z, xc.w, vx[1]};
    double yv[4];
    bool done = false;
    if (__double_as_longlong(K) != 0 && !cf) {  // uniform over a block but for its coarse/fine faces
      done = true;
#pragma unroll
      for (int n = 0; n < 4; n++) {
        float v[2 * ND];
        v[0] = xv[n];
        v[1] = xv[n + 2];
#pragma unroll
        for (int q = 0; q < 2 * (ND - 1); q++) v[2 + q] = n == 0 ? r[q].x : n == 1 ? r[q].y : n == 2 ? r[q].z : r[q].w;
        const double dl = dfl::exact_delta<ND>(nrow + (n == 0 ? nl : 0.f) + (n == 3 ? nr : 0.f), xv[n + 1], v);
        // an overflow of the FP32 sums: the general form
        done = done && (__double2hiint(dl) & 0x7ff00000) != 0x7ff00000;
        yv[n] = K * dl;
      }
    }
    if (!done) {
      const long fb = (long)b * t.nfb;
      const int row = ijk[1] + nb * ijk[2];
      const double *tx = c.tff[0] + fb + (nb + 1) * row + ijk[0];
      const double2 *p2 = reinterpret_cast<const double2 *>(P + cb + ci), *s2 = reinterpret_cast<const double2 *>(S + cb + ci);
      const double2 pa = p2[0], pb = p2[1], sa = s2[0], sb = s2[1];
      double xw[6], tk[5];
#pragma unroll
      for (int n = 0; n < 6; n++) xw[n] = fpint::widen(xv[n]);
#pragma unroll
      for (int n = 0; n < 5; n++) tk[n] = tx[n];
      // left and right, the first and last cell's across the block's edge
      const double4 zero = make_double4(0.0, 0.0, 0.0, 0.0);
      double l0 = __fma_rn(tk[0], xw[0], 0.0);
      if (cf && ijk[0] == 0 && face_type_of(ft, 0) > 1) l0 = op_cross<ND, 1>(c.cf, x, e, nb, nc, 0, ijk[1], ijk[2], zero).x;
      double4 off = make_double4(__fma_rn(tk[1], xw[2], l0), __fma_rn(tk[2], xw[3], __fma_rn(tk[1], xw[1], 0.0)),
                                 __fma_rn(tk[3], xw[4], __fma_rn(tk[2], xw[2], 0.0)), __fma_rn(tk[3], xw[3], 0.0));
      if (cf && ijk[0] + 4 == nb && face_type_of(ft, 1) > 1)
        off.w = op_cross<ND, 1>(c.cf, x, e, nb, nc, 1, ijk[1], ijk[2], make_double4(off.w, 0.0, 0.0, 0.0)).x;
      else
        off.w = __fma_rn(tk[4], xw[5], off.w);
#pragma unroll
      for (int f = 2; f < 2 * ND; f++) {
        const int d = f >> 1, s = f & 1;
        if (cf && (s ? ijk[d] == nb - 1 : ijk[d] == 0) && face_type_of(ft, f) > 1) {
          off = op_cross<ND, 4>(c.cf, x, e, nb, nc, f, ijk[0], d == 1 ? ijk[2] : ijk[1], off);
        } else {
          const long fx = d == 1 ? ijk[0] + nb * (ijk[1] + s + (nb + 1) * ijk[2]) : ci + s * nb * nb;
          const double2 *tf = reinterpret_cast<const double2 *>(c.tff[d] + fb + fx);
          const double2 ka = tf[0], kb = tf[1];
          const float4 q = r[f - 2];
          off.x = __fma_rn(ka.x, fpint::widen(q.x), off.x);
          off.y = __fma_rn(ka.y, fpint::widen(q.y), off.y);
          off.z = __fma_rn(kb.x, fpint::widen(q.z), off.z);
          off.w = __fma_rn(kb.y, fpint::widen(q.w), off.w);
        }
      }
      yv[0] = __fma_rn(xw[1], pa.x, -off.x * sa.x);
      yv[1] = __fma_rn(xw[2], pa.y, -off.y * sa.y);
      yv[2] = __fma_rn(xw[3], pb.x, -off.z * sb.x);
      yv[3] = __fma_rn(xw[4], pb.y, -off.w * sb.y);
    }
    *reinterpret_cast<double2 *>(y + cb + ci) = make_double2(yv[0], yv[1]);
    *reinterpret_cast<double2 *>(y + cb + ci + 2) = make_double2(yv[2], yv[3]);
    const double wv[4] = {wa.x, wa.y, wb.x, wb.y};
#pragma unroll
    for (int n = 0; n < 4; n++) {
      acc[0] = __fma_rn(wv[n], yv[n], acc[0]);
      if (MODE == 1) acc[1] = __fma_rn(yv[n], yv[n], acc[1]);
    }
  }
  if (MODE == 0) {
    double a[1] = {acc[0]};
    seg_reduce<1>(a, 0u, partials, wk.counter, wk.first, wk.count, wk.slot, EpiAlpha{st});
  } else {
    seg_reduce<2>(acc, 0u, partials, wk.counter, wk.first, wk.count, wk.slot, EpiOmega{st});
  }
}

// while verifying: x0 += x, x = 0 (the pass's solution folded into x0)
template <bool MULTI>
__global__ void __launch_bounds__(kTPB) k_verify_fold(BlockList L, int ncell, Chunks ch, const FState *stb,
                                                    double *x0, double *x) {
  pdl_enter();
  const Work wk = work_of<MULTI>(ch, const_cast<FState *>(stb), list_count(L) * ncell, nullptr);
  if (!wk.st->verify) return;
  for (int it = wk.it0; it < wk.it1; it += wk.step) {
    const long q = cell_of(L, ncell, it);
    x0[q] = x0[q] + x[q];
    x[q] = 0.0;
  }
}

// dense bottom solve: corr(level 1) = Binv * resid(level 1), one CTA per
// tile of rows of one component
template <typename T>
__global__ void __launch_bounds__(kTPB) k_bottom_gemv(BottomDev bd, const T *__restrict__ resid,
                                                    T *__restrict__ corr, const FState *st) {
  pdl_enter();
  if (st && st->done) return;
  extern __shared__ double rv[];
  stencil::bottom_tile<T>(bd, blockIdx.x, resid, corr, rv);
}

// Gauss-Jordan inversion step k of nmat matrices of order m at offsets offs
// (no pivoting: the pinned, row-scaled bottom operator has positive pivots),
// from a into b (there at offsets `to`), so that one launch per step is enough:
// the pivot row and column are read where they are while every other entry is
// written.  One CTA per matrix row; the row of the next pivot also writes its reciprocal,
// ipiv[mat][k + 1], so that no CTA waits for a division.  (With the row and
// column saved by a launch of their own and the step in place, an inversion
// of order 512 took 2.6 ms, half of it the saving launches.)
__global__ void k_gj_first(int m, int nmat, const long long *__restrict__ offs, const double *__restrict__ a,
                           double *__restrict__ ipiv) {
  const int mat = blockIdx.x * blockDim.x + threadIdx.x;
  if (mat < nmat) ipiv[(long)mat * m] = 1.0 / a[offs[mat]];
}
__global__ void __launch_bounds__(kTPB) k_gj_step(int m, int k, int nmat, const long long *__restrict__ offs,
                                                const double *__restrict__ a, const long long *__restrict__ to,
                                                double *__restrict__ b, double *__restrict__ ipiv) {
  const long rows = (long)nmat * m;
  for (long r = blockIdx.x; r < rows; r += gridDim.x) {
    const int mat = (int)(r / m), i = (int)(r - (long)mat * m);
    const double *am = a + offs[mat], *rw = am + (long)k * m, *ar = am + (long)i * m;
    double *br = b + to[mat] + (long)i * m;
    const double ip = ipiv[(long)mat * m + k];
    if (i == k) {
      for (int j = threadIdx.x; j < m; j += blockDim.x) br[j] = j == k ? ip : rw[j] * ip;
    } else {
      const double f = ar[k] * ip;
      for (int j = threadIdx.x; j < m; j += blockDim.x) {
        const double v = j == k ? -f : __fma_rn(-f, rw[j], ar[j]);
        br[j] = v;
        if (i == k + 1 && j == i) ipiv[(long)mat * m + i] = 1.0 / v;
      }
    }
  }
}
// zero column col of the order-m matrix at off (a pinned Neumann cell)
// FP16 copy of the bottom inverse, one CTA per row: scale = max |a| of the
// row, h = a / scale rounded to nearest
__global__ void __launch_bounds__(kTPB) k_half_rows(int nrows, const long long *row_off, const int *row_m,
                                                  const double *a, unsigned short *h, float *scale) {
  __shared__ double sh[kTPB / 32];
  for (int g = blockIdx.x; g < nrows; g += gridDim.x) {
    const double *ar = a + row_off[g];
    const int m = row_m[g];
    double mx = 0.0;
    for (int j = threadIdx.x; j < m; j += blockDim.x) mx = fmax(mx, fabs(ar[j]));
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = mx;
    __syncthreads();
    mx = 0.0;
    for (int q = 0; q < kTPB / 32; q++) mx = fmax(mx, sh[q]);
    const double inv = mx > 0 ? 1.0 / mx : 0.0;
    for (int j = threadIdx.x; j < m; j += blockDim.x)
      h[row_off[g] + j] = __half_as_ushort(__double2half(ar[j] * inv));
    if (threadIdx.x == 0) scale[g] = (float)mx;
    __syncthreads();
  }
}

// FP32 copy of the bottom inverse
__global__ void k_narrow(long long n, const double *a, float *b) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    b[i] = (float)a[i];
}

__global__ void k_zero_col(long long off, int m, int col, double *a) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < m; r += gridDim.x * blockDim.x) a[off + (long)r * m + col] = 0.0;
}

// nearest double-float pairs of FP64 values
__global__ void k_split_df(long n, const double *src, float2 *dst) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const dfl::df v = dfl::from_double(src[i]);
    dst[i] = make_float2(v.hi, v.lo);
  }
}

__global__ void k_to_f32(long n, const double *src, float *dst) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    dst[i] = fpint::narrow(src[i]);  // a hardware conversion is an FP64-pipe operation
}

}  // namespace

// ---------------------------------------------------------------------------
void MacGpu::ensure_fast_buffers() {
  if (fast_ready_) return;
  const int nd = tt_.ndim, nbk = tt_.num_blocks;
  const size_t nc = (size_t)nbk * ncell_, nf = (size_t)nbk * nfb_;
  auto fa = [&](size_t n) {
    float *p = nullptr;
    if (dev_malloc(&p, std::max<size_t>(n, 1) * sizeof(float)) != cudaSuccess) fail("out of device memory (fp32)");
    else cudaMemsetAsync(p, 0, std::max<size_t>(n, 1) * sizeof(float), stream_);
    return p;
  };
  for (int d = 0; d < nd; d++) {
    d_tff32_[d] = fa(nf);
    d_bcoef32_[d] = fa(nf);
    d_afrac32_[d] = fa(nf);
  }
  d_vf32_ = fa(nc);
  d_geom32_ = fa((size_t)nbk * 8);
  d_resid32_ = fa(nc);
  d_corr32_ = fa(nc);
  d_corr32b_ = fa(nc);
  if (dev_malloc(&d_corr64b_, nc * sizeof(double)) != cudaSuccess) fail("out of device memory (correction)");
  else cudaMemsetAsync(d_corr64b_, 0, nc * sizeof(double), stream_);
  if (dev_malloc(&d_opP_, nc * sizeof(double)) != cudaSuccess) fail("out of device memory (operator factors)");
  if (dev_malloc(&d_opS_, nc * sizeof(double)) != cudaSuccess) fail("out of device memory (operator factors)");
  if (dev_malloc(&d_opP2_, nc * sizeof(float2)) != cudaSuccess ||
      dev_malloc(&d_opS2_, nc * sizeof(float2)) != cudaSuccess ||
      dev_malloc(&d_uni2_, (size_t)std::max(nbk, 1) * kUni * sizeof(float2)) != cudaSuccess)
    fail("out of device memory (operator factors)");
  else
    cudaMemsetAsync(d_uni2_, 0, (size_t)std::max(nbk, 1) * kUni * sizeof(float2), stream_);
  if (dev_malloc(&d_uni64_, (size_t)std::max(nbk, 1) * kUni * sizeof(double)) != cudaSuccess ||
      dev_malloc(&d_uni32_, (size_t)std::max(nbk, 1) * kUni * sizeof(float)) != cudaSuccess ||
      dev_malloc(&d_iso_, (size_t)std::max(nbk, 1) * sizeof(double)) != cudaSuccess)
    fail("out of device memory (block records)");
  else {
    cudaMemsetAsync(d_uni64_, 0, (size_t)std::max(nbk, 1) * kUni * sizeof(double), stream_);
    cudaMemsetAsync(d_iso_, 0, (size_t)std::max(nbk, 1) * sizeof(double), stream_);
    cudaMemsetAsync(d_uni32_, 0, (size_t)std::max(nbk, 1) * kUni * sizeof(float), stream_);
  }
  if (dev_malloc(&d_st_, sizeof(FState)) != cudaSuccess) fail("alloc state");
  if (cudaMallocHost(&h_st_, sizeof(FState)) != cudaSuccess) fail("alloc pinned state");
  if (cudaMallocHost(&h_err_, sizeof(int)) != cudaSuccess) fail("alloc pinned error word");
  if (dev_malloc(&d_part_, sizeof(double) * kMaxRedBlocks * 4) != cudaSuccess) fail("alloc partials");
  if (dev_malloc(&d_cnt_, sizeof(unsigned) * 4) != cudaSuccess) fail("alloc counter");
  cudaMemsetAsync(d_cnt_, 0, sizeof(unsigned) * 4, stream_);
  {
    const size_t ncf = (size_t)std::max(nbk, 1) * 2 * nd * (nd == 3 ? tt_.nb * tt_.nb : tt_.nb);
    if (dev_malloc(&d_cf64_, ncf * sizeof(double)) != cudaSuccess ||
        dev_malloc(&d_cf32_, ncf * sizeof(float)) != cudaSuccess) {
      fail("out of device memory (coarse/fine faces)");
    } else {
      cudaMemsetAsync(d_cf64_, 0, ncf * sizeof(double), stream_);
      cudaMemsetAsync(d_cf32_, 0, ncf * sizeof(float), stream_);
    }
  }
  c32_.geom = d_geom32_;
  for (int d = 0; d < 3; d++) {
    const int dd = d < nd ? d : 0;
    c32_.tff[d] = d_tff32_[dd];
    c32_.bcoef[d] = d_bcoef32_[dd];
    c32_.afrac[d] = d_afrac32_[dd];
  }
  c32_.vf = d_vf32_;
  fast_ready_ = true;
}

// the FP64 smoother factors of the current coefficients, built on first need
void MacGpu::ensure_smooth_factors() {
  if (sfac_version_ == coef_version_) return;
  build_smooth_factors();
  sfac_version_ = coef_version_;
}

// FP64 smoother factors for the towers the V-cycle smooths (2 .. finest)
void MacGpu::build_smooth_factors() {
  if ((int)d_sfac_.size() < finest_ + 1) d_sfac_.resize(finest_ + 1, nullptr);
  for (int l = 2; l <= finest_; l++) {
    const BlockList TL = tower_list(l);
    const long w = (long)TL.n * ncell_;
    if (w == 0) continue;
    if (!d_sfac_[l] && dev_malloc(&d_sfac_[l], 2 * w * sizeof(double)) != cudaSuccess) {
      d_sfac_[l] = nullptr;
      fail("out of device memory (smoother factors)");
      return;
    }
    if (tt_.ndim == 2)
      k_smooth_factors<2><<<ew_grid(w), kTPB, 0, stream_>>>(topo_, c64_, TL, d_sfac_[l], d_sfac_[l] + w);
    else
      k_smooth_factors<3><<<ew_grid(w), kTPB, 0, stream_>>>(topo_, c64_, TL, d_sfac_[l], d_sfac_[l] + w);
    CK(cudaGetLastError());
  }
  // the same factors for the parity-grouped lists (same cells, regrouped)
  if ((int)d_pfac_.size() < finest_ + 1) d_pfac_.resize(finest_ + 1, nullptr);
  for (int l = 2; l <= finest_; l++) {
    const DevTower &tw = towers_[l];
    const BlockList PL{tw.par.blocks, tw.par.ftypes, tw.par.n};
    const long w = (long)PL.n * ncell_;
    if (w == 0) continue;
    if (!d_pfac_[l] && dev_malloc(&d_pfac_[l], 2 * w * sizeof(double)) != cudaSuccess) {
      d_pfac_[l] = nullptr;
      fail("out of device memory (smoother factors)");
      return;
    }
    if (tt_.ndim == 2)
      k_smooth_factors<2><<<ew_grid(w), kTPB, 0, stream_>>>(topo_, c64_, PL, d_pfac_[l], d_pfac_[l] + w);
    else
      k_smooth_factors<3><<<ew_grid(w), kTPB, 0, stream_>>>(topo_, c64_, PL, d_pfac_[l], d_pfac_[l] + w);
    CK(cudaGetLastError());
  }
}

// Autotuner of the device smoother: every launch-bounds variant (register
// cap) of k_rbgs is timed on the finest level of the finest tower -- the
// largest smoother launch of a V-cycle -- and the fastest is used by the
// V-cycle from then on.  The variants compute identical values, so the
// choice changes timing only.  Runs once per solver and precision (again
// after a forced variant is released), before the graph is captured.
void MacGpu::tune_smoother(int precision) {
  const int pi = precision == 1 ? 1 : 0;
  if (prm_.smooth_variant >= 0) {
    rbgs_variant_[pi] = std::min(prm_.smooth_variant, kRbgsVariants - 1);
    return;
  }
  if (rbgs_variant_[pi] >= 0 && rbgs_us_[pi][0] > 0) return;
  solve_lists_ = true;  // the list the solve will walk
  const BlockList sl = sublevel_list(finest_, finest_);
  solve_lists_ = false;
  if (sl.n == 0) {
    rbgs_variant_[pi] = 2;
    return;
  }
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  // with one state per problem the sweeps leave finished problems alone, and
  // after a solve all of them are: no problem is finished while they are timed
  if (multi()) {
    CK(cudaMemcpyAsync(h_stc_, d_stc_, ncomp_ * sizeof(FState), cudaMemcpyDeviceToHost, stream_));
    CK(cudaMemsetAsync(d_stc_, 0, ncomp_ * sizeof(FState), stream_));
  }
  const int reps = 6;
  float best = 1e30f;
  int bi = 2;
  for (int v = 0; v < kRbgsVariants; v++) {
    auto go = [&](int color) {
      if (pi)
        launch_rbgs<float>(topo_, c32_, sl, color, d_corr32_, d_resid32_, nullptr, stream_, false, v);
      else
        launch_rbgs<double>(topo_, cd64_, sl, color, vec_[kCORR], vec_[kRESID], nullptr, stream_, false, v);
    };
    go(0);
    go(1);
    CK(cudaEventRecord(e0, stream_));
    for (int r = 0; r < reps; r++) go(r & 1);
    CK(cudaEventRecord(e1, stream_));
    CK(cudaEventSynchronize(e1));
    float ms = 0.f;
    CK(cudaEventElapsedTime(&ms, e0, e1));
    rbgs_us_[pi][v] = ms * 1e3f / reps;
    // a variant whose bounded waits ran out is not a candidate
    if (rbgs_bulk_error(topo_.err, stream_, true) != 0) rbgs_us_[pi][v] = 1e30f;
    if (rbgs_us_[pi][v] < best) {
      best = rbgs_us_[pi][v];
      bi = v;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  // (the last solve's states can still be asked for)
  if (multi())
    CK(cudaMemcpyAsync(d_stc_, h_stc_, ncomp_ * sizeof(FState), cudaMemcpyHostToDevice, stream_));
  rbgs_variant_[pi] = bi;
  // the sweeps above scribbled on the V-cycle work vectors
  const size_t n = (size_t)tt_.num_blocks * ncell_;
  if (pi) {
    CK(cudaMemsetAsync(d_corr32_, 0, n * sizeof(float), stream_));
    CK(cudaMemsetAsync(d_resid32_, 0, n * sizeof(float), stream_));
  } else {
    CK(cudaMemsetAsync(vec_[kCORR], 0, n * sizeof(double), stream_));
    CK(cudaMemsetAsync(vec_[kRESID], 0, n * sizeof(double), stream_));
  }
}

int MacGpu::tuned_smoother(int precision, float *us, int n) const {
  const int pi = precision == 1 ? 1 : 0;
  for (int v = 0; v < n && v < kRbgsVariants; v++) us[v] = rbgs_us_[pi][v];
  return rbgs_variant_[pi];
}

// per-cell factors of the device solve's FP64 operator on the finest tower
void MacGpu::build_op_factors() {
  const BlockList TL = tower_list(finest_);
  const long w = (long)TL.n * ncell_;
  if (w == 0) return;
  Coef<double> cc = c64_;
  cc.cf = d_cf64_;
  cc.ut = d_uni64_;
  if (tt_.ndim == 2)
    k_op_prep<2><<<ew_grid(32l * TL.n), kTPB, 0, stream_>>>(topo_, cc, TL, d_opP_, d_opS_);
  else
    k_op_prep<3><<<ew_grid(32l * TL.n), kTPB, 0, stream_>>>(topo_, cc, TL, d_opP_, d_opS_);
  CK(cudaGetLastError());
}

// double-float pairs of the operator factors and block records, for the
// double-float operator only (params.vcycle_out 1)
void MacGpu::ensure_df_factors() {
  if (df_version_ == coef_version_) return;
  const long nc = (long)tt_.num_blocks * ncell_, nu = (long)tt_.num_blocks * kUni;
  k_split_df<<<ew_grid(nc), kTPB, 0, stream_>>>(nc, d_opP_, d_opP2_);
  k_split_df<<<ew_grid(nc), kTPB, 0, stream_>>>(nc, d_opS_, d_opS2_);
  k_split_df<<<ew_grid(nu), kTPB, 0, stream_>>>(nu, d_uni64_, d_uni2_);
  CK(cudaGetLastError());
  df_version_ = coef_version_;
}

// The arrays that only some parameters read, from the current coefficients: the
// FP64 smoother factors (the FP64 V-cycle and the learned correction), the
// double-float factors (vcycle_out 1) and the FP32 copies of B and the area
// fractions (the learned correction).  A solve without a captured graph may run
// with other parameters than its preparation saw, so every solve asks for what
// it reads; all three return at once where nothing changed.
void MacGpu::ensure_derived() {
  if (prm_.precision == 0 || learned_active()) ensure_smooth_factors();
  if (prm_.vcycle_out == 1) ensure_df_factors();
  if (learned_active()) ensure_fp32_faces();
}

// the coarse/fine face tables from the current coefficients
void MacGpu::build_cf() {
  const long n = (long)tt_.num_blocks * 2 * tt_.ndim * (tt_.ndim == 3 ? tt_.nb * tt_.nb : tt_.nb);
  if (n == 0) return;
  auto go = [&](auto k64, auto k32) {
    k64<<<ew_grid(n), kTPB, 0, stream_>>>(topo_, c64_, d_cf64_);
    k32<<<ew_grid(n), kTPB, 0, stream_>>>(topo_, c64_, d_cf32_);
  };
  if (tt_.ndim == 2)
    go(k_cf_faces<double, 2>, k_cf_faces<float, 2>);
  else
    go(k_cf_faces<double, 3>, k_cf_faces<float, 3>);
  CK(cudaGetLastError());
}

// constant-coefficient block records from the current coefficients (after
// refresh_fp32: the FP32 record takes the FP32 face coefficients)
void MacGpu::build_uniform() {
  const int nbk = tt_.num_blocks;
  if (nbk == 0) return;
  const int grid = std::min(nbk, 152 * 8);
  Coef<float> c32 = c32_;
  c32.cf = d_cf32_;
  if (tt_.ndim == 2)
    k_uniform<2><<<grid, kTPB, 0, stream_>>>(topo_, c64_, c32, d_uni64_, d_uni32_);
  else
    k_uniform<3><<<grid, kTPB, 0, stream_>>>(topo_, c64_, c32, d_uni64_, d_uni32_);
  k_iso<<<std::min((nbk + kTPB - 1) / kTPB, 152 * 8), kTPB, 0, stream_>>>(nbk, tt_.ndim, alpha_, d_uni64_, d_iso_);
  CK(cudaGetLastError());
}

// the coefficients the device solve's kernels read: with params.uniform the
// records of the constant-coefficient blocks, else the face arrays only
void MacGpu::bind_uniform() {
  cd64_ = c64_;
  cd64_.ut = prm_.uniform ? d_uni64_ : nullptr;
  c32_.ut = prm_.uniform ? d_uni32_ : nullptr;
  cd64_.cf = d_cf64_;
  c32_.cf = d_cf32_;
  // the smoothers' relaxation weight (1: plain Gauss-Seidel, the reference's)
  cd64_.omega = prm_.relax_omega;
  c32_.omega = (float)prm_.relax_omega;
}

// FP32 copies of the coefficients for the FP32 V-cycle
void MacGpu::refresh_fp32() {
  const int nd = tt_.ndim, nbk = tt_.num_blocks;
  const long nc = (long)nbk * ncell_, nf = (long)nbk * nfb_;
  for (int d = 0; d < nd; d++) {
    k_to_f32<<<ew_grid(nf), kTPB, 0, stream_>>>(nf, d_tff_[d], d_tff32_[d]);
  }
  k_to_f32<<<ew_grid(nc), kTPB, 0, stream_>>>(nc, d_vf_, d_vf32_);
  k_to_f32<<<ew_grid((long)nbk * 8), kTPB, 0, stream_>>>((long)nbk * 8, d_geom_, d_geom32_);
  c32_.alpha = (float)alpha_;
  c32_.beta = (float)beta_;
}

// FP32 copies of B and the area fractions, which only the learned correction
// reads (the V-cycle takes its coarse/fine coefficients from Coef::cf)
void MacGpu::ensure_fp32_faces() {
  if (faces32_version_ == coef_version_) return;
  const long nf = (long)tt_.num_blocks * nfb_;
  for (int d = 0; d < tt_.ndim; d++) {
    k_to_f32<<<ew_grid(nf), kTPB, 0, stream_>>>(nf, d_bcoef_[d], d_bcoef32_[d]);
    k_to_f32<<<ew_grid(nf), kTPB, 0, stream_>>>(nf, d_afrac_[d], d_afrac32_[d]);
  }
  CK(cudaGetLastError());
  faces32_version_ = coef_version_;
}

// Level of the dense bottom solve.  Level 1 always works (it is uniform and
// every level-1 face is a same-level or physical face); a finer level B
// replaces the V-cycle's levels 1..B by one dense solve when tower B is one
// uniform level (no coarse leaves, no coarse/fine faces) whose connected
// components have at most kBottomMaxCells cells and whose inverses fit in
// kBottomMaxBytes.  The auto choice takes the finest such level below the
// finest level, with components of at most kBottomAutoCells[ndim] cells: the
// dense product of a 4096-cell component streams a 64 MB FP32 matrix from
// DRAM per V-cycle (and pushes the V-cycle's working set out of L2), which
// in 2D costs as much as the cheap coarse levels it replaces (the 2D
// benchmark workload: 4.48 vs 4.02 ms per solve), while in 3D it replaces
// dearer levels and saves iterations (the elbow workload: 46.8 vs 53.5 ms,
// 11 vs 13 iterations).
constexpr int kBottomMaxCells = 4096;
constexpr int kBottomAutoCells[4] = {0, 0, 1024, 4096};
constexpr double kBottomMaxBytes = 1.0e9;
int MacGpu::choose_bottom_level(std::string *why) const {
  const int nd = tt_.ndim;
  auto usable = [&](int B, int max_cells) {
    const DevTower &tw = towers_[B];
    const int n = (int)tw.blocks.size();
    if (n == 0 || tw.end[B] - tw.begin[B] != n) return false;
    std::vector<int> pos(tt_.num_blocks, -1);
    for (int p = 0; p < n; p++) pos[tw.blocks[p]] = p;
    std::vector<int> comp(n, -1);
    double bytes = 0.0;
    for (int p0 = 0; p0 < n; p0++) {
      if (comp[p0] >= 0) continue;
      std::vector<int> stack{p0};
      comp[p0] = p0;
      long cells = 0;
      while (!stack.empty()) {
        const int p = stack.back();
        stack.pop_back();
        cells += ncell_;
        for (int f = 0; f < 2 * nd; f++) {
          const int nbr = tt_.neighbor[tw.blocks[p] * 6 + f];
          if (nbr <= kPhysBndry) continue;
          if (nbr < 0 || pos[nbr] < 0) return false;  // coarse/fine face
          if (comp[pos[nbr]] < 0) {
            comp[pos[nbr]] = p0;
            stack.push_back(pos[nbr]);
          }
        }
      }
      if (B > 1 && cells > max_cells) return false;
      bytes += 8.0 * (double)cells * (double)cells;
    }
    return bytes <= (B > 1 ? kBottomMaxBytes : 4.0e9);
  };
  if (prm_.bottom_level >= 1) {
    const int B = std::min(prm_.bottom_level, std::max(1, finest_ - 1));
    if (!usable(B, kBottomMaxCells)) {
      *why = "bottom_level " + std::to_string(B) + ": tower is not one uniform level small enough for the dense solve";
      return -1;
    }
    return B;
  }
  int best = 1;
  for (int B = 2; B < finest_ && usable(B, kBottomAutoCells[nd]); B++) best = B;
  return best;
}

// Dense FP64 inverse of the bottom level's operator (the bottom tower is
// one uniform level: faces FINE_FINE or FINE_BC only), one per connected
// component, rows in tower order within a component, cells in block order.
void MacGpu::build_bottom() {
  const int nd = tt_.ndim, nb = tt_.nb;
  std::string why;
  const int LB = choose_bottom_level(&why);
  if (LB < 1) {
    fail(why);
    return;
  }
  bot_level_ = LB;
  bot_param_ = prm_.bottom_level;
  const std::vector<int> &B1 = towers_[LB].blocks;
  // the bottom blocks' coefficients (compact, in B1 order), assembled on the host
  std::vector<double> vfB, bB[3], aB[3];
  pull_block_coefs(B1, vfB, bB, aB);
  const int nblk1 = (int)B1.size();
  n_bot_ = nblk1 * ncell_;
  if (n_bot_ == 0) return;
  std::vector<int> pos1(tt_.num_blocks, -1);
  for (int p = 0; p < nblk1; p++) pos1[B1[p]] = p;
  // connected components of the level-1 blocks; within a component the
  // blocks keep their tower order
  std::vector<int> bcomp(nblk1, -1);
  std::vector<std::vector<int>> comps;
  for (int p0 = 0; p0 < nblk1; p0++) {
    if (bcomp[p0] >= 0) continue;
    const int c = (int)comps.size();
    comps.emplace_back();
    std::vector<int> stack{p0};
    bcomp[p0] = c;
    while (!stack.empty()) {
      const int p = stack.back();
      stack.pop_back();
      comps[c].push_back(p);
      for (int f = 0; f < 2 * nd; f++) {
        const int nbr = tt_.neighbor[B1[p] * 6 + f];
        if (nbr < 0) continue;
        if (pos1[nbr] < 0) {
          fail("bottom-level neighbour outside the bottom tower");
          return;
        }
        if (bcomp[pos1[nbr]] < 0) {
          bcomp[pos1[nbr]] = c;
          stack.push_back(pos1[nbr]);
        }
      }
    }
    std::sort(comps[c].begin(), comps[c].end());
  }
  const int nc = (int)comps.size();
  std::vector<int> order, comp_row0(nc), comp_n(nc), rowpos(tt_.num_blocks, -1);
  std::vector<long long> comp_off(nc);
  long long tot = 0;
  int max_n = 0;
  for (int c = 0; c < nc; c++) {
    comp_row0[c] = (int)order.size() * ncell_;
    comp_n[c] = (int)comps[c].size() * ncell_;
    comp_off[c] = tot;
    tot += (long long)comp_n[c] * comp_n[c];
    max_n = std::max(max_n, comp_n[c]);
    for (int p : comps[c]) {
      rowpos[B1[p]] = (int)order.size();
      order.push_back(B1[p]);
    }
  }
  if ((double)tot * 8 > 4.0e9 || (double)max_n * 8 > 200.0 * 1024) {
    fail("bottom-level problem too large for the dense bottom solve");
    return;
  }
  std::vector<double> A((size_t)tot, 0.0);
  std::vector<int> dir_touch(n_bot_, 0), rcomp(n_bot_);
  std::vector<std::vector<int>> adj(n_bot_);  // global rows, face coefficient > 0
  auto fidx = [&](int d, const int ijk[3], int s) {
    int f[3] = {ijk[0], ijk[1], ijk[2]};
    f[d] += s;
    const int e0 = nb + (d == 0), e1 = nb + (d == 1);
    return f[0] + e0 * (f[1] + e1 * f[2]);
  };
  for (int c = 0; c < nc; c++) {
    const int m = comp_n[c], r0 = comp_row0[c];
    double *Ac = A.data() + comp_off[c];
    for (int p : comps[c]) {
      const int b = B1[p];
      const double dv = geom_[b * 8 + 6];
      for (int cc = 0; cc < ncell_; cc++) {
        const int g = rowpos[b] * ncell_ + cc, row = g - r0;
        rcomp[g] = c;
        int ijk[3] = {cc % nb, nd >= 2 ? (cc / nb) % nb : 0, nd == 3 ? cc / (nb * nb) : 0};
        const double vf = vfB[(size_t)pos1[b] * ncell_ + cc];
        if (!(vf > 0)) {
          Ac[(size_t)row * m + row] = 1.0;
          continue;
        }
        double diag = 0.0;
        for (int f = 0; f < 2 * nd; f++) {
          const int d = f >> 1, s = f & 1;
          const bool bnd = s ? ijk[d] == nb - 1 : ijk[d] == 0;
          const int fx = fidx(d, ijk, s);
          double T = beta_ * geom_[b * 8 + 3 + d] / geom_[b * 8 + d];
          T = T * bB[d][(size_t)pos1[b] * nfb_ + fx];
          T = T * aB[d][(size_t)pos1[b] * nfb_ + fx];
          int ncol = -1;
          if (!bnd) {
            int q[3] = {ijk[0], ijk[1], ijk[2]};
            q[d] += s ? 1 : -1;
            ncol = rowpos[b] * ncell_ + (q[0] + nb * (q[1] + nb * q[2]));
          } else {
            const int nbr = tt_.neighbor[b * 6 + f];
            if (nbr >= 0) {
              int q[3] = {ijk[0], ijk[1], ijk[2]};
              q[d] = s ? 0 : nb - 1;
              ncol = rowpos[nbr] * ncell_ + (q[0] + nb * (q[1] + nb * q[2]));
            } else {
              const int bct = bc_type_[b * 6 + f];
              if (bct == kBCNeumann) T = 0.0;
              else {
                T = 2.0 * T;
                if (T > 0) dir_touch[g] = 1;
              }
            }
          }
          diag += T;
          if (ncol >= 0) {
            Ac[(size_t)row * m + (ncol - r0)] -= T / dv / vf;
            if (T > 0) adj[g].push_back(ncol);
          }
        }
        Ac[(size_t)row * m + row] += diag / dv / vf;
      }
    }
  }
  // pin one cell of every fluid component that has no Dirichlet face
  std::vector<int> seen(n_bot_, -1), pins;
  for (int r0 = 0; r0 < n_bot_; r0++) {
    const int b = order[r0 / ncell_];
    if (seen[r0] >= 0 || !(vfB[(size_t)pos1[b] * ncell_ + r0 % ncell_] > 0)) continue;
    std::vector<int> stack{r0};
    seen[r0] = r0;
    bool dirichlet = false;
    while (!stack.empty()) {
      const int r = stack.back();
      stack.pop_back();
      dirichlet |= dir_touch[r] != 0;
      for (int q : adj[r])
        if (seen[q] < 0) {
          seen[q] = r0;
          stack.push_back(q);
        }
    }
    if (!dirichlet) {
      const int c = rcomp[r0], m = comp_n[c], lr = r0 - comp_row0[c];
      double *Ac = A.data() + comp_off[c];
      for (int j = 0; j < m; j++) Ac[(size_t)lr * m + j] = 0.0;
      Ac[(size_t)lr * m + lr] = 1.0;
      pins.push_back(r0);
    }
  }
  // Rows per CTA: one per warp while those CTAs run at the same time (152 SMs,
  // 8 each) or rows are long, else four, as a row of 256 cells (one load per
  // lane) costs less than starting the CTA and gathering the component's
  // residual: 256 components of 256 cells, FP16 rows, 53.7 -> 27.2 us; 32 of
  // 1024 cells, FP64 rows, would take 113 instead of 104.
  std::vector<int> tile_comp, tile_row0;
  long nrows = 0;
  int longest = 0;
  for (int c = 0; c < nc; c++) nrows += comp_n[c], longest = std::max(longest, comp_n[c]);
  const int tile_rows =
      longest <= 512 && nrows > (long)152 * 8 * kBottomWarps ? 4 * kBottomWarps : kBottomWarps;
  for (int c = 0; c < nc; c++)
    for (int r = 0; r < comp_n[c]; r += tile_rows) {
      tile_comp.push_back(c);
      tile_row0.push_back(r);
    }
  // The structure (level, components, row order) depends on the tree
  // alone: after a coefficient change the device arrays are rewritten in
  // place, so that a captured solve graph, which holds their addresses,
  // stays valid.
  const bool reuse = d_binv_ && bot_built_level_ == LB && bot_built_tot_ == tot && bot_built_half_ == prm_.bottom_half;
  if (!reuse) bottom_free();
  auto up = [&](auto *&dptr, const auto &v) {
    using E = typename std::remove_reference<decltype(v[0])>::type;
    if (dev_malloc(&dptr, std::max<size_t>(v.size(), 1) * sizeof(E)) != cudaSuccess) {
      fail("out of device memory (bottom solve)");
      return;
    }
    if (!v.empty()) CK_(cudaMemcpyAsync(dptr, v.data(), v.size() * sizeof(E), cudaMemcpyHostToDevice, stream_));
  };
  if (reuse) {
    CK_(cudaMemcpyAsync(d_binv_, A.data(), A.size() * sizeof(double), cudaMemcpyHostToDevice, stream_));
  } else {
    up(d_binv_, A);
    up(d_bot_blocks_, order);
    up(d_comp_row0_, comp_row0);
    up(d_comp_n_, comp_n);
    up(d_comp_off_, comp_off);
    up(d_tile_comp_, tile_comp);
    up(d_tile_row0_, tile_row0);
  }
  if (!err_.empty()) return;
  bot_built_level_ = LB;
  bot_built_tot_ = tot;
  bot_built_half_ = prm_.bottom_half;
  // Gauss-Jordan, batched over the components of equal order
  std::vector<int> sizes(comp_n);
  std::sort(sizes.begin(), sizes.end());
  sizes.erase(std::unique(sizes.begin(), sizes.end()), sizes.end());
  for (int m : sizes) {
    std::vector<long long> offs;
    for (int c = 0; c < nc; c++)
      if (comp_n[c] == m) offs.push_back(comp_off[c]);
    const int nmat = (int)offs.size();
    const long long mm = (long long)m * m;
    // the matrices after every other step: all at once, or as many as there is
    // memory for
    char *mem = nullptr;
    int per = nmat;
    // (halves where both copies of a half fit the L2, 129 MB, and both of the
    // group do not: 8 matrices of order 1024 take 38 ms together and 34 as halves)
    const long long copy = nmat * mm * 8, l2 = 100ll << 20;
    if (nmat > 1 && copy <= l2 && 2 * copy > l2) per = (nmat + 1) / 2;
    while (per > 1 && !optional_malloc(&mem, (size_t)per * mm * sizeof(double))) per = (per + 1) / 2;
    if (!mem) CK_(dev_malloc(&mem, (size_t)mm * sizeof(double)));
    double *const other = reinterpret_cast<double *>(mem);
    for (int q = 0; q < nmat; q++) offs.push_back(q % per * mm);
    long long *d_offs = nullptr;
    double *ipiv = nullptr;
    CK_(dev_malloc(&d_offs, offs.size() * sizeof(long long)));
    CK_(dev_malloc(&ipiv, (size_t)per * m * sizeof(double)));
    CK_(cudaMemcpyAsync(d_offs, offs.data(), offs.size() * sizeof(long long), cudaMemcpyHostToDevice, stream_));
    for (int q = 0; q < nmat; q += per) {
      const int n = std::min(per, nmat - q), grid = (int)std::min<long>((long)n * m, 152 * 16);
      const long long *at = d_offs + q, *at2 = d_offs + nmat + q;
      k_gj_first<<<(n + kTPB - 1) / kTPB, kTPB, 0, stream_>>>(m, n, at, d_binv_, ipiv);
      // (the order is even, as the blocks' sides are: the last step ends in d_binv_)
      for (int k = 0; k < m; k += 2) {
        k_gj_step<<<grid, kTPB, 0, stream_>>>(m, k, n, at, d_binv_, at2, other, ipiv);
        k_gj_step<<<grid, kTPB, 0, stream_>>>(m, k + 1, n, at2, other, at, d_binv_, ipiv);
      }
    }
    CK_(cudaGetLastError());
    CK_(cudaStreamSynchronize(stream_));
    dev_free(d_offs);
    dev_free(other);
    dev_free(ipiv);
  }
  for (int r0 : pins) {
    const int c = rcomp[r0];
    k_zero_col<<<(comp_n[c] + kTPB - 1) / kTPB, kTPB, 0, stream_>>>(comp_off[c], comp_n[c], r0 - comp_row0[c], d_binv_);
  }
  // an FP32 (or FP16) copy for the FP32 V-cycle: the product is large when
  // the bottom is above level 1 (up to kBottomMaxCells^2 per component) or
  // when a forest has one component per problem (the batch workload: 584 MB
  // of FP64 inverse per product), and FP64 multiply-adds run at 1/64 of the
  // FP32 rate here
  bot_half_ = prm_.bottom_half;
  // the FP16 product reads rows in 16-byte pieces: every row must start on
  // a 16-byte boundary (component orders that are multiples of 8)
  bool rows16 = true;
  for (int c = 0; c < nc; c++) rows16 = rows16 && comp_n[c] % 8 == 0 && comp_off[c] % 8 == 0;
  if (prm_.bottom_half && rows16) {
    // FP16 rows with one scale each: half the bytes of the FP32 copy
    std::vector<long long> row_off(n_bot_);
    std::vector<int> row_m(n_bot_);
    for (int g = 0; g < n_bot_; g++) {
      const int c = rcomp[g];
      row_off[g] = comp_off[c] + (long long)(g - comp_row0[c]) * comp_n[c];
      row_m[g] = comp_n[c];
    }
    long long *d_ro = nullptr;
    int *d_rm = nullptr;
    if ((!d_binv16_ && dev_malloc(&d_binv16_, (size_t)tot * sizeof(unsigned short)) != cudaSuccess) ||
        (!d_rscale_ && dev_malloc(&d_rscale_, (size_t)n_bot_ * sizeof(float)) != cudaSuccess) ||
        dev_malloc(&d_ro, (size_t)n_bot_ * sizeof(long long)) != cudaSuccess ||
        dev_malloc(&d_rm, (size_t)n_bot_ * sizeof(int)) != cudaSuccess) {
      if (d_ro) dev_free(d_ro);
      fail("out of device memory (bottom solve)");
      return;
    }
    CK_(cudaMemcpyAsync(d_ro, row_off.data(), row_off.size() * sizeof(long long), cudaMemcpyHostToDevice, stream_));
    CK_(cudaMemcpyAsync(d_rm, row_m.data(), row_m.size() * sizeof(int), cudaMemcpyHostToDevice, stream_));
    k_half_rows<<<std::min(n_bot_, 152 * 16), kTPB, 0, stream_>>>(n_bot_, d_ro, d_rm, d_binv_, d_binv16_, d_rscale_);
    CK_(cudaStreamSynchronize(stream_));
    dev_free(d_ro);
    dev_free(d_rm);
  } else {
    if (!d_binv32_ && dev_malloc(&d_binv32_, (size_t)tot * sizeof(float)) != cudaSuccess) {
      d_binv32_ = nullptr;
      fail("out of device memory (bottom solve)");
      return;
    }
    k_narrow<<<ew_grid(tot), kTPB, 0, stream_>>>(tot, d_binv_, d_binv32_);
  }
  CK_(cudaStreamSynchronize(stream_));
  bot_ = BottomDev{d_binv_, d_bot_blocks_, d_comp_row0_, d_comp_n_, d_comp_off_, d_tile_comp_, d_tile_row0_,
                   (int)tile_comp.size(), ncell_, max_n};
  bot_.binv32 = d_binv32_;
  bot_.binv16 = d_binv16_;
  bot_.rscale = d_rscale_;
  bot_.tile_rows = tile_rows;
  n_pins_ = (int)pins.size();
  n_bot_comp_ = nc;
  bottom_ready_ = true;
}

void MacGpu::bottom_free() {
  for (void *p : {(void *)d_binv16_, (void *)d_rscale_, (void *)d_binv32_, (void *)d_binv_, (void *)d_bot_blocks_, (void *)d_comp_row0_, (void *)d_comp_n_,
                  (void *)d_comp_off_, (void *)d_tile_comp_, (void *)d_tile_row0_})
    if (p) dev_free(p);
  d_binv_ = nullptr;
  d_binv32_ = nullptr;
  d_binv16_ = nullptr;
  d_rscale_ = nullptr;
  d_bot_blocks_ = d_comp_row0_ = d_comp_n_ = d_tile_comp_ = d_tile_row0_ = nullptr;
  d_comp_off_ = nullptr;
  bot_ = BottomDev{};
  bot_built_level_ = -1;
  bot_built_tot_ = -1;
}

// one V-cycle with zero initial guess in precision T; the input residual
// (masked rhs) is already in `resid`, the result goes to `out` (FP64)
template <typename T>
void MacGpu::vcycle_device(int L, T *resid, T *corr, const Coef<T> &c, double *out) {
  const int *guard = &d_st_->done;
  const int LB = bot_level_;
  for (int l = L; l >= LB + 1; l--) {
    if (l - 1 >= tt_.max_level || levels_[l - 1].n == 0 || levels_[l].n == 0) continue;
    launch_restrict<T>(topo_, c, nonleaf_list(l - 1), resid, guard, stream_, prm_.pdl != 0);
  }
  // Block-hybrid passes read one correction vector and write the other.  A
  // tower holds every block that the next one reads (its leaves and the
  // parents of the next level), so the vectors simply change places from
  // tower to tower, and the bottom starts in the one from which the last pass
  // of the finest tower ends in corr.
  T *main = corr, *other = prm_.smoother == 1 ? corr_alt<T>() : corr;
  if (prm_.smoother == 1) {
    int passes = 0;
    for (int l = LB + 1; l <= L; l++) passes += levels_[l].n > 0 ? prm_.n_post : 0;
    if (passes & 1) std::swap(main, other);
  }
  bottom_launch<T>(resid, main);
  for (int l = LB + 1; l <= L; l++) {
    if (levels_[l].n == 0) continue;
    if (prm_.smoother == 1) {
      // over every sublevel of tower l at once; the first pass prolongs
      const BlockList TL = smooth_list(l);
      const bool fused = prm_.n_post > 0 && bhgs_prolongs<T>(topo_, c, TL) && sublevel_list(l, l).n == levels_[l].n;
      if (!fused) launch_prolong<T>(topo_, c, level_list(l), main, guard, stream_, prm_.pdl != 0);
      for (int s = 0; s < prm_.n_post; s++) {
        launch_bhgs<T>(topo_, c, TL, prm_.inner_sweeps, main, other, resid, guard, stream_, prm_.pdl != 0,
                       fused && s == 0 ? l : 0);
        std::swap(main, other);
      }
      continue;
    }
    // the level's own sublevel of tower l holds every block of the level, so
    // the prolongation and the red sweep that follows it can be one launch
    const BlockList top = sublevel_list(l, l);
    const bool fused = prm_.fuse_prolong && prm_.n_post > 0 && top.n == levels_[l].n;
    if constexpr (sizeof(T) == 4) {
      // the whole tower in one launch, where its blocks fit the device
      if (fused && solve_lists_ && flow_fits(l)) {
        // (a moving body may change the number of active blocks up to the
        // capacity without another capture)
        const int grid = std::min(towers_[l].par.n, flow_capacity_);
        CK(launch_flow(topo_, c, parity_list(l, 0, false), parity_list(l, 1, false), l, prm_.n_post, grid, corr, resid,
                       guard, d_flow_words_, d_flow_epoch_, reduced() ? d_active_ : nullptr, stream_));
        continue;
      }
    }
    // with the parity order, the red sweep of the rest of group 0 (leaf
    // sublevels l-2, l-4, ...) rides in the same launch
    const BlockList rest0 = prm_.sublevel_order == 1 ? parity_list(l, 0, true) : BlockList{nullptr, nullptr, 0};
    if (fused)
      launch_prolong_red<T>(topo_, c, top, corr, resid, guard, stream_, prm_.pdl != 0, rest0, prm_.prolong_form);
    else
      launch_prolong<T>(topo_, c, level_list(l), corr, guard, stream_, prm_.pdl != 0);
    for (int s = 0; s < prm_.n_post; s++) {
      if (prm_.sublevel_order == 1) {
        // one launch per colour and level parity: within a launch no cell
        // reads another that the launch writes (same-level neighbours have
        // the other colour, coarse/fine neighbours the other parity)
        for (int rb = 0; rb < 2; rb++)
          for (int g = 0; g < 2; g++) {
            if (fused && s == 0 && rb == 0 && g == 0) continue;  // done by the fused launch
            const BlockList gl = parity_list(l, g, false);
            if (gl.n > 0) launch_rbgs<T>(topo_, c, gl, rb, corr, resid, guard, stream_, prm_.pdl != 0, rbgs_var<T>());
          }
        continue;
      }
      for (int ll = l; ll >= 1; ll--) {
        BlockList sl = sublevel_list(l, ll);
        if (sl.n == 0) break;
        for (int rb = 0; rb < 2; rb++) {
          if (fused && s == 0 && ll == l && rb == 0) continue;
          launch_rbgs<T>(topo_, c, sl, rb, corr, resid, guard, stream_, prm_.pdl != 0, rbgs_var<T>());
        }
      }
    }
  }
  if (out) vc_out_launch<T>(tower_list(L), corr, out);
}

// tower l can be smoothed by launch_flow
int MacGpu::flow_entries(int l) const {
  return reduced() && l < (int)n_act_par_.size() ? n_act_par_[l] : towers_[l].par.n;
}
bool MacGpu::flow_fits(int l) const {
  return d_flow_words_ && prm_.sublevel_order == 1 && prm_.prolong_form == 1 &&
         prm_.n_post < (int)kFlowTags - 1 && flow_entries(l) > 0 && flow_entries(l) <= flow_capacity_;
}
unsigned MacGpu::flow_mask() const {
  unsigned m = 0;
  if (prm_.precision == 1 && prm_.smoother == 0 && prm_.vcycle_kernel == 0)
    for (int l = 2; l <= finest_ && l < 32; l++) m |= flow_fits(l) ? 1u << l : 0u;
  return m;
}

// the exchange buffers of launch_flow, if any tower fits it (where they cannot be
// had, towers keep their separate launches)
void MacGpu::ensure_flow() {
  if (d_flow_words_) return;
  if (flow_capacity_ < 0) flow_capacity_ = flow_capacity(topo_);
  bool any = false;
  for (int l = 2; l <= finest_; l++) any = any || (flow_entries(l) > 0 && flow_entries(l) <= flow_capacity_);
  if (!any) return;
  const size_t n = flow_words(topo_) * sizeof(unsigned long long) + 2 * sizeof(unsigned);
  char *mem = nullptr;
  if (!optional_malloc(&mem, n)) return;
  CK(cudaMemsetAsync(mem, 0, n, stream_));
  d_flow_words_ = reinterpret_cast<unsigned long long *>(mem);
  d_flow_epoch_ = reinterpret_cast<unsigned *>(d_flow_words_ + flow_words(topo_));
}

// V-cycle result on the tower, widened to FP64: out = 0 + corr
template <typename T>
void MacGpu::vc_out_launch(const BlockList &TL, T *corr, double *out) {
  launch_k(prm_.pdl != 0, k_vc_out<T>, ew_grid((long)TL.n * ncell_), kTPB, 0, stream_, TL, ncell_,
           (const FState *)d_st_, (const T *)corr, out);
}
template void MacGpu::vc_out_launch<float>(const BlockList &, float *, double *);
template void MacGpu::vc_out_launch<double>(const BlockList &, double *, double *);

// dense bottom solve of the level-1 problem: corr = Binv * resid
template <typename T>
void MacGpu::bottom_launch(T *resid, T *corr) {
  if (bot_.ntiles == 0) return;
  const size_t smem = (size_t)bot_.max_n * sizeof(double);
  if (smem > 48 * 1024)
    ensure_max_smem((const void *)k_bottom_gemv<T>, (int)smem);
  BottomDev bd = bot_;
  if (solve_lists_ && multi()) {
    bd.comp = d_comp_;
    bd.stc = d_stc_;
  }
  launch_k(prm_.pdl != 0, k_bottom_gemv<T>, bot_.ntiles, kTPB, smem, stream_, bd, (const T *)resid, corr,
           (const FState *)d_st_);
}
template void MacGpu::bottom_launch<float>(float *, float *);
template void MacGpu::bottom_launch<double>(double *, double *);

// one preconditioner application: the V-cycle, then (FP32, when enabled and
// trained) the learned block correction, then the widening into out
template <typename T>
void MacGpu::precondition(int L, T *resid, T *corr, const Coef<T> &c, double *out) {
  const bool nn = sizeof(T) == 4 && learned_active();
  double *o = nn ? nullptr : out;
  const bool fused = prm_.smoother == 0 && !(solve_lists_ && multi());
  if (prm_.vcycle_kernel == 2 && fused)
    vcycle_cluster<T>(resid, corr, c, o);
  else if (prm_.vcycle_kernel == 1 && fused)
    vcycle_coop<T>(resid, corr, c, o);
  else
    vcycle_device<T>(L, resid, corr, c, o);
  if (nn) {
    learned_apply(reinterpret_cast<float *>(resid), reinterpret_cast<float *>(corr));
    if (out) vc_out_launch<T>(tower_list(L), corr, out);
  }
}

// FP32 V-cycle output read in place by the BiCGSTAB kernels, widened exactly
// on the integer pipe where they read it, or widened once into FP64 phat /
// shat.  params.vcycle_out 0 (auto): in place in 2D and on 3D towers of at
// most 2M cells, where it saves two launches per iteration and the operator forms
// its differences on the FP32 pipe (256 problems, 2D, 29 M cells: 35.8 ms in place,
// 41.9 widened, 44.5 with the double-float operator), and on larger 3D towers
// of which at least half the blocks have one face coefficient and whose blocks'
// side is a multiple of four, whose operator is formed on the FP32 pipe from the
// FP32 values (k_op_rows; 15.9 M cells of 16^3 blocks: 16.2 in place, 20.0
// widened).  Other large 3D towers widen, since the general 3D operator reads seven
// cells and widens each on the integer pipe: no difference on 3.9 M cells of 10^3
// blocks (10.9 ms).  (16^3 blocks of variable B, which this rule widens too, take
// 22.7 ms widened and 20.0 in place: the rows form gains there as well.)  1 = in place with the operator in double-float, 2 = always
// widened, 3 = always in place.
constexpr long kDirectF32Cells = 1l << 21;
bool MacGpu::vcycle_in_place() const {
  if (learned_active() || prm_.precision != 1) return false;
  if (prm_.vcycle_out != 0) return prm_.vcycle_out != 2;
  const DevList &top = towers_[finest_].all;
  return tt_.ndim == 2 || (long)top.n * ncell_ <= kDirectF32Cells ||
         (tt_.nb % 4 == 0 && !multi() && act_version_ == coef_version_ && 2l * n_iso_ >= n_act_);
}
template <typename T>
void MacGpu::iteration_device(T *resid, T *corr, const Coef<T> &c) {
  if constexpr (sizeof(T) == 4) {
    if (vcycle_in_place()) {
      iteration_body<T, float>(resid, corr, c, corr, corr, nullptr, nullptr);
      return;
    }
    iteration_body<T, double>(resid, corr, c, vec_[kPHAT], vec_[kSHAT], vec_[kPHAT], vec_[kSHAT]);
  } else {
    iteration_body<T, double>(resid, corr, c, corr, corr, nullptr, nullptr);
  }
}

// the operator by rows on the blocks of the finest tower that the solve walks
template <int M>
void MacGpu::launch_op_rows(const float *x, double *y, const double *w) {
  const bool mp = multi();
  const BlockList TL =
      mp ? BlockList{tlc_.blocks, tlc_.ftypes, tlc_.n, nullptr, nullptr, tlc_.hx} : tower_list(finest_);
  // threads at work per CTA: 32 .. 256, enough for about two CTAs per SM
  const long cells = (long)TL.n * ncell_, groups = std::max<long>(1, cells / 4), cap = red_grid(cells);
  const int per = (int)std::min<long>(kTPB, std::max<long>(32, (groups / (152 * 2) + 31) / 32 * 32));
  const int g = mp ? nchunks_ : (int)std::min<long>(std::max<long>(cap, 152 * 2), (groups + per - 1) / per);
  auto rows = [&](auto kern) {
    launch_k(prm_.pdl != 0, kern, g, kTPB, 0, stream_, topo_, cd64_, TL, chunks(), x, y, w, (const double *)d_opP_,
             (const double *)d_opS_, mp ? d_stc_ : d_st_, mp ? d_cpart_ : d_part_, mp ? d_ccnt_ : d_cnt_,
             (const double *)d_iso_, per);
  };
  if (tt_.ndim == 2)
    mp ? rows(k_op_rows<2, M, true>) : rows(k_op_rows<2, M, false>);
  else
    mp ? rows(k_op_rows<3, M, true>) : rows(k_op_rows<3, M, false>);
}

// One BiCGSTAB iteration.  The V-cycle's output PH (the first
// preconditioner application) is consumed by the operator and the x update
// before the second application overwrites it (SH); out_p / out_s, when
// given, receive the output widened to FP64 (PH / SH point there).
template <typename T, typename TO>
void MacGpu::iteration_body(T *resid, T *corr, const Coef<T> &c, const TO *PH, const TO *SH, double *out_p,
                            double *out_s) {
  const int L = finest_;
  const bool mp = multi();
  // the BiCGSTAB kernels: the finest tower (problem by problem and one CTA
  // per chunk with one state per problem, else grid-stride with one state)
  const BlockList TL = mp ? BlockList{tlc_.blocks, tlc_.ftypes, tlc_.n, nullptr, nullptr, tlc_.hx} : tower_list(L);
  const long w = (long)TL.n * ncell_;
  const Chunks ch = chunks();
  FState *ST = mp ? d_stc_ : d_st_;
  double *PART = mp ? d_cpart_ : d_part_;
  unsigned *CNT = mp ? d_ccnt_ : d_cnt_;
  const int gr = mp ? nchunks_ : red_grid(w), ge = mp ? nchunks_ : ew_grid(w);
  double *R = vec_[kR], *RHAT = vec_[kRHAT], *P = vec_[kP], *S = vec_[kS];
  double *V = vec_[kV], *Tt = vec_[kT], *X = vec_[kX];
  const bool pdl = prm_.pdl != 0;
  const double *OP = d_opP_, *OS = d_opS_;
  const float2 *OP2 = d_opP2_, *OS2 = d_opS2_, *U2 = d_uni2_;
  // params.vcycle_out 1: the operator of the FP32 V-cycle's output in double-float
  const bool dfop = prm_.vcycle_out == 1;
  auto op = [&](auto mode, const auto *x, double *y, const double *wv, double *y2) {
    constexpr int M = decltype(mode)::value;
    using TX = std::remove_const_t<std::remove_pointer_t<decltype(x)>>;
    auto go = [&](auto df) {
      constexpr bool D = decltype(df)::value;
      if (tt_.ndim == 2) {
        if (mp)
          launch_k(pdl, k_op_red<2, M, TX, true, D>, gr, kTPB, 0, stream_, topo_, cd64_, TL, ch, x, y, wv, OP, OS, ST,
                   PART, CNT, y2, OP2, OS2, U2);
        else
          launch_k(pdl, k_op_red<2, M, TX, false, D>, gr, kTPB, 0, stream_, topo_, cd64_, TL, ch, x, y, wv, OP, OS,
                   ST, PART, CNT, y2, OP2, OS2, U2);
      } else {
        if (mp)
          launch_k(pdl, k_op_red<3, M, TX, true, D>, gr, kTPB, 0, stream_, topo_, cd64_, TL, ch, x, y, wv, OP, OS, ST,
                   PART, CNT, y2, OP2, OS2, U2);
        else
          launch_k(pdl, k_op_red<3, M, TX, false, D>, gr, kTPB, 0, stream_, topo_, cd64_, TL, ch, x, y, wv, OP, OS,
                   ST, PART, CNT, y2, OP2, OS2, U2);
      }
    };
    if constexpr (sizeof(TX) == 4 && M < 2) {
      if (!dfop && tt_.nb % 4 == 0) {
        launch_op_rows<M>(x, y, wv);
        return;
      }
      if (dfop) {
        go(std::true_type{});
        return;
      }
    }
    go(std::false_type{});
  };
  if (mp)
    launch_k(pdl, k_pupdate<T, true>, ge, kTPB, 0, stream_, TL, ncell_, ch, ST, (const double *)R, P,
             (const double *)V, (const double *)d_vf_, resid);
  else
    launch_k(pdl, k_pupdate<T, false>, ge, kTPB, 0, stream_, TL, ncell_, ch, ST, (const double *)R, P,
             (const double *)V, (const double *)d_vf_, resid);
  precondition<T>(L, resid, corr, c, out_p);
  op(std::integral_constant<int, 0>{}, PH, V, (const double *)RHAT, (double *)nullptr);
  if (mp)
    launch_k(pdl, k_supdate<T, TO, true>, gr, kTPB, 0, stream_, TL, ncell_, ch, ST, (const double *)R,
             (const double *)V, S, X, PH, (const double *)d_vf_, resid, PART, CNT);
  else
    launch_k(pdl, k_supdate<T, TO, false>, gr, kTPB, 0, stream_, TL, ncell_, ch, ST, (const double *)R,
             (const double *)V, S, X, PH, (const double *)d_vf_, resid, PART, CNT);
  precondition<T>(L, resid, corr, c, out_s);
  op(std::integral_constant<int, 1>{}, SH, Tt, (const double *)S, (double *)nullptr);
  if (mp)
    launch_k(pdl, k_rupdate<TO, true>, gr, kTPB, 0, stream_, TL, ncell_, ch, ST, X, SH, R, (const double *)S,
             (const double *)Tt, (const double *)RHAT, PART, CNT);
  else
    launch_k(pdl, k_rupdate<TO, false>, gr, kTPB, 0, stream_, TL, ncell_, ch, ST, X, SH, R, (const double *)S,
             (const double *)Tt, (const double *)RHAT, PART, CNT);
  // verified convergence (both kernels return at once unless a pass converged)
  double *X0 = vec_[kX0];
  if (mp)
    launch_k(pdl, k_verify_fold<true>, ge, kTPB, 0, stream_, TL, ncell_, ch, (const FState *)ST, X0, X);
  else
    launch_k(pdl, k_verify_fold<false>, ge, kTPB, 0, stream_, TL, ncell_, ch, (const FState *)ST, X0, X);
  op(std::integral_constant<int, 3>{}, (const double *)X0, R, (const double *)vec_[kRHS], RHAT);
}

// the chunk table of the per-problem states (empty with one shared state)
Chunks MacGpu::chunks() const {
  Chunks ch{};
  if (!multi()) return ch;
  ch.comp = d_chunk_;
  ch.beg = d_chunk_ + nchunks_;
  ch.end = d_chunk_ + 2 * nchunks_;
  ch.c0 = d_chunk_ + 3 * nchunks_;
  ch.cn = d_chunk_ + 3 * nchunks_ + ncomp_;
  return ch;
}

void MacGpu::drop_graph() {
  if (graph_exec_) {
    cudaGraphExecDestroy(graph_exec_);
    graph_exec_ = nullptr;
  }
  if (graph_) {
    cudaGraphDestroy(graph_);
    graph_ = nullptr;
  }
}

void MacGpu::capture_loop(int precision) {
  drop_graph();
  CK_(cudaGraphCreate(&graph_, 0));
  cudaGraphConditionalHandle h;
  CK_(cudaGraphConditionalHandleCreate(&h, graph_, 1, cudaGraphCondAssignDefault));
  cudaGraphNodeParams np = {};
  np.type = cudaGraphNodeTypeConditional;
  np.conditional.handle = h;
  np.conditional.type = cudaGraphCondTypeWhile;
  np.conditional.size = 1;
  cudaGraphNode_t node;
  CK_(cudaGraphAddNode(&node, graph_, nullptr, nullptr, 0, &np));
  cudaGraph_t body = np.conditional.phGraph_out[0];
  CK_(cudaStreamBeginCaptureToGraph(stream_, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
  solve_lists_ = true;
  if (precision == 1)
    iteration_device<float>(d_resid32_, d_corr32_, c32_);
  else
    iteration_device<double>(vec_[kRESID], vec_[kCORR], cd64_);
  solve_lists_ = false;
  if (multi())
    launch_k(prm_.pdl != 0, k_set_cond_multi, 1, 256, 0, stream_, h, (const FState *)d_stc_, ncomp_, d_st_,
             (const int *)topo_.err);
  else
    launch_k(prm_.pdl != 0, k_set_cond, 1, 1, 0, stream_, h, (const FState *)d_st_, (const int *)topo_.err);
  cudaGraph_t out = nullptr;
  CK_(cudaStreamEndCapture(stream_, &out));
  // count the kernel nodes of one iteration (reported as launches per step)
  size_t nn = 0;
  CK_(cudaGraphGetNodes(body, nullptr, &nn));
  std::vector<cudaGraphNode_t> nodes(nn);
  if (nn) CK_(cudaGraphGetNodes(body, nodes.data(), &nn));
  kernels_per_iter_ = 0;
  for (auto nd : nodes) {
    cudaGraphNodeType ty;
    if (cudaGraphNodeGetType(nd, &ty) == cudaSuccess && ty == cudaGraphNodeTypeKernel) kernels_per_iter_++;
  }
  CK_(cudaGraphInstantiate(&graph_exec_, graph_, 0));
  graph_prec_ = precision;
  graph_npost_ = prm_.n_post;
  graph_coop_ = prm_.vcycle_kernel;
  graph_pdl_ = prm_.pdl;
  graph_cc_ = prm_.cluster_cells;
  graph_var_ = rbgs_variant_[precision == 1];
  graph_nn_ = (int)learned_active();
  graph_order_ = prm_.sublevel_order;
  graph_smoother_ = prm_.smoother;
  graph_inner_ = prm_.inner_sweeps;
  graph_multi_ = (int)multi();
  graph_uniform_ = prm_.uniform;
  graph_pform_ = prm_.prolong_form;
  graph_vout_ = prm_.vcycle_out;
  graph_omega_ = prm_.relax_omega;
  graph_act_ = (int)reduced();
  graph_direct_ = (int)vcycle_in_place();
  graph_flow_ = flow_mask();
}

// the captured graph was recorded with other parameters than the current ones
bool MacGpu::graph_stale() const {
  return !graph_exec_ || graph_prec_ != prm_.precision || graph_npost_ != prm_.n_post ||
         graph_coop_ != prm_.vcycle_kernel || graph_pdl_ != prm_.pdl || graph_cc_ != prm_.cluster_cells ||
         graph_var_ != rbgs_variant_[prm_.precision == 1] || graph_nn_ != (int)learned_active() ||
         graph_order_ != prm_.sublevel_order || graph_smoother_ != prm_.smoother ||
         graph_inner_ != prm_.inner_sweeps || graph_multi_ != (int)multi() || graph_uniform_ != prm_.uniform ||
         graph_pform_ != prm_.prolong_form || graph_vout_ != prm_.vcycle_out ||
         graph_omega_ != prm_.relax_omega || graph_act_ != (int)reduced() ||
         graph_direct_ != (int)vcycle_in_place() || graph_flow_ != flow_mask();
}

int MacGpu::cg_solve_device(SolveInfo *info) {
  if (prepare_device() != 0) return -1;
  auto t0 = std::chrono::steady_clock::now();
  if (enqueue_solve() != 0) return -1;
  if (solve_state(info) != 0) return -1;
  info->seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  return info->status == 1 ? 1 : 0;
}

// asynchronous solve for benchmarking: everything enqueued on `stream_`,
// no host synchronisation in graph mode (the caller times it with events)
int MacGpu::cg_solve_enqueue() {
  ensure_fast_buffers();
  // coefficients changed since sayaka_mac_prepare: the fast-path data and the
  // graph must be rebuilt first
  if (!err_.empty() || !bottom_ready_ || coef_version_ != fast_coef_version_ || bot_param_ != prm_.bottom_level ||
      bot_half_ != prm_.bottom_half)
    return -1;
  if (prm_.graph && graph_stale())
    return -1;
  if (prm_.vcycle_kernel && (program_npost_ != prm_.n_post || program_order_ != prm_.sublevel_order ||
                             program_bot_ != bot_level_))
    return -1;
  ensure_derived();
  if (!err_.empty()) return -1;
  return enqueue_solve();
}

int MacGpu::enqueue_solve() {
  const int L = finest_;
  const bool mp = multi();
  const BlockList TL = mp ? BlockList{tlc_.blocks, tlc_.ftypes, tlc_.n, nullptr, nullptr, tlc_.hx} : tower_list(L);
  const long w = (long)TL.n * ncell_;
  const Chunks ch = chunks();
  FState *ST = mp ? d_stc_ : d_st_;
  const int gr = mp ? nchunks_ : red_grid(w), ge = mp ? nchunks_ : ew_grid(w);
  FState init{};
  init.tol_rel = prm_.tol_rel;
  init.tol_abs = prm_.tol_abs;
  init.max_iter = prm_.max_iter;
  init.nn_on = learned_active() ? 1 : 0;
  init.nn_best = 1e300;
  *h_st_ = init;
  CKR_(cudaMemcpyAsync(d_st_, h_st_, sizeof(FState), cudaMemcpyHostToDevice, stream_), -1);
  if (mp) {
    for (int c = 0; c < ncomp_; c++) h_stc_[c] = init;
    CKR_(cudaMemcpyAsync(d_stc_, h_stc_, ncomp_ * sizeof(FState), cudaMemcpyHostToDevice, stream_), -1);
  }
  if (reduced()) zero_solid();
  // prologue: x0 = sol, x = 0, r = rhs - A x0, rhat = r, |r0|, rho
  k_pro_copy<<<ew_grid(w), kTPB, 0, stream_>>>(TL, ncell_, vec_[kSOL], vec_[kX0], vec_[kX]);
  double *PART = mp ? d_cpart_ : d_part_;
  unsigned *CNT = mp ? d_ccnt_ : d_cnt_;
  solve_lists_ = true;  // r and rhat are read on the blocks the solve walks
  const BlockList RL = mp ? TL : tower_list(L);
  solve_lists_ = false;
  auto resid = [&](auto kern) {
    kern<<<gr, kTPB, 0, stream_>>>(topo_, cd64_, RL, ch, vec_[kX0], vec_[kR], vec_[kRHS], d_opP_, d_opS_, ST, PART,
                                   CNT, vec_[kRHAT], nullptr, nullptr, nullptr);
  };
  if (tt_.ndim == 2)
    mp ? resid(k_op_red<2, 2, double, true>) : resid(k_op_red<2, 2, double, false>);
  else
    mp ? resid(k_op_red<3, 2, double, true>) : resid(k_op_red<3, 2, double, false>);
  if (mp) k_set_cond_multi<<<1, 256, 0, stream_>>>(0, d_stc_, ncomp_, d_st_, topo_.err);
  if (prm_.max_iter > 0) {
    if (prm_.graph) {
      CKR_(cudaGraphLaunch(graph_exec_, stream_), -1);
    } else {
      // the captured iteration's kernels, launched directly; the host reads
      // the convergence flag after every iteration
      for (int it = 0; it < prm_.max_iter; it++) {
        solve_lists_ = true;
        if (prm_.precision == 1)
          iteration_device<float>(d_resid32_, d_corr32_, c32_);
        else
          iteration_device<double>(vec_[kRESID], vec_[kCORR], cd64_);
        solve_lists_ = false;
        if (mp) k_set_cond_multi<<<1, 256, 0, stream_>>>(0, d_stc_, ncomp_, d_st_, topo_.err);
        if (record_) {  // a collection solve keeps every iterate
          double *cp = nullptr;
          const size_t n = (size_t)tt_.num_blocks * ncell_;
          if (dev_malloc(&cp, n * sizeof(double)) != cudaSuccess) {
            fail("out of device memory (recorded iterates)");
            return -1;
          }
          CKR_(cudaMemcpyAsync(cp, vec_[kX], n * sizeof(double), cudaMemcpyDeviceToDevice, stream_), -1);
          record_->push_back(cp);
        }
        CKR_(cudaMemcpyAsync(h_st_, d_st_, sizeof(FState), cudaMemcpyDeviceToHost, stream_), -1);
        CKR_(cudaMemcpyAsync(h_err_, topo_.err, sizeof(int), cudaMemcpyDeviceToHost, stream_), -1);
        CKR_(cudaStreamSynchronize(stream_), -1);
        if (h_st_->done || *h_err_) break;
      }
    }
  }
  if (mp)
    k_finish<true><<<ge, kTPB, 0, stream_>>>(TL, ncell_, ch, ST, vec_[kX0], vec_[kX], vec_[kSOL]);
  else
    k_finish<false><<<ge, kTPB, 0, stream_>>>(TL, ncell_, ch, ST, vec_[kX0], vec_[kX], vec_[kSOL]);
  last_multi_ = mp;
  return err_.empty() ? 0 : -1;
}

}  // namespace sayaka_gb300

namespace sayaka_gb300 {

// everything a device-resident solve needs, built ahead of the timed region
int MacGpu::prepare_device() {
  ensure_fast_buffers();
  if (!err_.empty()) return -1;
  if (coef_version_ != fast_coef_version_) {
    // Every array of the coefficient set is rewritten in place (stream
    // order keeps it behind any solve in flight), so a captured graph,
    // which holds kernel arguments by value, stays valid -- unless the
    // bottom solve's arrays had to be allocated afresh.
    const BottomDev before = bot_;
    refresh_fp32();
    build_cf();
    build_uniform();
    build_op_factors();
    if (prm_.bottom_refresh || !bottom_ready_ || bot_param_ != prm_.bottom_level || bot_half_ != prm_.bottom_half)
      build_bottom();
    fast_coef_version_ = coef_version_;
    if (!err_.empty()) return -1;
    if (std::memcmp(&before, &bot_, sizeof(BottomDev)) != 0) {
      CKR_(cudaStreamSynchronize(stream_), -1);
      drop_graph();
    }
  } else if (bot_param_ != prm_.bottom_level || bot_half_ != prm_.bottom_half) {  // another bottom asked for
    CKR_(cudaStreamSynchronize(stream_), -1);
    drop_graph();
    build_bottom();
    if (!err_.empty()) return -1;
  }
  bind_uniform();
  choose_active();
  ensure_derived();
  tune_smoother(prm_.precision);
  if (prm_.precision == 1) ensure_flow();
  if (learned_active()) learned_prepare();
  if (!err_.empty()) return -1;
  if (prm_.vcycle_kernel && (program_npost_ != prm_.n_post || program_order_ != prm_.sublevel_order ||
                             program_bot_ != bot_level_))
    build_vcycle_program();
  if (prm_.graph && graph_stale())
    capture_loop(prm_.precision);
  return err_.empty() ? 0 : -1;
}

}  // namespace sayaka_gb300

namespace sayaka_gb300 {

int MacGpu::solve_state(SolveInfo *info) {
  CKR_(cudaMemcpyAsync(h_st_, d_st_, sizeof(FState), cudaMemcpyDeviceToHost, stream_), -1);
  CKR_(cudaStreamSynchronize(stream_), -1);
  if (d_bar_) {
    unsigned w[4];
    CKR_(cudaMemcpy(w, d_bar_, sizeof(w), cudaMemcpyDeviceToHost), -1);
    if (w[2] != 0) {
      cudaMemsetAsync(d_bar_, 0, 4 * sizeof(unsigned), stream_);
      fail("cooperative V-cycle: grid barrier timed out");
      return -1;
    }
  }
  if (rbgs_bulk_error(topo_.err, stream_, true) > 0) {
    fail("device smoother: a bounded wait timed out");
    return -1;
  }
  if (learned_active() && nn_tc_error(true) > 0) {
    fail("learned correction: a tensor-core wait timed out");
    return -1;
  }
  if (last_multi_) {
    // one state per problem: the largest iteration count and initial
    // residual, rnorm / rnorm0 = the largest relative residual; breakdown if
    // any problem broke down, not converged if any did not converge
    CKR_(cudaMemcpy(h_stc_, d_stc_, ncomp_ * sizeof(FState), cudaMemcpyDeviceToHost), -1);
    int its = 0, stat = 0, unconv = 0, nnoff = 0;
    double r0 = 0.0, rel = 0.0;
    for (int c = 0; c < ncomp_; c++) {
      const FState &q = h_stc_[c];
      its = std::max(its, q.trivial ? 0 : q.iter);
      stat |= q.stat;
      unconv |= !(q.conv || q.trivial);
      nnoff |= q.nn_off;
      r0 = std::max(r0, q.rnorm0);
      if (q.rnorm0 > 0) rel = std::max(rel, q.rnorm / q.rnorm0);
      if (q.rnorm != q.rnorm) rel = q.rnorm;
    }
    info->iterations = its;
    info->rnorm0 = r0;
    info->rnorm = rel * r0;
    info->status = stat ? 1 : (unconv ? 2 : (nnoff ? 3 : 0));
    info->seconds = 0;
    return 0;
  }
  const FState &st = *h_st_;
  info->iterations = st.trivial ? 0 : st.iter;
  info->rnorm0 = st.rnorm0;
  info->rnorm = st.rnorm;
  info->status = st.stat ? 1 : ((st.conv || st.trivial) ? (st.nn_off ? 3 : 0) : 2);
  info->seconds = 0;
  return 0;
}

int MacGpu::problem_states(int *iterations, double *rel_resid, int n) {
  if (!last_multi_) return -1;
  CKR_(cudaMemcpy(h_stc_, d_stc_, ncomp_ * sizeof(FState), cudaMemcpyDeviceToHost), -1);
  for (int c = 0; c < ncomp_ && c < n; c++) {
    const FState &q = h_stc_[c];
    if (iterations) iterations[c] = q.trivial ? 0 : q.iter;
    if (rel_resid) rel_resid[c] = q.rnorm0 > 0 ? q.rnorm / q.rnorm0 : 0.0;
  }
  return ncomp_;
}

int MacGpu::uniform_blocks() {
  if (prepare_device() != 0) return -1;
  std::vector<double> u((size_t)tt_.num_blocks * kUni);
  if (u.empty()) return 0;
  CKR_(cudaMemcpyAsync(u.data(), d_uni64_, u.size() * sizeof(double), cudaMemcpyDeviceToHost, stream_), -1);
  CKR_(cudaStreamSynchronize(stream_), -1);
  int n = 0;
  for (int b = 0; b < tt_.num_blocks; b++) n += u[(size_t)b * kUni + 3] != 0.0;
  return n;
}

int MacGpu::tower_size(int L, int sublevel) const {
  if (L < 1 || L > tt_.max_level) return -1;
  const DevTower &t = towers_[L];
  if (sublevel <= 0) return t.all.n;
  if (sublevel > L || t.all.n == 0) return 0;
  return t.end[sublevel] - t.begin[sublevel];
}

int MacGpu::enqueue_kernel(int which, int L) {
  if (L < 1 || L > tt_.max_level || towers_[L].all.n == 0) return -1;
  ensure_fast_buffers();
  bind_uniform();
  if (which == 2) ensure_smooth_factors();
  if (which == 0) {
    launch_apply<double>(topo_, c64_, tower_list(L), vec_[kSOL], vec_[kV], nullptr, nullptr, stream_);
  } else if (which == 1) {
    launch_rbgs<float>(topo_, c32_, sublevel_list(L, L), 0, d_corr32_, d_resid32_, nullptr, stream_, false,
                       rbgs_var<float>());
  } else if (which == 2) {
    launch_rbgs<double>(topo_, cd64_, sublevel_list(L, L), 0, vec_[kCORR], vec_[kRESID], nullptr, stream_, false,
                        rbgs_var<double>());
  } else if (which == 3) {
    if (L != finest_) return -1;
    const BlockList TL = tower_list(L);
    const long w = (long)TL.n * ncell_;
    CKR_(cudaMemsetAsync(d_st_, 0, sizeof(FState), stream_), -1);
    if (tt_.ndim == 2)
      k_op_red<2, 0, double, false><<<red_grid(w), kTPB, 0, stream_>>>(topo_, cd64_, TL, Chunks{}, vec_[kSOL], vec_[kV],
                                                                      vec_[kRHAT], d_opP_, d_opS_, d_st_, d_part_,
                                                                      d_cnt_);
    else
      k_op_red<3, 0, double, false><<<red_grid(w), kTPB, 0, stream_>>>(topo_, cd64_, TL, Chunks{}, vec_[kSOL], vec_[kV],
                                                                      vec_[kRHAT], d_opP_, d_opS_, d_st_, d_part_,
                                                                      d_cnt_);
  } else {
    return -1;
  }
  return err_.empty() ? 0 : -1;
}

// Test hook: the device solve's own FP64 kernels on given compact all-block
// arrays (host pointers), for comparison with the reference arithmetic.
// which 0: out = A in on the finest tower with the solve's operator (per-cell
// factors P, S and FMA, k_op_red); which 1: one smoothing pass of tower L
// (sublevels finest to coarsest, red then black, as mg_smooth_level) with the
// solve's FP64 sweep, launch variant `variant` (-1: the tuned one); in = phi,
// in2 = rhs.  Uses (and clobbers) the handle's work vectors.
int MacGpu::device_kernel_compact(int which, int L, int variant, const double *in, const double *in2, double *out) {
  if (which < 0 || which > 8 || !in || !out || ((which == 1 || which == 2 || which == 7) && !in2)) return 1;
  if ((which == 1 || which == 2 || which == 7) && (L < 1 || L > finest_ || towers_[L].all.n == 0)) return 1;
  if (which == 1 && variant >= kRbgsVariants) return 1;
  if (which == 2 && (variant < 1 || variant > 1024)) return 1;
  if (which == 7 && (variant < 1 || variant > 4 * 1024)) return 1;
  if (which == 4 && (variant < 1 || variant > kFlowPolls || L < 2 || L > finest_)) return 1;
  if (which == 6) {
    deny_optional_ = variant != 0;
    return 0;
  }
  if (prepare_device() != 0) return 2;
  ensure_smooth_factors();
  if (which == 4) {
    // the one-launch smoothing of tower L without the blocks of its second
    // parity group: no one writes the words that the first group waits for
    // across coarse/fine faces
    const int m = L < (int)towers_.size() && flow_fits(L) ? parity_list(L, 0, false).n : 0;
    if (m == 0 || m > flow_capacity_) return 1;
    CKR_(cudaMemsetAsync(d_st_, 0, sizeof(FState), stream_), 2);
    CKR_(launch_flow(topo_, c32_, parity_list(L, 0, false), BlockList{nullptr, nullptr, 0}, L, prm_.n_post, m,
                     d_corr32_, d_resid32_, &d_st_->done, d_flow_words_, d_flow_epoch_, nullptr, stream_, variant),
         2);
  } else if (which == 5) {  // as a wait that ran out leaves the solver's error word
    const int one = 1;
    CKR_(cudaMemcpyAsync(topo_.err, &one, sizeof(int), cudaMemcpyHostToDevice, stream_), 2);
    CKR_(cudaStreamSynchronize(stream_), 2);
    return 0;
  }
  const size_t n = (size_t)tt_.num_blocks * ncell_;
  if (which == 0) {
    const BlockList TL = tower_list(finest_);
    const long w = (long)TL.n * ncell_;
    CKR_(cudaMemcpyAsync(vec_[kTMP], in, n * sizeof(double), cudaMemcpyHostToDevice, stream_), 2);
    CKR_(cudaMemsetAsync(vec_[kV], 0, n * sizeof(double), stream_), 2);
    CKR_(cudaMemsetAsync(vec_[kRHAT], 0, n * sizeof(double), stream_), 2);
    CKR_(cudaMemsetAsync(d_st_, 0, sizeof(FState), stream_), 2);
    if (tt_.ndim == 2)
      k_op_red<2, 0, double, false><<<red_grid(w), kTPB, 0, stream_>>>(topo_, cd64_, TL, Chunks{}, vec_[kTMP],
                                                                      vec_[kV], vec_[kRHAT], d_opP_, d_opS_, d_st_,
                                                                      d_part_, d_cnt_);
    else
      k_op_red<3, 0, double, false><<<red_grid(w), kTPB, 0, stream_>>>(topo_, cd64_, TL, Chunks{}, vec_[kTMP],
                                                                      vec_[kV], vec_[kRHAT], d_opP_, d_opS_, d_st_,
                                                                      d_part_, d_cnt_);
    CKR_(cudaGetLastError(), 2);
    CKR_(cudaMemcpyAsync(out, vec_[kV], n * sizeof(double), cudaMemcpyDeviceToHost, stream_), 2);
  } else if (which == 3) {
    ensure_df_factors();
    // the operator of the BiCGSTAB iteration on an FP32 input (double-float
    // path): in rounded to FP32, then y = A x on the finest tower
    const BlockList TL = tower_list(finest_);
    const long w = (long)TL.n * ncell_;
    CKR_(cudaMemcpyAsync(vec_[kTMP], in, n * sizeof(double), cudaMemcpyHostToDevice, stream_), 2);
    k_narrow<<<ew_grid((long)n), kTPB, 0, stream_>>>((long long)n, vec_[kTMP], d_corr32_);
    CKR_(cudaMemsetAsync(vec_[kV], 0, n * sizeof(double), stream_), 2);
    CKR_(cudaMemsetAsync(vec_[kRHAT], 0, n * sizeof(double), stream_), 2);
    CKR_(cudaMemsetAsync(d_st_, 0, sizeof(FState), stream_), 2);
    if (tt_.ndim == 2)
      k_op_red<2, 0, float, false, true><<<red_grid(w), kTPB, 0, stream_>>>(
          topo_, cd64_, TL, Chunks{}, d_corr32_, vec_[kV], vec_[kRHAT], d_opP_, d_opS_, d_st_, d_part_, d_cnt_,
          nullptr, d_opP2_, d_opS2_, d_uni2_);
    else
      k_op_red<3, 0, float, false, true><<<red_grid(w), kTPB, 0, stream_>>>(
          topo_, cd64_, TL, Chunks{}, d_corr32_, vec_[kV], vec_[kRHAT], d_opP_, d_opS_, d_st_, d_part_, d_cnt_,
          nullptr, d_opP2_, d_opS2_, d_uni2_);
    CKR_(cudaGetLastError(), 2);
    CKR_(cudaMemcpyAsync(out, vec_[kV], n * sizeof(double), cudaMemcpyDeviceToHost, stream_), 2);
  } else if (which == 4) {
    // (above)
  } else if (which == 8) {
    // the operator by rows on the lists that a solve walks, in rounded to FP32
    if (tt_.nb % 4 != 0) return 1;
    CKR_(cudaMemcpyAsync(vec_[kTMP], in, n * sizeof(double), cudaMemcpyHostToDevice, stream_), 2);
    k_narrow<<<ew_grid((long)n), kTPB, 0, stream_>>>((long long)n, vec_[kTMP], d_corr32_);
    CKR_(cudaMemsetAsync(vec_[kV], 0, n * sizeof(double), stream_), 2);
    CKR_(cudaMemsetAsync(vec_[kRHAT], 0, n * sizeof(double), stream_), 2);
    CKR_(cudaMemsetAsync(d_st_, 0, sizeof(FState), stream_), 2);
    if (multi()) CKR_(cudaMemsetAsync(d_stc_, 0, ncomp_ * sizeof(FState), stream_), 2);
    solve_lists_ = true;
    launch_op_rows<0>(d_corr32_, vec_[kV], vec_[kRHAT]);
    solve_lists_ = false;
    CKR_(cudaGetLastError(), 2);
    CKR_(cudaMemcpyAsync(out, vec_[kV], n * sizeof(double), cudaMemcpyDeviceToHost, stream_), 2);
  } else if (which == 7) {
    // the FP32 pass, as the V-cycle runs it or by the general kernel (a list
    // without halo descriptors), from in or with level L prolonged first
    const int sweeps = (variant - 1) % 1024 + 1, form = (variant - 1) / 1024;
    const bool general = form & 1, top = form & 2;
    float *a = d_corr32_, *b = corr_alt<float>();
    std::vector<float> h(n);
    if (!err_.empty()) return 2;
    for (const auto &[src, dst] : {std::pair(in, a), std::pair(in2, d_resid32_)}) {
      for (size_t i = 0; i < n; i++) h[i] = (float)src[i];
      CKR_(cudaMemcpyAsync(dst, h.data(), n * sizeof(float), cudaMemcpyHostToDevice, stream_), 2);
      CKR_(cudaStreamSynchronize(stream_), 2);
    }
    BlockList TL = smooth_list(L);
    if (general) TL.hx = nullptr;
    const bool fused = top && !general && bhgs_prolongs<float>(topo_, c32_, TL);
    if (top && !fused) launch_prolong<float>(topo_, c32_, level_list(L), a, nullptr, stream_);
    CKR_(cudaMemcpyAsync(b, a, n * sizeof(float), cudaMemcpyDeviceToDevice, stream_), 2);
    launch_bhgs<float>(topo_, c32_, TL, sweeps, a, b, d_resid32_, nullptr, stream_, false, fused ? L : 0);
    CKR_(cudaGetLastError(), 2);
    CKR_(cudaMemcpyAsync(h.data(), b, n * sizeof(float), cudaMemcpyDeviceToHost, stream_), 2);
    CKR_(cudaStreamSynchronize(stream_), 2);
    for (size_t i = 0; i < n; i++) out[i] = (double)h[i];
  } else if (which == 2) {
    // one block-hybrid pass over every sublevel of tower L, `variant`
    // red-black sweeps per block: in (frozen) -> out
    CKR_(cudaMemcpyAsync(vec_[kTMP], in, n * sizeof(double), cudaMemcpyHostToDevice, stream_), 2);
    CKR_(cudaMemcpyAsync(vec_[kRESID], in2, n * sizeof(double), cudaMemcpyHostToDevice, stream_), 2);
    CKR_(cudaMemcpyAsync(vec_[kCORR], in, n * sizeof(double), cudaMemcpyHostToDevice, stream_), 2);
    launch_bhgs<double>(topo_, cd64_, smooth_list(L), variant, vec_[kTMP], vec_[kCORR], vec_[kRESID], nullptr,
                        stream_, false);
    CKR_(cudaGetLastError(), 2);
    CKR_(cudaMemcpyAsync(out, vec_[kCORR], n * sizeof(double), cudaMemcpyDeviceToHost, stream_), 2);
  } else {
    const int v = variant >= 0 ? variant : rbgs_var<double>();
    CKR_(cudaMemcpyAsync(vec_[kCORR], in, n * sizeof(double), cudaMemcpyHostToDevice, stream_), 2);
    CKR_(cudaMemcpyAsync(vec_[kRESID], in2, n * sizeof(double), cudaMemcpyHostToDevice, stream_), 2);
    for (int ll = L; ll >= 1; ll--) {
      const BlockList sl = sublevel_list(L, ll);
      if (sl.n == 0) continue;
      for (int rb = 0; rb < 2; rb++)
        launch_rbgs<double>(topo_, cd64_, sl, rb, vec_[kCORR], vec_[kRESID], nullptr, stream_, false, v);
    }
    CKR_(cudaGetLastError(), 2);
    CKR_(cudaMemcpyAsync(out, vec_[kCORR], n * sizeof(double), cudaMemcpyDeviceToHost, stream_), 2);
  }
  CKR_(cudaStreamSynchronize(stream_), 2);
  if (rbgs_bulk_error(topo_.err, stream_, true) > 0) {
    fail("device smoother: a bounded wait timed out");
    return 2;
  }
  return err_.empty() ? 0 : 2;
}

// self-test of the integer-pipe conversions against the hardware ones
__global__ void k_fp_selftest(int n, const double *d, const float *f, float *nar, float *nar_hw, double *wid,
                              double *wid_hw, double *wid0, double *wid0_hw) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    nar[i] = fpint::narrow(d[i]);
    nar_hw[i] = (float)d[i];
    wid[i] = fpint::widen(f[i]);
    wid_hw[i] = (double)f[i];
    wid0[i] = fpint::widen_plus0(f[i]);
    wid0_hw[i] = 0.0 + (double)f[i];
  }
}

int fp_selftest(const double *d, const float *f, int n, float *nar, float *nar_hw, double *wid, double *wid_hw,
                double *wid0, double *wid0_hw) {
  if (n <= 0) return 0;
  unsigned char *buf = nullptr;
  const size_t fb = (size_t)n * sizeof(float), db = (size_t)n * sizeof(double);
  if (dev_malloc(&buf, 3 * fb + 5 * db) != cudaSuccess) return 2;
  double *dd = (double *)buf, *w = dd + n, *whw = w + n, *w0 = whw + n, *w0hw = w0 + n;
  float *ff = (float *)(w0hw + n), *nr = ff + n, *nrhw = nr + n;
  cudaMemcpy(dd, d, db, cudaMemcpyHostToDevice);
  cudaMemcpy(ff, f, fb, cudaMemcpyHostToDevice);
  k_fp_selftest<<<std::min((n + 255) / 256, 1024), 256>>>(n, dd, ff, nr, nrhw, w, whw, w0, w0hw);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e == cudaSuccess) {
    cudaMemcpy(nar, nr, fb, cudaMemcpyDeviceToHost);
    cudaMemcpy(nar_hw, nrhw, fb, cudaMemcpyDeviceToHost);
    cudaMemcpy(wid, w, db, cudaMemcpyDeviceToHost);
    cudaMemcpy(wid_hw, whw, db, cudaMemcpyDeviceToHost);
    cudaMemcpy(wid0, w0, db, cudaMemcpyDeviceToHost);
    cudaMemcpy(wid0_hw, w0hw, db, cudaMemcpyDeviceToHost);
  }
  dev_free(buf);
  return e == cudaSuccess ? 0 : 2;
}

}  // namespace sayaka_gb300
