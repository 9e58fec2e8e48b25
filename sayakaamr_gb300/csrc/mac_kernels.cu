// Stencil, smoother and inter-level transfer kernels of the MAC solver.
//
// Every kernel works on one block list (a tower, one level of a tower, or a
// tree level) in a single launch, one thread per (block, cell).  Values that
// the reference obtains through ghost-cell fills and coarse/fine flux
// registers are gathered directly:
//   FINE_FINE face : the neighbour block's boundary cell
//                    (src/SayakaFillPatch.cpp:92-190)
//   FINE_CRSE face : the coarse leaf behind the parent's face, injected
//                    (src/SayakaFillPatch.cpp:192-299, src/SayakaInterpPatch.cpp:157-189)
//   CRSE_FINE face : sum over the fine faces of T_fine * phi_fine, i.e. the
//                    fine-side save + RESTRICT_SUM + copy of
//                    src/SayakaTower.cpp:298-415, src/SayakaInterpPatch.cpp:627-691
// The arithmetic is written operation by operation in the reference's order
// (src/SayakaMacOperator.cpp:1115-1459) and this file is compiled without
// FMA contraction, so FP64 results are bit-identical to the reference's.
#include <algorithm>
#include <cstdint>

#include "mac_device.h"
#include "mac_stencil.cuh"
#include "launch.cuh"

namespace sayaka_gb300 {

namespace {

constexpr int kThreads = 256;
// CTAs over a reduced list (BlockList::pb), whose length the host does not
// know: about two rounds of resident CTAs, which walk it in strides, instead
// of one CTA per entry of the full list, most of which would only read the
// bounds and leave
constexpr int kReducedGrid = 152 * 16;
using namespace stencil;

// ---------------------------------------------------------------------------
// MAC operator L(phi) = (phi_c*sum T - sum T*phi_nb) / (dv*vf)
// (src/SayakaMacOperator.cpp:1325-1459); residual variant
// r = rhs - L(phi) (src/SayakaMacUtil.cpp:9-49)
template <typename T, int ND>
__global__ void __launch_bounds__(kThreads) k_apply(Topo t, Coef<T> c, BlockList L, const T *__restrict__ x,
                                                    T *__restrict__ y, const T *__restrict__ rhs, const int *guard) {
  pdl_enter();
  if (guard && *guard) return;
  const int ncell = t.ncell;
  const long total = (long)L.n * ncell;
  for (long it = blockIdx.x * (long)blockDim.x + threadIdx.x; it < total; it += (long)gridDim.x * blockDim.x) {
    const int p = (int)(it / ncell);
    const int ci = (int)(it - (long)p * ncell);
    const int b = L.blocks[p];
    if (block_off(L, b)) continue;
    const long q = (long)b * ncell + ci;
    T out = apply_cell<T, ND>(t, c, b, L.ftypes[p], ci, x);
    if (rhs) out = c.vf[q] > 0 ? rhs[q] - out : (T)0;
    y[q] = out;
  }
}

// ---------------------------------------------------------------------------
// red-black Gauss-Seidel, one colour over one level of a tower
// (src/SayakaMacOperator.cpp:1191-1323).  Colour = (i+j+k)%2 in block-local
// indices; nb is even so colours match across same-level block faces.
template <typename T, int ND>
__global__ void __launch_bounds__(kThreads) k_smooth(Topo t, Coef<T> c, BlockList L, int color, T *__restrict__ phi,
                                                     const T *__restrict__ rhs, const int *guard) {
  pdl_enter();
  if (guard && *guard) return;
  const int nhalf = t.ncell >> 1;
  const long total = (long)L.n * nhalf;
  for (long it = blockIdx.x * (long)blockDim.x + threadIdx.x; it < total; it += (long)gridDim.x * blockDim.x) {
    const int p = (int)(it / nhalf);
    int ijk[3];
    color_cell<ND>((int)(it - (long)p * nhalf), t.nb, color, ijk);
    smooth_cell<T, ND>(t, c, L.blocks[p], L.ftypes[p], ijk, phi, rhs);
  }
}

// the device solve's smoother (smooth_cell_fast): blockIdx.y walks the
// blocks of the list, blockIdx.x the chunks of a block's half cells, so the
// block id and face types are uniform across a CTA and no thread divides
template <typename T, int ND, int MINB>
__global__ void __launch_bounds__(kThreads, MINB) k_rbgs(Topo t, Coef<T> c, BlockList L, int color,
                                                         T *__restrict__ phi, const T *__restrict__ rhs,
                                                         const int *guard) {
  pdl_enter();
  if (guard && *guard) return;
  const int h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= (t.ncell >> 1)) return;
  int ijk[3];
  color_cell_fast<ND>(h, t, color, ijk);
  const ListRange lr = list_range(L);
  for (int p = lr.a + blockIdx.y; p < lr.b; p += gridDim.y) {
    const long fo = factor_entry(L, p) * t.ncell;
    if (L.stc && block_off(L, L.hx ? L.hx[(long)p * kHX + kHXBlock] : L.blocks[p])) continue;
    if (L.hx) {
      const int *e = L.hx + (long)p * kHX;
      smooth_cell_fast<T, ND>(t, c, e[kHXBlock], (uint16_t)(e[kHXInfo] & 0xffff), ijk, phi, rhs,
                              L.sa ? L.sa + fo : nullptr, L.ia ? L.ia + fo : nullptr, e);
    } else {
      smooth_cell_fast<T, ND>(t, c, L.blocks[p], L.ftypes[p], ijk, phi, rhs, L.sa ? L.sa + fo : nullptr,
                              L.ia ? L.ia + fo : nullptr);
    }
  }
}

// the same sweep with CPT cells per thread, the same cell of CPT blocks
// (entries p, p + G, ..., G = gridDim.y): every cell's operands are gathered
// before any is updated, so that a thread keeps CPT cells' loads in flight
// (smooth_gather / smooth_update: the values of smooth_cell_fast)
template <typename T, int ND, int MINB, int CPT, bool FAC>
__global__ void __launch_bounds__(kThreads, MINB) k_rbgs_ilp(Topo t, Coef<T> c, BlockList L, int color,
                                                             T *__restrict__ phi, const T *__restrict__ rhs,
                                                             const int *guard) {
  pdl_enter();
  if (guard && *guard) return;
  const int h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= (t.ncell >> 1)) return;
  int ijk[3];
  color_cell_fast<ND>(h, t, color, ijk);
  const int G = gridDim.y;
  const ListRange lr = list_range(L);
  for (int p0 = lr.a + blockIdx.y; p0 < lr.b; p0 += CPT * G) {
    SmoothOps<T, ND, FAC> o[CPT];
    bool on[CPT];
#pragma unroll
    for (int k = 0; k < CPT; k++) {
      const int p = p0 + k * G;
      on[k] = false;
      if (p >= lr.b) continue;
      const long fo = factor_entry(L, p) * t.ncell;
      const int *e = L.hx ? L.hx + (long)p * kHX : nullptr;
      const int b = e ? e[kHXBlock] : L.blocks[p];
      if (L.stc && block_off(L, b)) continue;
      const uint16_t ft = e ? (uint16_t)(e[kHXInfo] & 0xffff) : L.ftypes[p];
      smooth_gather<T, ND, FAC>(t, c, b, ft, ijk, phi, rhs, FAC ? L.sa + fo : nullptr, FAC ? L.ia + fo : nullptr, e,
                                o[k]);
      on[k] = true;
    }
#pragma unroll
    for (int k = 0; k < CPT; k++)
      if (on[k]) smooth_update<T, ND, FAC>(c, o[k], phi);
  }
}

// (fluid: block b is known to have vf = 1 everywhere)
template <typename T, int ND>
__device__ __forceinline__ T prolonged_value(const Topo &t, const Coef<T> &c, int b, const int ijk[3],
                                             const T *__restrict__ phi, int pw = -1, bool fluid = false) {
  const int nb = t.nb, half = nb >> 1;
  const int P = pw >= 0 ? pw >> 3 : t.parent[b], wc = pw >= 0 ? pw & 7 : t.which_child[b];
  int pc[3] = {0, 0, 0};
  for (int q = 0; q < ND; q++) pc[q] = ((wc >> q) & 1) * half + (ijk[q] >> 1);
  const long q = (long)b * t.ncell + encode(ijk, nb);
  return (fluid || positive(c.vf[q])) ? phi[(long)P * t.ncell + encode(pc, nb)] : (T)0;
}

// ---- 2D FP32 blocks of 16x16 cells, one warp per block --------------------
// Lane l holds the cells of row l/2, columns 8(l%2) .. 8(l%2)+7, in registers.
// What crosses the block's boundary is gathered first, one boundary face cell
// per lane, into 64 slots of the warp's shared memory (slot 16 f + m: face f,
// m-th cell along it): the face's part of the diagonal, its off-diagonal
// factor and the value behind it, by face type as smooth_cell_fast takes them
// (same-level: T, T and the neighbour's cell; physical: 0 or 2T, 0 and 0;
// FINE_CRSE: T/1.5 twice and the coarse cell; CRSE_FINE: T/0.75, 1 and the
// sum over the fine faces).  Blocks with a body's surface, a density front
// or a coarse/fine face then take the same few instructions per cell as the
// others; cell by cell (smooth_cell_fast) they took about five times as many,
// and they are the greater part of a tree's finest level, which is refined
// where they lie.  Bound by the latency of the loads (descriptor, then
// record, rows, halo and coefficients at once) and by issue, not by bytes.
constexpr int kW16Slots = 64;
struct W16Halo {
  float dp[kW16Slots], k[kW16Slots], v[kW16Slots];
};

// slot of face f, m-th face cell: its contribution to the cell of the block
// behind it (PROLONG: a same-level neighbour's value prolonged from that
// neighbour's parent).  The gathers of mac_stencil.cuh for 2D blocks of 16,
// without their arrays: the direction differs from lane to lane, and arrays
// indexed by it would live in local memory.
// (FINE: the finer blocks behind a refined face hold prolonged values too,
// those of this block's neighbour there, their parent)
template <bool PROLONG, bool FINE = false>
__device__ __forceinline__ void w16_halo_slot(const Topo &t, const Coef<float> &c, const int *e, int b, int info,
                                              const float *u, int f, int m, const float *__restrict__ phi, float &dp,
                                              float &k, float &v) {
  constexpr int NB = 16, NC = 256;
  const int d = f >> 1, s = f & 1;
  const int ty = face_type_of((uint16_t)(info & 0xffff), f);
  const float *tff = d ? c.tff[1] : c.tff[0];
  const long fx = (long)b * t.nfb + (d ? m + NB * (s * NB) : s * NB + (NB + 1) * m);
  const int across = s ? 0 : NB - 1;  // the neighbour's cell layer at the face
  dp = k = v = 0.f;
  if (ty == 0) {
    const long n = e[f];
    dp = k = u ? u[d] : tff[fx];
    if constexpr (PROLONG) {
      const int pw = e[kHXPar + f], wc = pw & 7;
      const int i = d ? m : across, j = d ? across : m;
      const bool fluid = c.vf[n * NC + i + NB * j] > 0;
      const float pv = phi[(long)(pw >> 3) * NC + 8 * (wc & 1) + (i >> 1) + NB * (8 * ((wc >> 1) & 1) + (j >> 1))];
      v = fluid ? pv : 0.f;
    } else {
      v = phi[n * NC + (d ? m + NB * across : across + NB * m)];
    }
  } else if (ty == 1) {
    if (t.bc_type[b * 6 + f] != kBCNeumann) dp = (u ? u[d] : tff[fx]) * 2.0f;
  } else if (ty == 2) {
    const int tc = 8 * ((info >> (17 - d)) & 1) + (m >> 1);  // which_child >> (1 - d)
    dp = k = c.cf[((long)b * 4 + f) * NB + m];
    v = phi[(long)e[f] * NC + (d ? tc + NB * across : across + NB * tc)];
  } else {
    const int half = m >> 3, F = e[kHXKids + 4 * f + half], t0 = 2 * (m - 8 * half);
    dp = c.cf[((long)b * 4 + f) * NB + m];
    k = 1.f;
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const float tf = c.cf[((long)F * 4 + (f ^ 1)) * NB + t0 + q];
      const long fc = (long)F * NC + (d ? t0 + q + NB * across : across + NB * (t0 + q));
      if constexpr (FINE)
        v += tf * (c.vf[fc] > 0 ? phi[(long)t.neighbor[b * 6 + f] * NC + (d ? m + NB * across : across + NB * m)] : 0.f);
      else
        v += tf * phi[fc];
    }
  }
}

// the cells of colour `color` of list entry e (its halo descriptor): the
// values and operations of smooth_cell_fast (PROLONG: of k_prolong_red) in
// the same order, so the same bits.  A row's cells of the colour are the
// columns 2q + par, q < 4; they stay in cc, the others in oc.
template <bool PROLONG>
__device__ __forceinline__ void w16_sweep(const Topo &t, const Coef<float> &c, const BlockList &L, const int *e,
                                          int color, float *__restrict__ phi, const float *__restrict__ rhs, int lane,
                                          W16Halo &sh) {
  constexpr int NB = 16, NC = 256;
  const int j = lane >> 1, hh = lane & 1, c0 = 8 * hh, par = (color + j) & 1;
  const int2 ib = *reinterpret_cast<const int2 *>(e + kHXInfo);
  const int b = ib.y;
  const long cb = (long)b * NC, fb = (long)b * t.nfb;
  const float *u = uniform_of(c, b);
  const float dv = geom(c, b, 6);
  float cc[4], oc[4];
  if constexpr (PROLONG) {
    // columns 2q and 2q+1 of the row have the same parent cell
    const int pw = e[kHXPar + 6], P = pw >> 3, wc = pw & 7;
    const float4 q4 = *reinterpret_cast<const float4 *>(phi + (long)P * NC + (8 * ((wc >> 1) & 1) + (j >> 1)) * NB +
                                                         8 * (wc & 1) + 4 * hh);
    cc[0] = oc[0] = q4.x, cc[1] = oc[1] = q4.y, cc[2] = oc[2] = q4.z, cc[3] = oc[3] = q4.w;
  } else {
    const float4 *src = reinterpret_cast<const float4 *>(phi + cb + j * NB + c0);
    const float4 p0 = src[0], p1 = src[1];
    cc[0] = par ? p0.y : p0.x, cc[1] = par ? p0.w : p0.z, cc[2] = par ? p1.y : p1.x, cc[3] = par ? p1.w : p1.z;
    oc[0] = par ? p0.x : p0.y, oc[1] = par ? p0.z : p0.w, oc[2] = par ? p1.x : p1.y, oc[3] = par ? p1.z : p1.w;
  }
  const float4 *rsrc = reinterpret_cast<const float4 *>(rhs + cb + j * NB + c0);
  const float4 r0 = rsrc[0], r1 = rsrc[1];
  const float r[4] = {par ? r0.y : r0.x, par ? r0.w : r0.z, par ? r1.y : r1.x, par ? r1.w : r1.z};
  // the boundary face cells of the colour: eight per face, one per lane
  const int hf = lane >> 3, hm = 2 * (lane & 7) + ((color + (hf & 1)) & 1);
  float hdp, hk, hv;
  w16_halo_slot<PROLONG>(t, c, e, b, ib.x, u, hf, hm, phi, hdp, hk, hv);
  // face coefficients and volume fractions of the colour's cells
  float tx[8], ty0[4], ty1[4], vf[4];
  if (u) {
    const float T0 = u[0], T1 = u[1];
#pragma unroll
    for (int q = 0; q < 4; q++) tx[2 * q] = tx[2 * q + 1] = T0, ty0[q] = ty1[q] = T1, vf[q] = 1.f;
  } else {
    const float *x = c.tff[0] + fb + (NB + 1) * j + c0 + par;
#pragma unroll
    for (int n = 0; n < 8; n++) tx[n] = x[n];
    const float *y = c.tff[1] + fb + NB * j + c0 + par;
    const float *w = c.vf + cb + NB * j + c0;
#pragma unroll
    for (int q = 0; q < 4; q++) ty0[q] = y[2 * q], ty1[q] = y[2 * q + NB];
    const float4 w0 = *reinterpret_cast<const float4 *>(w), w1 = *reinterpret_cast<const float4 *>(w + 4);
    vf[0] = par ? w0.y : w0.x, vf[1] = par ? w0.w : w0.z, vf[2] = par ? w1.y : w1.x, vf[3] = par ? w1.w : w1.z;
    if constexpr (PROLONG) {
      const float ov[4] = {par ? w0.x : w0.y, par ? w0.z : w0.w, par ? w1.x : w1.y, par ? w1.z : w1.w};
#pragma unroll
      for (int q = 0; q < 4; q++) {
        if (!(vf[q] > 0.f)) cc[q] = 0.f;
        if (!(ov[q] > 0.f)) oc[q] = 0.f;
      }
    }
  }
  if (L.stc && block_off(L, b)) return;  // a finished problem; uniform over the warp
  __syncwarp();                          // the slots of the warp's previous block have been read
  sh.dp[16 * hf + hm] = hdp;
  sh.k[16 * hf + hm] = hk;
  sh.v[16 * hf + hm] = hv;
  __syncwarp();
  // the neighbours of a cell have the other colour: rows j-1 and j+1 hold
  // them in oc of lanes l-2 and l+2, the row's own are oc[q-1], oc[q] (par 0)
  // or oc[q], oc[q+1] (par 1), the outermost from the other half of the row
  const float fl = __shfl_up_sync(0xffffffffu, oc[3], 1), fr = __shfl_down_sync(0xffffffffu, oc[0], 1);
  float dn[4], up[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    dn[q] = __shfl_up_sync(0xffffffffu, oc[q], 2);
    up[q] = __shfl_down_sync(0xffffffffu, oc[q], 2);
  }
#pragma unroll
  for (int q = 0; q < 4; q++) {
    float kl = tx[2 * q], kr = tx[2 * q + 1], kd = ty0[q], ku = ty1[q];
    float dl = kl, dr = kr, dd = kd, du = ku;
    float vl = par ? oc[q] : (q > 0 ? oc[q > 0 ? q - 1 : 0] : fl);
    float vr = par ? (q < 3 ? oc[q < 3 ? q + 1 : 3] : fr) : oc[q];
    float vd = dn[q], vu = up[q];
    const int i = c0 + 2 * q + par;
    if (q == 0 && i == 0) dl = sh.dp[j], kl = sh.k[j], vl = sh.v[j];
    if (q == 3 && i == NB - 1) dr = sh.dp[16 + j], kr = sh.k[16 + j], vr = sh.v[16 + j];
    if (j == 0) dd = sh.dp[32 + i], kd = sh.k[32 + i], vd = sh.v[32 + i];
    if (j == NB - 1) du = sh.dp[48 + i], ku = sh.k[48 + i], vu = sh.v[48 + i];
    float diag = c.alpha * dv, off = 0.f;
    diag += dl;
    off = fma_t(kl, vl, off);
    diag += dr;
    off = fma_t(kr, vr, off);
    diag += dd;
    off = fma_t(kd, vd, off);
    diag += du;
    off = fma_t(ku, vu, off);
    cc[q] = (vf[q] > 0.f && diag > 0.f) ? relax(c.omega, fast_div(fma_t(r[q] * dv, vf[q], off), diag), cc[q]) : 0.f;
  }
  // the block is written back whole, the other colour's cells with the values
  // that concurrent readers see in any case
  float4 *dst = reinterpret_cast<float4 *>(phi + cb + j * NB + c0);
  dst[0] = par ? make_float4(oc[0], cc[0], oc[1], cc[1]) : make_float4(cc[0], oc[0], cc[1], oc[1]);
  dst[1] = par ? make_float4(oc[2], cc[2], oc[3], cc[3]) : make_float4(cc[2], oc[2], cc[3], oc[3]);
}

// prolongation of a level fused with its first red sweep (k_prolong_red's
// values), one warp per block of L, then one warp per block of X for the red
// sweep of the coarser same-parity sublevels
template <int MINB>
__global__ void __launch_bounds__(kThreads, MINB) k_prolong_red_warp16(Topo t, Coef<float> c, BlockList L,
                                                                       float *__restrict__ phi,
                                                                       const float *__restrict__ rhs,
                                                                       const int *guard, BlockList X) {
  __shared__ W16Halo sh[kThreads / 32];
  pdl_enter();
  if (guard && *guard) return;
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const ListRange lr = list_range(L), xr = list_range(X);
  const int nl = lr.b - lr.a, nx = xr.b - xr.a;
  for (int p = blockIdx.x * warps + (threadIdx.x >> 5); p < nl + nx; p += gridDim.x * warps) {
    if (p < nl)
      w16_sweep<true>(t, c, L, L.hx + (long)(lr.a + p) * kHX, 0, phi, rhs, lane, sh[threadIdx.x >> 5]);
    else
      w16_sweep<false>(t, c, X, X.hx + (long)(xr.a + p - nl) * kHX, 0, phi, rhs, lane, sh[threadIdx.x >> 5]);
  }
}

// one colour of a red-black sweep, one warp per block
template <int MINB>
__global__ void __launch_bounds__(kThreads, MINB) k_rbgs_warp16(Topo t, Coef<float> c, BlockList L, int color,
                                                                float *__restrict__ phi, const float *__restrict__ rhs,
                                                                const int *guard) {
  __shared__ W16Halo sh[kThreads / 32];
  pdl_enter();
  if (guard && *guard) return;
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const ListRange lr = list_range(L);
  for (int p = lr.a + blockIdx.x * warps + (threadIdx.x >> 5); p < lr.b; p += gridDim.x * warps)
    w16_sweep<false>(t, c, L, L.hx + (long)p * kHX, color, phi, rhs, lane, sh[threadIdx.x >> 5]);
}

// The block-hybrid pass (k_bhgs) over 2D FP32 blocks of 16x16 cells, one warp
// per block: nsweep red-black sweeps of the block in registers with the values
// outside it frozen, from src into dst.  Everything the sweeps read is loaded
// once, at the start; a sweep is then shuffles and arithmetic, without the
// shared-memory tile, the reloads of coefficients and right-hand side and the
// two CTA barriers per sweep that the CTA form has.  The values and operations
// of k_bhgs in the same order: a frozen neighbour's part enters as 1 * (T
// value), its rounded product.  Bound by the latency of one round of loads.
// TOP: src holds no values yet for the blocks of level `top`, which start from
// their parents' (k_prolong's values).
template <bool TOP>
__device__ __forceinline__ void h16_pass(const Topo &t, const Coef<float> &c, const BlockList &L, const int *e,
                                         int top, int nsweep, const float *__restrict__ src, float *__restrict__ dst,
                                         const float *__restrict__ rhs, int lane, W16Halo &sh) {
  constexpr int NB = 16, NC = 256;
  const int j = lane >> 1, hh = lane & 1, c0 = 8 * hh, par = j & 1;  // red cells: columns 2q + par
  const int2 ib = *reinterpret_cast<const int2 *>(e + kHXInfo);
  const int b = ib.y;
  const long cb = (long)b * NC, fb = (long)b * t.nfb;
  const float *u = uniform_of(c, b);
  const float dv = geom(c, b, 6);
  const int below = TOP ? top - e[kHXLevel] : -1;  // 0: the block itself is prolonged, 1: the finer ones at its faces
  float4 p0, p1;
  if (TOP && below == 0) {
    const int pw = e[kHXPar + 6], wc = pw & 7;
    const float4 q4 = *reinterpret_cast<const float4 *>(src + (long)(pw >> 3) * NC +
                                                         (8 * ((wc >> 1) & 1) + (j >> 1)) * NB + 8 * (wc & 1) + 4 * hh);
    p0 = make_float4(q4.x, q4.x, q4.y, q4.y);
    p1 = make_float4(q4.z, q4.z, q4.w, q4.w);
  } else {
    const float4 *s4 = reinterpret_cast<const float4 *>(src + cb + j * NB + c0);
    p0 = s4[0], p1 = s4[1];
  }
  const float4 *rsrc = reinterpret_cast<const float4 *>(rhs + cb + j * NB + c0);
  const float4 r0 = rsrc[0], r1 = rsrc[1];
  float hdp[2], hk[2], hv[2];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int f = (lane >> 4) + 2 * h, m = lane & 15;
    if (TOP && below == 0)
      w16_halo_slot<true>(t, c, e, b, ib.x, u, f, m, src, hdp[h], hk[h], hv[h]);
    else if (TOP && below == 1)
      w16_halo_slot<false, true>(t, c, e, b, ib.x, u, f, m, src, hdp[h], hk[h], hv[h]);
    else
      w16_halo_slot<false>(t, c, e, b, ib.x, u, f, m, src, hdp[h], hk[h], hv[h]);
  }
  // v[color][q]; the face coefficients, diagonal, rhs * dv and vf of the cell
  float v[2][4], kl[2][4], kr[2][4], kd[2][4], ku[2][4], diag[2][4], rd[2][4], vf[2][4];
  const float pv[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
  const float rv[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
#pragma unroll
  for (int q = 0; q < 4; q++) {
    v[0][q] = par ? pv[2 * q + 1] : pv[2 * q];
    v[1][q] = par ? pv[2 * q] : pv[2 * q + 1];
    rd[0][q] = (par ? rv[2 * q + 1] : rv[2 * q]) * dv;
    rd[1][q] = (par ? rv[2 * q] : rv[2 * q + 1]) * dv;
  }
  if (u) {
    const float T0 = u[0], T1 = u[1];
#pragma unroll
    for (int k = 0; k < 2; k++)
#pragma unroll
      for (int q = 0; q < 4; q++) kl[k][q] = kr[k][q] = T0, kd[k][q] = ku[k][q] = T1, vf[k][q] = 1.f;
  } else {
    const float *x = c.tff[0] + fb + (NB + 1) * j + c0;
    float tx[9];
#pragma unroll
    for (int n = 0; n < 9; n++) tx[n] = x[n];
    const float4 *y = reinterpret_cast<const float4 *>(c.vf + cb + NB * j + c0);
    const float4 w0 = y[0], w1 = y[1];
    const float wv[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
    const float *yd = c.tff[1] + fb + NB * j + c0;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      kl[0][q] = par ? tx[2 * q + 1] : tx[2 * q];
      kr[0][q] = par ? tx[2 * q + 2] : tx[2 * q + 1];
      kl[1][q] = par ? tx[2 * q] : tx[2 * q + 1];
      kr[1][q] = par ? tx[2 * q + 1] : tx[2 * q + 2];
      kd[0][q] = yd[2 * q + par];
      kd[1][q] = yd[2 * q + 1 - par];
      ku[0][q] = yd[2 * q + par + NB];
      ku[1][q] = yd[2 * q + 1 - par + NB];
      vf[0][q] = par ? wv[2 * q + 1] : wv[2 * q];
      vf[1][q] = par ? wv[2 * q] : wv[2 * q + 1];
      if (TOP && below == 0) {
        if (!(vf[0][q] > 0.f)) v[0][q] = 0.f;
        if (!(vf[1][q] > 0.f)) v[1][q] = 0.f;
      }
    }
  }
  if (L.stc && block_off(L, b)) return;  // a finished problem; uniform over the warp
  __syncwarp();                          // the slots of the warp's previous block have been read
#pragma unroll
  for (int h = 0; h < 2; h++) {
    // the frozen part: T * value (CRSE_FINE: the sum itself), rounded
    sh.dp[lane + 32 * h] = hdp[h];
    sh.v[lane + 32 * h] = hk[h] * hv[h];
  }
  __syncwarp();
  // boundary cells: the slot's diagonal part, factor 1, the frozen part as
  // the neighbour's value (hx: left or right, hy: below or above)
  float hx = 0.f, hy[2][4];
  const bool edge_y = j == 0 || j == NB - 1;
#pragma unroll
  for (int k = 0; k < 2; k++)
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int pk = k ? 1 - par : par, i = c0 + 2 * q + pk;
      float dl = kl[k][q], dr = kr[k][q], dd = kd[k][q], du = ku[k][q];
      if (q == 0 && i == 0) dl = sh.dp[j], kl[k][q] = 1.f, hx = sh.v[j];
      if (q == 3 && i == NB - 1) dr = sh.dp[16 + j], kr[k][q] = 1.f, hx = sh.v[16 + j];
      hy[k][q] = 0.f;
      if (j == 0) dd = sh.dp[32 + i], kd[k][q] = 1.f, hy[k][q] = sh.v[32 + i];
      if (j == NB - 1) du = sh.dp[48 + i], ku[k][q] = 1.f, hy[k][q] = sh.v[48 + i];
      float g = c.alpha * dv;
      g += dl;
      g += dr;
      g += dd;
      g += du;
      diag[k][q] = vf[k][q] > 0.f ? g : 0.f;  // 0: the cell stays at 0
    }
  for (int sw = 0; sw < nsweep; sw++) {
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const int pk = k ? 1 - par : par;
      float(&o)[4] = v[1 - k];
      const float fl = __shfl_up_sync(0xffffffffu, o[3], 1), fr = __shfl_down_sync(0xffffffffu, o[0], 1);
      float nd[4], nu[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        nd[q] = __shfl_up_sync(0xffffffffu, o[q], 2);
        nu[q] = __shfl_down_sync(0xffffffffu, o[q], 2);
      }
#pragma unroll
      for (int q = 0; q < 4; q++) {
        float vl = pk ? o[q] : (q > 0 ? o[q > 0 ? q - 1 : 0] : (hh ? fl : hx));
        float vr = pk ? (q < 3 ? o[q < 3 ? q + 1 : 3] : (hh ? hx : fr)) : o[q];
        const float vd = edge_y && j == 0 ? hy[k][q] : nd[q], vu = edge_y && j != 0 ? hy[k][q] : nu[q];
        float off = 0.f;
        off = fma_t(kl[k][q], vl, off);
        off = fma_t(kr[k][q], vr, off);
        off = fma_t(kd[k][q], vd, off);
        off = fma_t(ku[k][q], vu, off);
        v[k][q] = diag[k][q] > 0.f
                      ? relax(c.omega, fast_div(fma_t(rd[k][q], vf[k][q], off), diag[k][q]), v[k][q])
                      : 0.f;
      }
    }
  }
  float4 *d4 = reinterpret_cast<float4 *>(dst + cb + j * NB + c0);
  d4[0] = par ? make_float4(v[1][0], v[0][0], v[1][1], v[0][1]) : make_float4(v[0][0], v[1][0], v[0][1], v[1][1]);
  d4[1] = par ? make_float4(v[1][2], v[0][2], v[1][3], v[0][3]) : make_float4(v[0][2], v[1][2], v[0][3], v[1][3]);
}

constexpr int kH16Threads = 128;
template <int MINB, bool TOP>
__global__ void __launch_bounds__(kH16Threads, MINB) k_bhgs_warp16(Topo t, Coef<float> c, BlockList L, int nsweep,
                                                                   const float *__restrict__ src,
                                                                   float *__restrict__ dst,
                                                                   const float *__restrict__ rhs, const int *guard,
                                                                   int top) {
  __shared__ W16Halo sh[kH16Threads / 32];
  pdl_enter();
  if (guard && *guard) return;
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const ListRange lr = list_range(L);
  for (int p = lr.a + blockIdx.x * warps + (threadIdx.x >> 5); p < lr.b; p += gridDim.x * warps)
    h16_pass<TOP>(t, c, L, L.hx + (long)p * kHX, top, nsweep, src, dst, rhs, lane, sh[threadIdx.x >> 5]);
}

// ---- 3D FP32 blocks of 8^3 cells, one thread per row of cells along x ------
// A thread updates the four cells of the colour in its row.  Their neighbours
// are in the row itself and, at the same places, in the four adjoining rows,
// which it loads 32 bytes at a time from the block or from the block behind a
// same-level face, so a sweep needs no shared memory and no barrier and only
// coarse/fine faces take another path.  One thread per cell spends most of its
// instructions on indices and boundary tests.  PROLONG: the values are those of
// the parents (k_prolong_red's).  Bound by the latency of the loads.  13.75 M
// cells, 5,366 of 30,697 blocks without a cut: a sweep 16.5 -> 11.0 us, the
// fused prolongation 93 -> 29 us.  CTAs per SM of a sweep of the finest level:
// 23.1 us at 8, 19.0 at 12, 18.8 at 16 (one thread per cell: 33.2).
struct Row4 {  // diagonal and off-diagonal sums of the four cells
  float g[4], o[4];
};
// a coarser or refined neighbour behind y or z face f, cells a0, a0 + 2, ..
// along x, other transverse index a1 (with d = 0: one cell, a0 = j, a1 = k)
template <int N>
static __device__ __noinline__ Row4 rows8_cross(const float *__restrict__ cf, const float *__restrict__ phi,
                                                const int *__restrict__ e, int f, int a0, int a1, Row4 s) {
  constexpr int NB = 8, NC = 512, NF = 64;
  const int d = f >> 1, across = (f & 1) ? 0 : NB - 1, info = e[kHXInfo], b = e[kHXBlock];
  const int su = d == 0 ? NB : 1, sv = d == 2 ? NB : NB * NB, sd = d == 0 ? 1 : (d == 1 ? NB : NB * NB);
  const float *own = cf + ((long)b * 6 + f) * NF + NB * a1;
  if (((info >> (2 * f)) & 3) == 2) {
    const int wc = info >> 16, q0 = d == 0 ? 1 : 0, q1 = d == 2 ? 1 : 2;
    const float *x = phi + (long)e[f] * NC + across * sd + (4 * ((wc >> q1) & 1) + (a1 >> 1)) * sv;
    const int t0 = 4 * ((wc >> q0) & 1);
#pragma unroll
    for (int n = 0; n < N; n++) {
      const float k = own[a0 + 2 * n];
      s.g[n] += k;
      s.o[n] = fma_t(k, x[(t0 + ((a0 + 2 * n) >> 1)) * su], s.o[n]);
    }
    return s;
  }
  const int h1 = a1 >> 2;
#pragma unroll
  for (int n = 0; n < N; n++) {
    const int i = a0 + 2 * n, h0 = i >> 2;
    const long F = e[kHXKids + 4 * f + h0 + 2 * h1];
    const int t0 = 2 * (i - 4 * h0), t1 = 2 * (a1 - 4 * h1);
    const float *w = cf + (F * 6 + (f ^ 1)) * NF + t0 + NB * t1;
    const float *x = phi + F * NC + across * sd + t0 * su + t1 * sv;
    float v = 0.f;
    v += w[0] * x[0];
    v += w[1] * x[su];
    v += w[NB] * x[sv];
    v += w[NB + 1] * x[su + sv];
    s.g[n] += own[i];
    s.o[n] += v;
  }
  return s;
}

template <bool PROLONG>
__device__ __forceinline__ void rows8_sweep(const Topo &t, const Coef<float> &c, const BlockList &L, const int *e,
                                            int color, float *__restrict__ phi, const float *__restrict__ rhs) {
  constexpr int NB = 8, NC = 512;
  const int tid = threadIdx.x, j = tid & 7, k = tid >> 3, pk = (color + j + k) & 1;  // cells 2q + pk
  const int4 n03 = *reinterpret_cast<const int4 *>(e), n47 = *reinterpret_cast<const int4 *>(e + 4);
  const int info = n47.z, b = n47.w;
  const long cb = (long)b * NC, fb = (long)b * t.nfb;
  if (L.stc && block_off(L, b)) return;
  const float *u = uniform_of(c, b);
  const bool U = u != nullptr;
  const float dv = geom(c, b, 6);
  const float T0 = U ? u[0] : 0.f, T1 = U ? u[1] : 0.f, T2 = U ? u[2] : 0.f;
  struct Row {
    float4 a, b;
    __device__ __forceinline__ float at(int q, int odd) const {  // cell 2q + odd
      return q == 0 ? (odd ? a.y : a.x) : q == 1 ? (odd ? a.w : a.z) : q == 2 ? (odd ? b.y : b.x) : (odd ? b.w : b.z);
    }
  };
  auto load = [](const float *p) { return Row{reinterpret_cast<const float4 *>(p)[0], reinterpret_cast<const float4 *>(p)[1]}; };
  // row (jj, kk) of block n, prolonged from its parent pw (parent * 8 + child);
  // fluid: every cell of n is
  auto row_of = [&](long n, int pw, bool fluid, int jj, int kk) {
    if constexpr (PROLONG) {
      const int wc = pw & 7;
      const float4 q = *reinterpret_cast<const float4 *>(phi + (long)(pw >> 3) * NC + 4 * (wc & 1) +
                                                          NB * (4 * ((wc >> 1) & 1) + (jj >> 1) +
                                                                NB * (4 * ((wc >> 2) & 1) + (kk >> 1))));
      Row r{make_float4(q.x, q.x, q.y, q.y), make_float4(q.z, q.z, q.w, q.w)};
      if (!fluid) {
        const Row m = load(c.vf + n * NC + NB * (jj + NB * kk));
        if (!(m.a.x > 0.f)) r.a.x = 0.f;
        if (!(m.a.y > 0.f)) r.a.y = 0.f;
        if (!(m.a.z > 0.f)) r.a.z = 0.f;
        if (!(m.a.w > 0.f)) r.a.w = 0.f;
        if (!(m.b.x > 0.f)) r.b.x = 0.f;
        if (!(m.b.y > 0.f)) r.b.y = 0.f;
        if (!(m.b.z > 0.f)) r.b.z = 0.f;
        if (!(m.b.w > 0.f)) r.b.w = 0.f;
      }
      return r;
    } else {
      return load(phi + n * NC + NB * (jj + NB * kk));
    }
  };
  const int pw = PROLONG ? e[kHXPar + 6] : 0;
  const Row own = row_of(b, pw, U, j, k), rr = load(rhs + cb + NB * tid);
  Row vf{make_float4(1.f, 1.f, 1.f, 1.f), make_float4(1.f, 1.f, 1.f, 1.f)};
  if (!U) vf = load(c.vf + cb + NB * tid);
  const int nbr[6] = {n03.x, n03.y, n03.z, n03.w, n47.x, n47.y};
  Row4 s;
#pragma unroll
  for (int q = 0; q < 4; q++) s.g[q] = c.alpha * dv, s.o[q] = 0.f;
  // x faces
#pragma unroll
  for (int f = 0; f < 2; f++) {
    const float *fx = c.tff[0] + fb + (NB + 1) * tid + f;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const bool edge = f == 0 ? q == 0 && pk == 0 : q == 3 && pk == 1;
      const float T = U ? T0 : fx[2 * q + pk];
      if (!edge) {
        // left: cell 2q + pk - 1, right: 2q + pk + 1, both of the other colour
        const float v = f == 0 ? (pk ? own.at(q, 0) : own.at(q > 0 ? q - 1 : 0, 1)) : (pk ? own.at(q < 3 ? q + 1 : 3, 0) : own.at(q, 1));
        s.g[q] += T;
        s.o[q] = fma_t(T, v, s.o[q]);
        continue;
      }
      const int ty = (info >> (2 * f)) & 3, across = f ? 0 : NB - 1;
      if (ty == 0) {
        float v;
        if constexpr (PROLONG) {
          const int ijk[3] = {across, j, k};
          v = prolonged_value<float, 3>(t, c, nbr[f], ijk, phi, e[kHXPar + f]);
        } else {
          v = phi[(long)nbr[f] * NC + NB * tid + across];
        }
        s.g[q] += T;
        s.o[q] = fma_t(T, v, s.o[q]);
      } else if (ty == 1) {
        if (t.bc_type[b * 6 + f] != kBCNeumann) s.g[q] += T * 2.0f;
      } else {
        Row4 one;
        one.g[0] = s.g[q], one.o[0] = s.o[q];
        one = rows8_cross<1>(c.cf, phi, e, f, j, k, one);
        s.g[q] = one.g[0], s.o[q] = one.o[0];
      }
    }
  }
  // y and z faces: the row across, cells at the same places
#pragma unroll
  for (int f = 2; f < 6; f++) {
    const int d = f >> 1, side = f & 1, at = d == 1 ? j : k;
    const bool edge = side ? at == NB - 1 : at == 0;
    const int ty = edge ? (info >> (2 * f)) & 3 : 0;
    if (ty >= 2) {
      s = rows8_cross<4>(c.cf, phi, e, f, pk, d == 1 ? k : j, s);
      continue;
    }
    float T[4];
    if (U) {
#pragma unroll
      for (int q = 0; q < 4; q++) T[q] = d == 1 ? T1 : T2;
    } else {
      const Row w = load(c.tff[d] + fb + (d == 1 ? NB * (j + side + (NB + 1) * k) : NB * (j + NB * (k + side))));
#pragma unroll
      for (int q = 0; q < 4; q++) T[q] = pk ? w.at(q, 1) : w.at(q, 0);
    }
    if (ty == 1) {
      if (t.bc_type[b * 6 + f] != kBCNeumann) {
#pragma unroll
        for (int q = 0; q < 4; q++) s.g[q] += T[q] * 2.0f;
      }
      continue;
    }
    const int to = edge ? (side ? 0 : NB - 1) : (side ? at + 1 : at - 1);
    const Row v = row_of(edge ? nbr[f] : b, PROLONG ? (edge ? e[kHXPar + f] : pw) : 0, U && !edge, d == 1 ? to : j,
                         d == 1 ? k : to);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      s.g[q] += T[q];
      s.o[q] = fma_t(T[q], pk ? v.at(q, 1) : v.at(q, 0), s.o[q]);
    }
  }
  float n[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const float r = pk ? rr.at(q, 1) : rr.at(q, 0), w = pk ? vf.at(q, 1) : vf.at(q, 0);
    const float old = pk ? own.at(q, 1) : own.at(q, 0);
    n[q] = (w > 0.f && s.g[q] > 0.f) ? relax(c.omega, fast_div(fma_t(r * dv, w, s.o[q]), s.g[q]), old) : 0.f;
  }
  // the other colour's cells with the values that concurrent readers see anyway
  float4 *dst = reinterpret_cast<float4 *>(phi + cb + NB * tid);
  dst[0] = pk ? make_float4(own.a.x, n[0], own.a.z, n[1]) : make_float4(n[0], own.a.y, n[1], own.a.w);
  dst[1] = pk ? make_float4(own.b.x, n[2], own.b.z, n[3]) : make_float4(n[2], own.b.y, n[3], own.b.w);
}

template <int MINB>
__global__ void __launch_bounds__(64, MINB) k_rbgs_rows8(Topo t, Coef<float> c, BlockList L, int color,
                                                         float *__restrict__ phi, const float *__restrict__ rhs,
                                                         const int *guard) {
  pdl_enter();
  if (guard && *guard) return;
  const ListRange lr = list_range(L);
  for (int p = lr.a + blockIdx.x; p < lr.b; p += gridDim.x)
    rows8_sweep<false>(t, c, L, L.hx + (long)p * kHX, color, phi, rhs);
}
__global__ void __launch_bounds__(64, 12) k_prolong_red_rows8(Topo t, Coef<float> c, BlockList L,
                                                              float *__restrict__ phi, const float *__restrict__ rhs,
                                                              const int *guard, BlockList X) {
  pdl_enter();
  if (guard && *guard) return;
  const ListRange lr = list_range(L), xr = list_range(X);
  const int nl = lr.b - lr.a, nx = xr.b - xr.a;
  for (int p = blockIdx.x; p < nl + nx; p += gridDim.x) {
    if (p < nl)
      rows8_sweep<true>(t, c, L, L.hx + (long)(lr.a + p) * kHX, 0, phi, rhs);
    else
      rows8_sweep<false>(t, c, X, X.hx + (long)(xr.a + p - nl) * kHX, 0, phi, rhs);
  }
}

__device__ __forceinline__ bool same_bits(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b);
}
__device__ __forceinline__ bool same_bits(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }

// ---------------------------------------------------------------------------
// volume-weighted restriction onto the non-leaf blocks of a level:
// coarse = avg(fine*vf_fine)/vf_coarse (src/SayakaMacIB.cpp:157-232 with
// src/SayakaInterpPatch.cpp:398-444)
template <typename T, int ND>
__global__ void __launch_bounds__(kThreads) k_restrict(Topo t, Coef<T> c, BlockList L, T *__restrict__ phi,
                                                       const int *guard) {
  pdl_enter();
  if (guard && *guard) return;
  const int ncell = t.ncell;
  const long total = (long)list_count(L) * ncell;
  for (long it = blockIdx.x * (long)blockDim.x + threadIdx.x; it < total; it += (long)gridDim.x * blockDim.x) {
    const int p = (int)(it / ncell);
    if (block_off(L, L.blocks[p])) continue;
    restrict_cell<T, ND>(t, c, L.blocks[p], (int)(it - (long)p * ncell), phi, L.links ? L.links + (long)p * 8 : nullptr);
  }
}

// the same with two coarse cells next to each other along x per thread, whose
// fine rows of four cells it loads at once (blocks' sides a multiple of four).
// A factor vf = 1 is not multiplied or divided by (the same bits; in FP64 the
// division alone is half of the kernel's FP64 work), and where a block's record
// says that all its cells have vf = 1 it isn't read.  Bound by bytes on large
// levels, where it is used (launch_restrict): 128 problems, FP32, 1.2 million
// cells, 25.7 us a launch with one cell per thread, 18.3 with two; 32 problems,
// FP64, 552 thousand cells, 27.7 and 23.4.
template <typename T>
struct alignas(16) Quad {
  T v[4];
};
template <typename T, int ND>
__global__ void __launch_bounds__(kThreads) k_restrict_pairs(Topo t, Coef<T> c, BlockList L, T *__restrict__ phi,
                                                             const int *guard) {
  pdl_enter();
  if (guard && *guard) return;
  const int nb = t.nb, half = nb >> 1, pairs = t.ncell >> 1, sh = t.lnb >= 0 ? ND * t.lnb - 1 : -1;
  const long total = (long)list_count(L) * pairs;
  const T wgt = (T)1.0 / (T)(1 << ND);
  for (long it = blockIdx.x * (long)blockDim.x + threadIdx.x; it < total; it += (long)gridDim.x * blockDim.x) {
    const int p = sh >= 0 ? (int)(it >> sh) : (int)(it / pairs);
    const int ci = 2 * (int)(it - (long)p * pairs), b = L.blocks[p];
    int ijk[3];
    if (t.lnb >= 0) {
      ijk[0] = ci & (nb - 1);
      ijk[1] = (ci >> t.lnb) & (nb - 1);
      ijk[2] = ND == 3 ? ci >> (2 * t.lnb) : 0;
    } else {
      decode<ND>(ci, nb, ijk);
    }
    int cidx = 0, f0 = 0, stride = 1;
#pragma unroll
    for (int q = 0; q < ND; q++) {
      const int sq = ijk[q] >= half ? 1 : 0;
      cidx |= sq << q;
      f0 += 2 * (ijk[q] - sq * half) * stride;
      stride *= nb;
    }
    const int F = L.links ? L.links[(long)p * 8 + cidx] : t.child[b * 8 + cidx];
    if (block_off(L, b)) continue;
    const long fine = (long)F * t.ncell + f0, coarse = (long)b * t.ncell + ci;
    constexpr int R = ND == 3 ? 4 : 2;
    Quad<T> x[R];
#pragma unroll
    for (int r = 0; r < R; r++)
      x[r] = *reinterpret_cast<const Quad<T> *>(phi + fine + (r & 1) * nb + (r >> 1) * nb * nb);
    const T one = (T)1;
    if (!uniform_of(c, F)) {
#pragma unroll
      for (int r = 0; r < R; r++) {
        const Quad<T> w = *reinterpret_cast<const Quad<T> *>(c.vf + fine + (r & 1) * nb + (r >> 1) * nb * nb);
        bool fluid = true;
#pragma unroll
        for (int q = 0; q < 4; q++) fluid = fluid && same_bits(w.v[q], one);
        if (!fluid) {
#pragma unroll
          for (int q = 0; q < 4; q++) x[r].v[q] = x[r].v[q] * w.v[q];
        }
      }
    }
    T vc[2] = {one, one};
    if (!uniform_of(c, b)) vc[0] = c.vf[coarse], vc[1] = c.vf[coarse + 1];
    const bool fluid = same_bits(vc[0], one) && same_bits(vc[1], one);
    T out[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      T sum = 0;
#pragma unroll
      for (int r = 0; r < R; r++) {
        sum += x[r].v[2 * k];
        sum += x[r].v[2 * k + 1];
      }
      out[k] = sum * wgt;
    }
    if (!fluid) {
#pragma unroll
      for (int k = 0; k < 2; k++) out[k] = vc[k] > 0 ? out[k] / vc[k] : (T)0;
    }
    phi[coarse] = out[0];
    phi[coarse + 1] = out[1];
  }
}

// masked injection onto every block of a level (src/SayakaMacIB.cpp:234-283)
template <typename T, int ND>
__global__ void __launch_bounds__(kThreads) k_prolong(Topo t, Coef<T> c, BlockList L, T *__restrict__ phi,
                                                      const int *guard) {
  pdl_enter();
  if (guard && *guard) return;
  const int ncell = t.ncell;
  const long total = (long)list_count(L) * ncell;
  for (long it = blockIdx.x * (long)blockDim.x + threadIdx.x; it < total; it += (long)gridDim.x * blockDim.x) {
    const int p = (int)(it / ncell);
    if (block_off(L, L.blocks[p])) continue;
    prolong_cell<T, ND>(t, c, L.blocks[p], (int)(it - (long)p * ncell), phi, L.links ? L.links[p] : -1);
  }
}

// same-level face coefficient ((beta*ds)/dx)*B*a for every face of every block
template <typename T>
__global__ void __launch_bounds__(kThreads) k_face_coef(Topo t, const double *geom64, const T *b0, const T *b1, const T *b2, const T *a0,
                            const T *a1, const T *a2, double beta, T *t0, T *t1, T *t2) {
  // One warp per block and direction divides once for all its faces (a
  // division is about 20 operations of the FP64 pipe, whatever the number of
  // lanes that need it), and a product with 1 is not formed: B and the area
  // fraction are 1 on most faces.  13.75 M cells: 1050 us with a
  // division per face, 587 with one per thread of a CTA, 262 now.
  const int lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
  for (long it = (blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5; it < (long)t.nblocks * t.ndim; it += warps) {
    const int b = (int)(it / t.ndim), d = (int)(it - (long)b * t.ndim);
    const T *B = d == 0 ? b0 : (d == 1 ? b1 : b2);
    const T *A = d == 0 ? a0 : (d == 1 ? a1 : a2);
    T *O = d == 0 ? t0 : (d == 1 ? t1 : t2);
    const T ds = (T)geom64[b * 8 + 3 + d], dx = (T)geom64[b * 8 + d];
    const T q = (T)beta * ds / dx;
    const long fb = (long)b * t.nfb;
    for (int i = lane; i < t.nfb; i += 32) {
      const T bv = B[fb + i], av = A[fb + i];
      T v = q;
      if (!same_bits(bv, (T)1)) v = v * bv;
      if (!same_bits(av, (T)1)) v = v * av;
      O[fb + i] = v;
    }
  }
}

// face flux -(phi_hi - phi_lo)/h on every face of direction `dir` of a tower
// (src/SayakaMacOperator.cpp:161-239 and :929-1025): FINE_BC faces get 0,
// FINE_CRSE faces use h = 1.5 dx with the injected coarse ghost, CRSE_FINE
// faces the average of the fine FINE_CRSE fluxes behind them (FLUX_SYNC_AVG).
template <int ND>
__global__ void k_flux(Topo t, Coef<double> c, BlockList L, int dir, const double *__restrict__ phi,
                       double *__restrict__ flux) {
  const int nb = t.nb, ncell = t.ncell, nfb = t.nfb;
  const long total = (long)L.n * nfb;
  for (long it = blockIdx.x * (long)blockDim.x + threadIdx.x; it < total; it += (long)gridDim.x * blockDim.x) {
    const int p = (int)(it / nfb);
    const int fxi = (int)(it - (long)p * nfb);
    const int *hxe = L.hx ? L.hx + (long)p * kHX : nullptr;
    const int b = hxe ? hxe[kHXBlock] : L.blocks[p];
    const uint16_t ft = hxe ? (uint16_t)(hxe[kHXInfo] & 0xffff) : L.ftypes[p];
    // decode the face-centred index: dimension dir has nb+1 entries
    const int e0 = nb + (dir == 0), e1 = nb + (dir == 1);
    int fi[3];
    fi[0] = fxi % e0;
    fi[1] = ND >= 2 ? (fxi / e0) % e1 : 0;
    fi[2] = ND == 3 ? fxi / (e0 * e1) : 0;
    const int m = fi[dir];
    const double dh = c.geom[b * 8 + dir];
    const long cb = (long)b * ncell;
    double out;
    if (m > 0 && m < nb) {
      int hi[3] = {fi[0], fi[1], fi[2]}, lo[3] = {fi[0], fi[1], fi[2]};
      lo[dir] = m - 1;
      out = -(phi[cb + encode(hi, nb)] - phi[cb + encode(lo, nb)]) / dh;
    } else {
      const int s = m == 0 ? 0 : 1;
      const int f = 2 * dir + s;
      const int ty = face_type_of(ft, f);
      int own[3] = {fi[0], fi[1], fi[2]};
      own[dir] = s == 0 ? 0 : nb - 1;
      const double po = phi[cb + encode(own, nb)];
      if (ty == 1) {
        out = 0;
      } else if (ty == 0) {
        const double g = same_level_ghost(t, b, f, own, phi);
        out = s == 0 ? -(po - g) / dh : -(g - po) / dh;
      } else if (ty == 2) {
        const double g = fine_crse_ghost<double, ND>(t, b, f, own, phi);
        const double h = dh * 1.5;
        out = s == 0 ? -(po - g) / h : -(g - po) / h;
      } else {
        // average of the fine FINE_CRSE fluxes on this face
        const int N = t.neighbor[b * 6 + f];
        const int half = nb >> 1;
        int cidx = (1 - s) << dir, base[3] = {0, 0, 0}, tq[2] = {0, 0}, nt = 0;
        for (int q = 0; q < ND; q++) {
          if (q == dir) continue;
          const int sq = own[q] >= half ? 1 : 0;
          cidx |= sq << q;
          base[q] = 2 * (own[q] - sq * half);
          tq[nt++] = q;
        }
        const int F = t.child[N * 8 + cidx];
        const double dhf = c.geom[F * 8 + dir] * 1.5;
        int fc[3];
        fc[dir] = s == 1 ? 0 : nb - 1;
        double sum = 0;
        for (int a1 = 0; a1 < (ND == 3 ? 2 : 1); a1++)
          for (int a0 = 0; a0 < 2; a0++) {
            fc[tq[0]] = base[tq[0]] + a0;
            if (ND == 3) fc[tq[1]] = base[tq[1]] + a1;
            if (ND == 2) fc[2] = 0;
            const double pf = phi[(long)F * ncell + encode(fc, nb)];
            // the fine block's ghost toward b is b's boundary cell `own`
            const double fl = s == 1 ? -(pf - po) / dhf : -(po - pf) / dhf;
            sum += fl;
          }
        out = sum * (ND == 3 ? 0.25 : 0.5);
      }
    }
    flux[(long)b * nfb + fxi] = out;
  }
}

// Dirichlet / SimpleFill lift of the right-hand side from BC values held in
// the ghost layer of phi (src/SayakaMacOperator.cpp:1470-1594)
template <int ND>
__global__ void k_fix_bc(Topo t, Coef<double> c, BlockList L, const double *__restrict__ phig, int ng,
                         double *__restrict__ rhs) {
  const int nb = t.nb, ncell = t.ncell;
  const int G = nb + 2 * ng;
  const long gstride = ND == 3 ? (long)G * G * G : (long)G * G;
  const long total = (long)L.n * ncell;
  for (long it = blockIdx.x * (long)blockDim.x + threadIdx.x; it < total; it += (long)gridDim.x * blockDim.x) {
    const int p = (int)(it / ncell);
    const int ci = (int)(it - (long)p * ncell);
    const int *hxe = L.hx ? L.hx + (long)p * kHX : nullptr;
    const int b = hxe ? hxe[kHXBlock] : L.blocks[p];
    const uint16_t ft = hxe ? (uint16_t)(hxe[kHXInfo] & 0xffff) : L.ftypes[p];
    int ijk[3];
    decode<ND>(ci, nb, ijk);
    const double dv = c.geom[b * 8 + 6];
    const long q = (long)b * ncell + ci;
    double r = rhs[q];
    for (int f = 0; f < 2 * ND; f++) {
      if (face_type_of(ft, f) != 1) continue;
      const int d = f >> 1, s = f & 1;
      if (ijk[d] != (s ? nb - 1 : 0)) continue;
      const int bct = t.bc_type[b * 6 + f];
      auto gidx = [&](int i, int j, int k) {
        return (long)b * gstride + (i + ng) + (long)G * ((j + ng) + (long)G * (ND == 3 ? k + ng : 0));
      };
      const double p0 = phig[gidx(ijk[0], ijk[1], ijk[2])];
      int gi[3] = {ijk[0], ijk[1], ijk[2]};
      gi[d] += s ? 1 : -1;
      const double p1 = phig[gidx(gi[0], gi[1], gi[2])];
      const int fx = face_index(d, ijk, s, nb);
      double coef = c.beta * c.geom[b * 8 + 3 + d] / c.geom[b * 8 + d];
      coef *= c.bcoef[d][(long)b * t.nfb + fx];
      coef *= c.afrac[d][(long)b * t.nfb + fx];
      double corr = 0;
      if (bct == kBCDirichlet) {
        const double pbc = 0.5 * (p0 + p1);
        corr = pbc * 2.0 * coef;
      } else if (bct == kBCSimpleFill) {
        const double pbc = p1;
        corr = pbc * 2.0 * coef;
      }
      const double vfv = c.vf[q];
      if (vfv > 0) {
        corr /= (dv * vfv);
        r += corr;
      }
    }
    rhs[q] = r;
  }
}

inline int grid_for(long work) {
  long g = (work + kThreads - 1) / kThreads;
  if (g < 1) g = 1;
  if (g > 152 * 32) g = 152 * 32;
  return (int)g;
}

}  // namespace

template <typename T>
void launch_face_coef(const Topo &t, const double *geom64, const T *bcoef[3], const T *afrac[3], double beta,
                      T *tff[3], cudaStream_t s) {
  const long rows = (long)t.nblocks * t.ndim;
  if (rows == 0 || t.nfb == 0) return;
  k_face_coef<T><<<grid_for(rows * 32), kThreads, 0, s>>>(t, geom64, bcoef[0], bcoef[1], bcoef[2], afrac[0], afrac[1],
                                                          afrac[2], beta, tff[0], tff[1], tff[2]);
}

template <typename T>
void launch_apply(const Topo &t, const Coef<T> &c, const BlockList &L, const T *x, T *y, const T *rhs,
                  const int *guard, cudaStream_t s, bool pdl) {
  const long work = (long)L.n * t.ncell;
  if (work == 0) return;
  if (t.ndim == 2)
    launch_k(pdl, k_apply<T, 2>, grid_for(work), kThreads, 0, s, t, c, L, x, y, rhs, guard);
  else
    launch_k(pdl, k_apply<T, 3>, grid_for(work), kThreads, 0, s, t, c, L, x, y, rhs, guard);
}

// The same sweep with the block staged in shared memory: one CTA per block
// of the list loads the block's phi tile (full sectors) and, once per
// boundary face cell of the sweep's colour, the face's contribution
// (diagonal part hc, off-diagonal factor hk and value hv: FINE_FINE and
// FINE_CRSE give T and the gathered ghost, CRSE_FINE the coarse-side T, 1 and
// the fine-side sum, physical faces 0 or 2T and 0); cells then read their
// neighbours from the tile.  Every value is combined in smooth_cell_fast's
// order with the same operations, so the result is bit-identical.  The tile
// (both colours, black cells unchanged) is written back whole.
template <typename T, int ND, int MINB>
__global__ void __launch_bounds__(kThreads, MINB) k_rbgs_tile(Topo t, Coef<T> c, BlockList L, int color,
                                                              T *__restrict__ phi, const T *__restrict__ rhs,
                                                              const int *guard) {
  extern __shared__ __align__(16) unsigned char rbgs_smem[];
  pdl_enter();
  if (guard && *guard) return;
  const int nb = t.nb, ncell = t.ncell, nhalf = ncell >> 1;
  const int nface = ND == 3 ? nb * nb : nb;  // cells on one block face
  T *tile = reinterpret_cast<T *>(rbgs_smem);
  T *hc = tile + ncell;
  T *hk = hc + 2 * ND * nface;
  T *hv = hk + 2 * ND * nface;
  const ListRange lr = list_range(L);
  for (int p = lr.a + blockIdx.x; p < lr.b; p += gridDim.x) {
    const int *hxe = L.hx ? L.hx + (long)p * kHX : nullptr;
    const int b = hxe ? hxe[kHXBlock] : L.blocks[p];
    if (block_off(L, b)) continue;  // uniform over the CTA
    const long f0 = factor_entry(L, p) * ncell;
    const uint16_t ft = hxe ? (uint16_t)(hxe[kHXInfo] & 0xffff) : L.ftypes[p];
    const long cb = (long)b * ncell;
    const long fb = (long)b * t.nfb;
    if ((ncell & 3) == 0 && sizeof(T) == 4) {
      const float4 *src = reinterpret_cast<const float4 *>(phi + cb);
      float4 *dst = reinterpret_cast<float4 *>(tile);
      for (int i = threadIdx.x; i < (ncell >> 2); i += blockDim.x) dst[i] = src[i];
    } else {
      for (int i = threadIdx.x; i < ncell; i += blockDim.x) tile[i] = phi[cb + i];
    }
    // boundary contributions of the cells of this colour
    for (int e = threadIdx.x; e < 2 * ND * nface; e += blockDim.x) {
      const int f = e / nface, m = e - f * nface;
      const int d = f >> 1, s = f & 1;
      int ijk[3];
      ijk[d] = s ? nb - 1 : 0;
      const int q0 = d == 0 ? 1 : 0, q1 = d == 2 ? 1 : 2;
      ijk[q0] = m % nb;
      if (ND == 3) ijk[q1] = m / nb;
      else if (d != 2) ijk[2] = 0;
      if (ND == 2) ijk[2] = 0;
      if (((ijk[0] + ijk[1] + ijk[2]) & 1) != color) continue;
      int fx;
      if (d == 0)
        fx = ijk[0] + s + (nb + 1) * (ijk[1] + nb * ijk[2]);
      else if (d == 1)
        fx = ijk[0] + nb * (ijk[1] + s + (nb + 1) * ijk[2]);
      else
        fx = encode(ijk, nb) + s * nb * nb;
      const int ty = face_type_of(ft, f);
      const T *u = uniform_of(c, b);
      T vc = 0, vk = 0, vv = 0;
      if (ty == 0) {
        vc = vk = u ? u[d] : c.tff[d][fb + fx];
        vv = same_level_ghost<T, false>(t, b, f, ijk, phi, hxe);
      } else if (ty == 1) {
        if (t.bc_type[b * 6 + f] != kBCNeumann) vc = (u ? u[d] : c.tff[d][fb + fx]) * (T)2.0;
      } else if (ty == 2) {
        vc = vk = cf_face<T, ND>(c, t, b, f, ijk);
        vv = fine_crse_ghost<T, ND, false>(t, b, f, ijk, phi, hxe);
      } else {
        vc = cf_face<T, ND>(c, t, b, f, ijk);
        vk = (T)1;
        vv = refined_sum<T, ND, false>(t, c, b, f, ijk, phi, hxe);
      }
      hc[e] = vc;
      hk[e] = vk;
      hv[e] = vv;
    }
    __syncthreads();
    const T dv = geom(c, b, 6);
    const T *u = uniform_of(c, b);  // constant coefficients: no face or vf loads
    // a cell's global operands (face coefficients, rhs and vf or the FP64
    // factors) are gathered before any update: a thread with two cells has
    // both cells' loads in flight together (the shared-memory tile written
    // by the updates may alias the operand pointers for the compiler)
    struct Ops {
      int ijk[3], ci;
      T coef[2 * ND], r, v;
      double sa, ia;
    };
    auto gather = [&](int h, Ops &o) {
      color_cell_fast<ND>(h, t, color, o.ijk);
      o.ci = t.lnb >= 0 ? o.ijk[0] + ((o.ijk[1] + (o.ijk[2] << t.lnb)) << t.lnb) : encode(o.ijk, nb);
#pragma unroll
      for (int f = 0; f < 2 * ND; f++) {
        const int d = f >> 1, s = f & 1;
        const bool bnd = s ? o.ijk[d] == nb - 1 : o.ijk[d] == 0;
        int fx;
        if (d == 0)
          fx = o.ijk[0] + s + (nb + 1) * (o.ijk[1] + nb * o.ijk[2]);
        else if (d == 1)
          fx = o.ijk[0] + nb * (o.ijk[1] + s + (nb + 1) * o.ijk[2]);
        else
          fx = o.ci + s * nb * nb;
        o.coef[f] = bnd ? (T)0 : (u ? u[d] : c.tff[d][fb + fx]);
      }
      o.r = rhs[cb + o.ci];
      if (sizeof(T) == 8 && L.sa) {
        bool inner = true;
#pragma unroll
        for (int q = 0; q < ND; q++) inner = inner && o.ijk[q] > 0 && o.ijk[q] < nb - 1;
        if (u && inner) {
          o.sa = u[6];
          o.ia = u[7];
        } else {
          const long fo = f0 + o.ci;
          o.sa = L.sa[fo];
          o.ia = L.ia[fo];
        }
        o.v = 0;
      } else {
        o.v = u ? (T)1 : c.vf[cb + o.ci];
        o.sa = o.ia = 0.0;
      }
    };
    auto update = [&](const Ops &o) {
      T diag = c.alpha * dv;
      T off = 0;
#pragma unroll
      for (int f = 0; f < 2 * ND; f++) {
        const int d = f >> 1, s = f & 1;
        const bool bnd = s ? o.ijk[d] == nb - 1 : o.ijk[d] == 0;
        if (!bnd) {
          const int stride = d == 0 ? 1 : (d == 1 ? nb : nb * nb);
          diag += o.coef[f];
          off = fma_t(o.coef[f], tile[o.ci + (s ? stride : -stride)], off);
        } else {
          const int q0 = d == 0 ? 1 : 0, q1 = d == 2 ? 1 : 2;
          const int m = o.ijk[q0] + (ND == 3 ? nb * o.ijk[q1] : 0);
          const int e = f * nface + m;
          diag += hc[e];
          off = fma_t(hk[e], hv[e], off);
        }
      }
      T unew = 0;
      if (sizeof(T) == 8 && L.sa) {
        unew = fma_t(o.r, (T)o.sa, off * (T)o.ia);
        if (o.ia != 0) unew = relax(c.omega, unew, tile[o.ci]);
      } else {
        if (o.v > 0 && diag > 0) unew = relax(c.omega, fast_div(fma_t(o.r * dv, o.v, off), diag), tile[o.ci]);
      }
      tile[o.ci] = unew;
    };
    for (int h = threadIdx.x; h < nhalf; h += 2 * blockDim.x) {
      const int h2 = h + blockDim.x;
      Ops o1, o2;
      gather(h, o1);
      if (h2 < nhalf) gather(h2, o2);
      update(o1);
      if (h2 < nhalf) update(o2);
    }
    __syncthreads();
    if ((ncell & 3) == 0 && sizeof(T) == 4) {
      const float4 *src = reinterpret_cast<const float4 *>(tile);
      float4 *dst = reinterpret_cast<float4 *>(phi + cb);
      for (int i = threadIdx.x; i < (ncell >> 2); i += blockDim.x) dst[i] = src[i];
    } else {
      for (int i = threadIdx.x; i < ncell; i += blockDim.x) phi[cb + i] = tile[i];
    }
    __syncthreads();
  }
}

// ---- Block-hybrid Gauss-Seidel: one pass over every block of a list (all
// sublevels of a tower at once).  Each CTA loads its block's tile from src,
// takes every value outside the block from src too (frozen for the pass:
// Jacobi between blocks), runs nsweep red-black sweeps on the tile in shared
// memory and writes the tile to dst.  src is not written during the pass, so
// the result does not depend on the order in which CTAs run: the pass is one
// fixed linear map, like the sweeps it replaces, but it moves a block's data
// once for nsweep sweeps and needs one launch per pass instead of one per
// colour, level parity and sweep.  The boundary faces are evaluated as in
// smooth_cell_fast (same-level, coarse/fine and physical faces).
template <typename T, int ND, int MINB>
__global__ void __launch_bounds__(kThreads, MINB) k_bhgs(Topo t, Coef<T> c, BlockList L, int nsweep,
                                                         const T *__restrict__ src, T *__restrict__ dst,
                                                         const T *__restrict__ rhs, const int *guard) {
  extern __shared__ __align__(16) unsigned char bhgs_smem[];
  pdl_enter();
  if (guard && *guard) return;
  const int nb = t.nb, ncell = t.ncell, nhalf = ncell >> 1;
  const int nface = ND == 3 ? nb * nb : nb;  // cells on one block face
  T *tile = reinterpret_cast<T *>(bhgs_smem);
  T *hc = tile + ncell;            // diagonal part of every boundary face of the block
  T *ho = hc + 2 * ND * nface;     // its off-diagonal part (frozen neighbour values)
  const ListRange lr = list_range(L);
  for (int p = lr.a + blockIdx.x; p < lr.b; p += gridDim.x) {
    const int *hxe = L.hx ? L.hx + (long)p * kHX : nullptr;
    const int b = hxe ? hxe[kHXBlock] : L.blocks[p];
    if (block_off(L, b)) continue;  // uniform over the CTA
    const long f0 = factor_entry(L, p) * ncell;
    const uint16_t ft = hxe ? (uint16_t)(hxe[kHXInfo] & 0xffff) : L.ftypes[p];
    const long cb = (long)b * ncell;
    const long fb = (long)b * t.nfb;
    if ((ncell & 3) == 0 && sizeof(T) == 4) {
      const float4 *s4 = reinterpret_cast<const float4 *>(src + cb);
      float4 *d4 = reinterpret_cast<float4 *>(tile);
      for (int i = threadIdx.x; i < (ncell >> 2); i += blockDim.x) d4[i] = s4[i];
    } else {
      for (int i = threadIdx.x; i < ncell; i += blockDim.x) tile[i] = src[cb + i];
    }
    for (int e = threadIdx.x; e < 2 * ND * nface; e += blockDim.x) {
      const int f = e / nface, m = e - f * nface;
      const int d = f >> 1, s = f & 1;
      int ijk[3] = {0, 0, 0};
      ijk[d] = s ? nb - 1 : 0;
      const int q0 = d == 0 ? 1 : 0, q1 = d == 2 ? 1 : 2;
      ijk[q0] = m % nb;
      if (ND == 3) ijk[q1] = m / nb;
      int fx;
      if (d == 0)
        fx = ijk[0] + s + (nb + 1) * (ijk[1] + nb * ijk[2]);
      else if (d == 1)
        fx = ijk[0] + nb * (ijk[1] + s + (nb + 1) * ijk[2]);
      else
        fx = encode(ijk, nb) + s * nb * nb;
      const int ty = face_type_of(ft, f);
      const T *u = uniform_of(c, b);
      T vc = 0, vo = 0;
      if (ty == 0) {
        vc = u ? u[d] : c.tff[d][fb + fx];
        vo = vc * same_level_ghost<T, false>(t, b, f, ijk, src, hxe);
      } else if (ty == 1) {
        if (t.bc_type[b * 6 + f] != kBCNeumann) vc = (u ? u[d] : c.tff[d][fb + fx]) * (T)2.0;
      } else if (ty == 2) {
        vc = cf_face<T, ND>(c, t, b, f, ijk);
        vo = vc * fine_crse_ghost<T, ND, false>(t, b, f, ijk, src, hxe);
      } else {
        vc = cf_face<T, ND>(c, t, b, f, ijk);
        vo = refined_sum<T, ND, false>(t, c, b, f, ijk, src, hxe);
      }
      hc[e] = vc;
      ho[e] = vo;
    }
    __syncthreads();
    const T dv = geom(c, b, 6);
    const T *u = uniform_of(c, b);  // constant coefficients: no face or vf loads
    for (int sw = 0; sw < nsweep; sw++) {
      for (int color = 0; color < 2; color++) {
        for (int h = threadIdx.x; h < nhalf; h += blockDim.x) {
          int ijk[3];
          color_cell_fast<ND>(h, t, color, ijk);
          const int ci = t.lnb >= 0 ? ijk[0] + ((ijk[1] + (ijk[2] << t.lnb)) << t.lnb) : encode(ijk, nb);
          T diag = c.alpha * dv;
          T off = 0;
#pragma unroll
          for (int f = 0; f < 2 * ND; f++) {
            const int d = f >> 1, s = f & 1;
            const bool bnd = s ? ijk[d] == nb - 1 : ijk[d] == 0;
            if (!bnd) {
              int fx;
              if (d == 0)
                fx = ijk[0] + s + (nb + 1) * (ijk[1] + nb * ijk[2]);
              else if (d == 1)
                fx = ijk[0] + nb * (ijk[1] + s + (nb + 1) * ijk[2]);
              else
                fx = ci + s * nb * nb;
              const T coef = u ? u[d] : c.tff[d][fb + fx];
              const int stride = d == 0 ? 1 : (d == 1 ? nb : nb * nb);
              diag += coef;
              off = fma_t(coef, tile[ci + (s ? stride : -stride)], off);
            } else {
              const int qa = d == 0 ? 1 : 0, qb = d == 2 ? 1 : 2;
              const int e = f * nface + ijk[qa] + (ND == 3 ? nb * ijk[qb] : 0);
              diag += hc[e];
              off += ho[e];
            }
          }
          T unew = 0;
          if (sizeof(T) == 8 && L.sa) {
            bool inner = true;
#pragma unroll
            for (int q = 0; q < ND; q++) inner = inner && ijk[q] > 0 && ijk[q] < nb - 1;
            const long fo = f0 + ci;
            const bool ui = u && inner;
            const T iav = ui ? u[7] : (T)L.ia[fo];  // 0 in a solid cell
            unew = fma_t(rhs[cb + ci], ui ? u[6] : (T)L.sa[fo], off * iav);
            if (iav != (T)0) unew = relax(c.omega, unew, tile[ci]);
          } else {
            const T vfv = u ? (T)1 : c.vf[cb + ci];
            if (vfv > 0 && diag > 0) unew = relax(c.omega, fast_div(fma_t(rhs[cb + ci] * dv, vfv, off), diag), tile[ci]);
          }
          tile[ci] = unew;
        }
        __syncthreads();
      }
    }
    if ((ncell & 3) == 0 && sizeof(T) == 4) {
      const float4 *s4 = reinterpret_cast<const float4 *>(tile);
      float4 *d4 = reinterpret_cast<float4 *>(dst + cb);
      for (int i = threadIdx.x; i < (ncell >> 2); i += blockDim.x) d4[i] = s4[i];
    } else {
      for (int i = threadIdx.x; i < ncell; i += blockDim.x) dst[cb + i] = tile[i];
    }
    __syncthreads();
  }
}

// ---- The block-hybrid pass over 3D FP32 blocks of 16^3 or 8^3 cells --------
// One CTA per block, one thread per row of cells along x, which keeps the
// row's values, diagonal and right-hand side in registers, split by colour.
// The tile in shared memory is split by colour too (tile[colour][quarter]
// [row], a float4 of four cells of one colour): the cells of a row that a
// half sweep updates have their y and z neighbours at the same places of the
// adjoining rows' other-colour part, so a thread reads them 16 bytes at a
// time without bank conflicts, and its x neighbours are in its registers.
// Rows outside the block hold the frozen neighbours' parts (T value, rounded)
// and enter with factor 1, so no cell takes a branch.  The values and
// operations of k_bhgs in the same order: the same bits.
//
// k_bhgs spends about 80 instructions on an update (index arithmetic, six
// boundary tests, reloads from global memory) and this form about 16; its
// bound moves from issue towards the three streams of a pass (src, rhs, dst).
template <int NB>
struct H3 {
  static constexpr int kRows = (NB + 2) * (NB + 2), kQ = NB / 2, kH = NB / 8, kFace = NB * NB;
  float4 tile[2][kH][kRows];
  float hc[6][kFace];   // diagonal part of every boundary face cell
  float hox[2][kFace];  // frozen parts across the x faces
  static __device__ __forceinline__ int row(int j, int k) { return j + 1 + (NB + 2) * (k + 1); }
};

// Coefficients and volume fractions of a block without a record, staged once:
// read from global memory row by row, every load of a warp touches 32 lines,
// and a pass of one such block took 19 us.  y and z faces and volume fractions
// are split by the parity of their indices like the tile: the lower face of a
// cell of colour c is in part c of its own row, its upper face in part 1 - c
// of the next row, at the same place.
template <int NB>
struct H3Var {
  static constexpr int kH = NB / 8;
  float fx[NB * NB][NB + 1];
  float4 fy[2][kH][NB * (NB + 1)], fz[2][kH][NB * (NB + 1)], vf[2][kH][NB * NB];
};
// rows x NB values of src, row m split by the parity of i + par(m)
template <int NB, int ROWS, class Par>
__device__ __forceinline__ void h3_stage(const float *__restrict__ src, float4 (&dst)[2][NB / 8][ROWS], Par par) {
  const float4 *s4 = reinterpret_cast<const float4 *>(src);
#pragma unroll
  for (int n = threadIdx.x; n < ROWS * (NB / 4); n += NB * NB) {
    const float4 w = s4[n];
    const int row = n / (NB / 4), q = 2 * (n % (NB / 4)), pr = par(row) & 1;
    float2 *e2 = reinterpret_cast<float2 *>(&dst[0][q >> 2][row]) + ((q >> 1) & 1);
    float2 *o2 = reinterpret_cast<float2 *>(&dst[1][q >> 2][row]) + ((q >> 1) & 1);
    *e2 = pr ? make_float2(w.y, w.w) : make_float2(w.x, w.z);
    *o2 = pr ? make_float2(w.x, w.z) : make_float2(w.y, w.w);
  }
}

// the sweeps of one block: row (j, k) of thread (U: a constant-coefficient
// block, coefficients T[]; else from the face arrays).  The diagonal is not
// kept per cell: in a constant-coefficient block every cell of a row but its
// two ends has the same (a boundary face's part is one value per face there,
// coarse/fine faces included: k_uniform), elsewhere it is summed along with the
// off-diagonal from the same loads.  Two CTAs of a 16^3 block fit an SM: 28.9 KB
// of H3 and 68.6 KB of H3Var each, reserved for blocks with a record too.
template <int NB, bool U>
__device__ __forceinline__ void h3_sweeps(const Topo &t, const Coef<float> &c, int b, const float *u, float dv,
                                          int nsweep, const float4 (&r4)[NB / 4], H3<NB> &sh,
                                          const H3Var<NB> &sv) {
  constexpr int Q = NB / 2, H = NB / 8;
  const int j = threadIdx.x % NB, k = threadIdx.x / NB, pr = (j + k) & 1, m = threadIdx.x;
  const int r = H3<NB>::row(j, k);
  const float T0 = U ? u[0] : 0.f, T1 = U ? u[1] : 0.f, T2 = U ? u[2] : 0.f;
  const float *fx = sv.fx[m];
  const int ry = j + (NB + 1) * k;  // row of the y faces below; above: the next
  float v[2][Q], rd[2][Q];
  const float kd = j == 0 ? 1.f : T1, ku = j == NB - 1 ? 1.f : T1;
  const float kb = k == 0 ? 1.f : T2, kf = k == NB - 1 ? 1.f : T2;
  const float hl = sh.hox[0][m], hr = sh.hox[1][m], cl = sh.hc[0][m], cr = sh.hc[1][m];
  // diagonal of the row's first, inner and last cells (U)
  float g0 = 0.f, gm = 0.f, g1 = 0.f;
  if (U) {
    const float ad = c.alpha * dv;
    const float yd = j == 0 ? sh.hc[2][NB * k] : T1, yu = j == NB - 1 ? sh.hc[3][NB * k] : T1;
    const float zb = k == 0 ? sh.hc[4][NB * j] : T2, zf = k == NB - 1 ? sh.hc[5][NB * j] : T2;
    g0 = ad + cl, gm = ad + T0, g1 = ad + T0;
    g0 += T0, gm += T0, g1 += cr;
    g0 += yd, gm += yd, g1 += yd;
    g0 += yu, gm += yu, g1 += yu;
    g0 += zb, gm += zb, g1 += zb;
    g0 += zf, gm += zf, g1 += zf;
  }
#pragma unroll
  for (int q = 0; q < Q; q += 2) {
    const float4 w = r4[q / 2];
    rd[0][q] = (pr ? w.y : w.x) * dv;
    rd[1][q] = (pr ? w.x : w.y) * dv;
    rd[0][q + 1] = (pr ? w.w : w.z) * dv;
    rd[1][q + 1] = (pr ? w.z : w.w) * dv;
  }
#pragma unroll
  for (int col = 0; col < 2; col++)
#pragma unroll
    for (int h = 0; h < H; h++) {
      const float4 w = sh.tile[col][h][r];
      v[col][4 * h] = w.x, v[col][4 * h + 1] = w.y, v[col][4 * h + 2] = w.z, v[col][4 * h + 3] = w.w;
    }
  for (int sw = 0; sw < nsweep; sw++) {
#pragma unroll
    for (int col = 0; col < 2; col++) {
      const int pk = col ? 1 - pr : pr;
      const float(&o)[Q] = v[1 - col];
#pragma unroll
      for (int h = 0; h < H; h++) {
        const float4 d4 = sh.tile[1 - col][h][r - 1], u4 = sh.tile[1 - col][h][r + 1];
        const float4 b4 = sh.tile[1 - col][h][r - (NB + 2)], f4 = sh.tile[1 - col][h][r + (NB + 2)];
        const float vd[4] = {d4.x, d4.y, d4.z, d4.w}, vu[4] = {u4.x, u4.y, u4.z, u4.w};
        const float vb[4] = {b4.x, b4.y, b4.z, b4.w}, vz[4] = {f4.x, f4.y, f4.z, f4.w};
        float4 tdv, tuv, tbv, tfv, vfv;
        if (!U) {
          tdv = sv.fy[col][h][ry], tuv = sv.fy[1 - col][h][ry + 1];
          tbv = sv.fz[col][h][m], tfv = sv.fz[1 - col][h][m + NB];
          vfv = sv.vf[col][h][m];
        }
#pragma unroll
        for (int n = 0; n < 4; n++) {
          const int q = 4 * h + n, i = 2 * q + pk;
          const bool first = q == 0 && i == 0, last = q == Q - 1 && i == NB - 1;
          float vl = pk ? o[q] : (q > 0 ? o[q > 0 ? q - 1 : 0] : hl);
          float vr = pk ? (q < Q - 1 ? o[q < Q - 1 ? q + 1 : q] : hr) : o[q];
          float off = 0.f, g, w = 1.f;
          if (U) {
            g = first ? g0 : last ? g1 : gm;
            off = fma_t(first ? 1.f : T0, vl, off);
            off = fma_t(last ? 1.f : T0, vr, off);
            off = fma_t(kd, vd[n], off);
            off = fma_t(ku, vu[n], off);
            off = fma_t(kb, vb[n], off);
            off = fma_t(kf, vz[n], off);
          } else {
            const float tl = fx[i], tr = fx[i + 1];
            const float td = n == 0 ? tdv.x : n == 1 ? tdv.y : n == 2 ? tdv.z : tdv.w;
            const float tu = n == 0 ? tuv.x : n == 1 ? tuv.y : n == 2 ? tuv.z : tuv.w;
            const float tb = n == 0 ? tbv.x : n == 1 ? tbv.y : n == 2 ? tbv.z : tbv.w;
            const float tf = n == 0 ? tfv.x : n == 1 ? tfv.y : n == 2 ? tfv.z : tfv.w;
            g = c.alpha * dv;
            g += first ? cl : tl;
            g += last ? cr : tr;
            g += j == 0 ? sh.hc[2][i + NB * k] : td;
            g += j == NB - 1 ? sh.hc[3][i + NB * k] : tu;
            g += k == 0 ? sh.hc[4][i + NB * j] : tb;
            g += k == NB - 1 ? sh.hc[5][i + NB * j] : tf;
            off = fma_t(first ? 1.f : tl, vl, off);
            off = fma_t(last ? 1.f : tr, vr, off);
            off = fma_t(j == 0 ? 1.f : td, vd[n], off);
            off = fma_t(j == NB - 1 ? 1.f : tu, vu[n], off);
            off = fma_t(k == 0 ? 1.f : tb, vb[n], off);
            off = fma_t(k == NB - 1 ? 1.f : tf, vz[n], off);
            w = n == 0 ? vfv.x : n == 1 ? vfv.y : n == 2 ? vfv.z : vfv.w;
          }
          v[col][q] = (w > 0.f && g > 0.f) ? relax(c.omega, fast_div(fma_t(rd[col][q], w, off), g), v[col][q]) : 0.f;
        }
        sh.tile[col][h][r] = make_float4(v[col][4 * h], v[col][4 * h + 1], v[col][4 * h + 2], v[col][4 * h + 3]);
      }
      __syncthreads();
    }
  }
}

// TOP: as in h16_pass
template <int NB, int MINB, bool TOP>
__global__ void __launch_bounds__(NB *NB, MINB) k_bhgs_rows(Topo t, Coef<float> c, BlockList L, int nsweep,
                                                            const float *__restrict__ src, float *__restrict__ dst,
                                                            const float *__restrict__ rhs, const int *guard, int top) {
  __shared__ H3<NB> sh;
  extern __shared__ __align__(16) unsigned char h3_smem[];
  H3Var<NB> &sv = *reinterpret_cast<H3Var<NB> *>(h3_smem);
  pdl_enter();
  if (guard && *guard) return;
  constexpr int NT = NB * NB, NC = NB * NB * NB;
  const ListRange lr = list_range(L);
  for (int p = lr.a + blockIdx.x; p < lr.b; p += gridDim.x) {
    const int *e = L.hx + (long)p * kHX;
    const int2 ib = *reinterpret_cast<const int2 *>(e + kHXInfo);
    const int b = ib.y;
    if (L.stc && block_off(L, b)) continue;  // uniform over the CTA
    const uint16_t ft = (uint16_t)(ib.x & 0xffff);
    const long cb = (long)b * NC, fb = (long)b * t.nfb;
    const float *u = uniform_of(c, b);
    const int below = TOP ? top - e[kHXLevel] : -1;  // 0: the block itself is prolonged, 1: the finer ones at its faces
    float4 r4[NB / 4];  // the thread's row of the right-hand side, in flight with the tile
#pragma unroll
    for (int n = 0; n < NB / 4; n++) r4[n] = reinterpret_cast<const float4 *>(rhs + cb + NB * (int)threadIdx.x)[n];
    const float dv = geom(c, b, 6);
    // the tile, four cells of a row per step: two of each colour
    const float4 *s4 = reinterpret_cast<const float4 *>(src + cb);
#pragma unroll
    for (int n = threadIdx.x; n < NC / 4; n += NT) {
      const int row = n / (NB / 4), q = 2 * (n % (NB / 4)), j = row % NB, k = row / NB, pr = (j + k) & 1;
      float4 w;
      if (TOP && below == 0) {
        const int pw = e[kHXPar + 6], wc = pw & 7;
        constexpr int hb = NB / 2;
        const float2 v2 = *reinterpret_cast<const float2 *>(src + (long)(pw >> 3) * NC + hb * (wc & 1) + q +
                                                             NB * (hb * ((wc >> 1) & 1) + (j >> 1) +
                                                                   NB * (hb * ((wc >> 2) & 1) + (k >> 1))));
        w = make_float4(v2.x, v2.x, v2.y, v2.y);
        if (!u) {
          const float4 m4 = *reinterpret_cast<const float4 *>(c.vf + cb + 4 * n);
          if (!(m4.x > 0.f)) w.x = 0.f;
          if (!(m4.y > 0.f)) w.y = 0.f;
          if (!(m4.z > 0.f)) w.z = 0.f;
          if (!(m4.w > 0.f)) w.w = 0.f;
        }
      } else {
        w = s4[n];
      }
      const int at = H3<NB>::row(j, k);
      float2 *r2 = reinterpret_cast<float2 *>(&sh.tile[0][q >> 2][at]) + ((q >> 1) & 1);
      float2 *b2 = reinterpret_cast<float2 *>(&sh.tile[1][q >> 2][at]) + ((q >> 1) & 1);
      *r2 = pr ? make_float2(w.y, w.w) : make_float2(w.x, w.z);
      *b2 = pr ? make_float2(w.x, w.z) : make_float2(w.y, w.w);
    }
    // the boundary face cells: diagonal and frozen parts
#pragma unroll
    for (int f = 0; f < 6; f++) {
      const int d = f >> 1, s = f & 1, m = threadIdx.x, a0 = m % NB, a1 = m / NB;
      const int ijk[3] = {d == 0 ? (s ? NB - 1 : 0) : a0, d == 0 ? a0 : (d == 1 ? (s ? NB - 1 : 0) : a1),
                          d == 2 ? (s ? NB - 1 : 0) : a1};
      const int fx = d == 0   ? ijk[0] + s + (NB + 1) * (ijk[1] + NB * ijk[2])
                     : d == 1 ? ijk[0] + NB * (ijk[1] + s + (NB + 1) * ijk[2])
                              : ijk[0] + NB * (ijk[1] + NB * (ijk[2] + s));
      const int ty = face_type_of(ft, f);
      float vc = 0.f, vo = 0.f;
      if (ty == 0) {
        vc = u ? u[d] : c.tff[d][fb + fx];
        if (TOP && below == 0) {
          const int ni[3] = {d == 0 ? NB - 1 - ijk[0] : ijk[0], d == 1 ? NB - 1 - ijk[1] : ijk[1],
                             d == 2 ? NB - 1 - ijk[2] : ijk[2]};
          vo = vc * prolonged_value<float, 3>(t, c, e[f], ni, src, e[kHXPar + f]);
        } else {
          vo = vc * same_level_ghost<float, false>(t, b, f, ijk, src, e);
        }
      } else if (ty == 1) {
        if (t.bc_type[b * 6 + f] != kBCNeumann) vc = (u ? u[d] : c.tff[d][fb + fx]) * 2.0f;
      } else if (ty == 2) {
        vc = cf_face<float, 3>(c, t, b, f, ijk);
        vo = vc * fine_crse_ghost<float, 3, false>(t, b, f, ijk, src, e);
      } else {
        vc = cf_face<float, 3>(c, t, b, f, ijk);
        vo = refined_sum<float, 3, false>(t, c, b, f, ijk, src, e, TOP && below == 1);
      }
      sh.hc[f][m] = vc;
      if (d == 0) {
        sh.hox[s][m] = vo;
      } else {
        // seen by the cell as its neighbour: the other colour, the same place
        const int col = (ijk[0] + ijk[1] + ijk[2]) & 1, q = ijk[0] >> 1;
        const int at = d == 1 ? H3<NB>::row(s ? NB : -1, ijk[2]) : H3<NB>::row(ijk[1], s ? NB : -1);
        reinterpret_cast<float *>(&sh.tile[1 - col][q >> 2][at])[q & 3] = vo;
      }
    }
    if (!u) {
      h3_stage<NB, NB *(NB + 1)>(c.tff[1] + fb, sv.fy, [](int row) { return row % (NB + 1) + row / (NB + 1); });
      h3_stage<NB, NB *(NB + 1)>(c.tff[2] + fb, sv.fz, [](int row) { return row % NB + row / NB; });
      h3_stage<NB, NB * NB>(c.vf + cb, sv.vf, [](int row) { return row % NB + row / NB; });
      for (int n = threadIdx.x; n < NT * (NB + 1); n += NT) (&sv.fx[0][0])[n] = c.tff[0][fb + n];
    }
    __syncthreads();
    if (u)
      h3_sweeps<NB, true>(t, c, b, u, dv, nsweep, r4, sh, sv);
    else
      h3_sweeps<NB, false>(t, c, b, u, dv, nsweep, r4, sh, sv);
    if (nsweep == 0) __syncthreads();
    float4 *d4 = reinterpret_cast<float4 *>(dst + cb);
#pragma unroll
    for (int n = threadIdx.x; n < NC / 4; n += NT) {
      const int row = n / (NB / 4), q = 2 * (n % (NB / 4)), j = row % NB, k = row / NB, pr = (j + k) & 1;
      const int at = H3<NB>::row(j, k);
      const float2 r2 = *(reinterpret_cast<const float2 *>(&sh.tile[0][q >> 2][at]) + ((q >> 1) & 1));
      const float2 b2 = *(reinterpret_cast<const float2 *>(&sh.tile[1][q >> 2][at]) + ((q >> 1) & 1));
      d4[n] = pr ? make_float4(b2.x, r2.x, b2.y, r2.y) : make_float4(r2.x, b2.x, r2.y, b2.y);
    }
    __syncthreads();  // the tile is free for the next block
  }
}

// ---- the same sweep with the block's phi tile and face coefficients staged
// by TMA bulk copies (cp.async.bulk, completion on an mbarrier): in the
// compact layout both are contiguous per block.  The boundary contributions
// are gathered while the copies are in flight; the update then reads tile
// and coefficients from shared memory.  The wait is bounded: a CTA that
// times out raises the solver's error word (Topo::err), waits (bounded) for
// its own copies and leaves the block unchanged.

__device__ __forceinline__ unsigned smem_addr(const void *p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long *mbar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(mbar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long *mbar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(mbar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, unsigned bytes, unsigned long long *mbar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(mbar))
      : "memory");
}
// bounded wait for phase `parity` of the mbarrier; true when it completed
__device__ __forceinline__ bool mbar_wait(unsigned long long *mbar, unsigned parity, long limit) {
  for (long i = 0; i < limit; i++) {
    unsigned done = 0;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_addr(mbar)), "r"(parity)
        : "memory");
    if (done) return true;
    if (i > 64) __nanosleep(64);
  }
  return false;
}

template <typename T, int ND>
__global__ void __launch_bounds__(kThreads, 2) k_rbgs_bulk(Topo t, Coef<T> c, BlockList L, int color,
                                                          T *__restrict__ phi, const T *__restrict__ rhs,
                                                          const int *guard) {
  extern __shared__ __align__(128) unsigned char rbgs_bulk_smem[];
  pdl_enter();
  if (guard && *guard) return;
  const int nb = t.nb, ncell = t.ncell, nhalf = ncell >> 1, nfb = t.nfb;
  const int nface = ND == 3 ? nb * nb : nb;
  unsigned long long *mbar = reinterpret_cast<unsigned long long *>(rbgs_bulk_smem);
  T *tile = reinterpret_cast<T *>(rbgs_bulk_smem + 16);
  T *tf[3];
  for (int d = 0; d < 3; d++) tf[d] = tile + ncell + d * nfb;
  T *hc = tile + ncell + ND * nfb;
  T *hk = hc + 2 * ND * nface;
  T *hv = hk + 2 * ND * nface;
  const int p = blockIdx.x;
  const int *hxe = L.hx ? L.hx + (long)p * kHX : nullptr;
  const int b = hxe ? hxe[kHXBlock] : L.blocks[p];
  const uint16_t ft = hxe ? (uint16_t)(hxe[kHXInfo] & 0xffff) : L.ftypes[p];
  const long cb = (long)b * ncell, fb = (long)b * nfb;
  const unsigned tile_bytes = (unsigned)(ncell * sizeof(T)), face_bytes = (unsigned)(nfb * sizeof(T));
  if (threadIdx.x == 0) mbar_init(mbar, 1);
  __syncthreads();
  if (threadIdx.x == 0) {
    mbar_expect_tx(mbar, tile_bytes + ND * face_bytes);
    bulk_copy(tile, phi + cb, tile_bytes, mbar);
    for (int d = 0; d < ND; d++) bulk_copy(tf[d], c.tff[d] + fb, face_bytes, mbar);
  }
  // boundary contributions of the cells of this colour, from global memory
  for (int e = threadIdx.x; e < 2 * ND * nface; e += blockDim.x) {
    const int f = e / nface, m = e - f * nface;
    const int d = f >> 1, s = f & 1;
    int ijk[3] = {0, 0, 0};
    ijk[d] = s ? nb - 1 : 0;
    const int q0 = d == 0 ? 1 : 0, q1 = d == 2 ? 1 : 2;
    ijk[q0] = m % nb;
    if (ND == 3) ijk[q1] = m / nb;
    if (((ijk[0] + ijk[1] + ijk[2]) & 1) != color) continue;
    int fx;
    if (d == 0)
      fx = ijk[0] + s + (nb + 1) * (ijk[1] + nb * ijk[2]);
    else if (d == 1)
      fx = ijk[0] + nb * (ijk[1] + s + (nb + 1) * ijk[2]);
    else
      fx = encode(ijk, nb) + s * nb * nb;
    const int ty = face_type_of(ft, f);
    T vc = 0, vk = 0, vv = 0;
    if (ty == 0) {
      vc = vk = c.tff[d][fb + fx];
      vv = same_level_ghost<T, false>(t, b, f, ijk, phi, hxe);
    } else if (ty == 1) {
      if (t.bc_type[b * 6 + f] != kBCNeumann) vc = c.tff[d][fb + fx] * (T)2.0;
    } else if (ty == 2) {
      vc = vk = cf_face<T, ND>(c, t, b, f, ijk);
      vv = fine_crse_ghost<T, ND, false>(t, b, f, ijk, phi, hxe);
    } else {
      vc = cf_face<T, ND>(c, t, b, f, ijk);
      vk = (T)1;
      vv = refined_sum<T, ND, false>(t, c, b, f, ijk, phi, hxe);
    }
    hc[e] = vc;
    hk[e] = vk;
    hv[e] = vv;
  }
  const long kWait = 1l << 22;  // about 0.3 s with the back-off: never reached unless the copy engine failed
  const bool ok = mbar_wait(mbar, 0, kWait);
  if (__syncthreads_or(!ok)) {
    if (threadIdx.x == 0) {
      // the error word makes the solve report a CUDA error; should this
      // bounded drain time out too, copies may still land in shared memory
      // the CTA released, so nothing the device computes after the flag is
      // set is trusted (the host reports the failure after the solve)
      if (t.err) atomicExch(t.err, 1);
      mbar_wait(mbar, 0, kWait);  // let the copies into this CTA's shared memory land before it exits
    }
    return;
  }
  const T dv = geom(c, b, 6);
  for (int h = threadIdx.x; h < nhalf; h += blockDim.x) {
    int ijk[3];
    color_cell_fast<ND>(h, t, color, ijk);
    const int ci = t.lnb >= 0 ? ijk[0] + ((ijk[1] + (ijk[2] << t.lnb)) << t.lnb) : encode(ijk, nb);
    T diag = c.alpha * dv;
    T off = 0;
#pragma unroll
    for (int f = 0; f < 2 * ND; f++) {
      const int d = f >> 1, s = f & 1;
      const bool bnd = s ? ijk[d] == nb - 1 : ijk[d] == 0;
      if (!bnd) {
        int fx;
        if (d == 0)
          fx = ijk[0] + s + (nb + 1) * (ijk[1] + nb * ijk[2]);
        else if (d == 1)
          fx = ijk[0] + nb * (ijk[1] + s + (nb + 1) * ijk[2]);
        else
          fx = ci + s * nb * nb;
        const T coef = tf[d][fx];
        const int stride = d == 0 ? 1 : (d == 1 ? nb : nb * nb);
        diag += coef;
        off = fma_t(coef, tile[ci + (s ? stride : -stride)], off);
      } else {
        const int q0 = d == 0 ? 1 : 0, q1 = d == 2 ? 1 : 2;
        const int m = ijk[q0] + (ND == 3 ? nb * ijk[q1] : 0);
        const int e = f * nface + m;
        diag += hc[e];
        off = fma_t(hk[e], hv[e], off);
      }
    }
    T unew = 0;
    if (sizeof(T) == 8 && L.sa) {
      const long fo = (long)p * ncell + ci;
      unew = fma_t(rhs[cb + ci], (T)L.sa[fo], off * (T)L.ia[fo]);
      if (L.ia[fo] != 0.0) unew = relax(c.omega, unew, tile[ci]);
    } else {
      const T vfv = c.vf[cb + ci];
      if (vfv > 0 && diag > 0) unew = relax(c.omega, fast_div(fma_t(rhs[cb + ci] * dv, vfv, off), diag), tile[ci]);
    }
    tile[ci] = unew;
  }
  __syncthreads();
  if ((ncell & 3) == 0 && sizeof(T) == 4) {
    const float4 *src = reinterpret_cast<const float4 *>(tile);
    float4 *dst = reinterpret_cast<float4 *>(phi + cb);
    for (int i = threadIdx.x; i < (ncell >> 2); i += blockDim.x) dst[i] = src[i];
  } else {
    for (int i = threadIdx.x; i < ncell; i += blockDim.x) phi[cb + i] = tile[i];
  }
}

// ---- persistent, double-buffered: one CTA per SM walks blocks p = blockIdx.x,
// blockIdx.x + gridDim.x, ...; while it gathers the boundary contributions of
// block i and updates it from shared memory, the copy engine streams block
// i+1's tile, face coefficients, rhs and vf into the other buffer.
constexpr int kStreamThreads = 512;

template <typename T, int ND>
__global__ void __launch_bounds__(kStreamThreads, 1) k_rbgs_stream(Topo t, Coef<T> c, BlockList L, int color,
                                                                   T *__restrict__ phi, const T *__restrict__ rhs,
                                                                   const int *guard) {
  extern __shared__ __align__(128) unsigned char rbgs_stream_smem[];
  pdl_enter();
  if (guard && *guard) return;
  const int nb = t.nb, ncell = t.ncell, nhalf = ncell >> 1, nfb = t.nfb;
  const int nface = ND == 3 ? nb * nb : nb;
  const size_t buf_elems = (size_t)3 * ncell + (size_t)ND * nfb;  // tile, rhs, vf, faces
  unsigned long long *mbar = reinterpret_cast<unsigned long long *>(rbgs_stream_smem);  // [2]
  T *buf0 = reinterpret_cast<T *>(rbgs_stream_smem + 16);
  T *hc = buf0 + 2 * buf_elems;
  T *hk = hc + 2 * ND * nface;
  T *hv = hk + 2 * ND * nface;
  const unsigned tile_bytes = (unsigned)(ncell * sizeof(T)), face_bytes = (unsigned)(nfb * sizeof(T));
  const unsigned tx = 3 * tile_bytes + ND * face_bytes;
  auto issue = [&](int pp, int j) {  // thread 0: copies of list entry pp into buffer j
    const int bb = L.blocks[pp];
    T *bt = buf0 + j * buf_elems;
    // buffer j was last read and written through the generic proxy (the
    // sweep and the copy-out, ordered before this point by __syncthreads);
    // the bulk copies write it through the async proxy
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_expect_tx(&mbar[j], tx);
    bulk_copy(bt, phi + (long)bb * ncell, tile_bytes, &mbar[j]);
    bulk_copy(bt + ncell, rhs + (long)bb * ncell, tile_bytes, &mbar[j]);
    bulk_copy(bt + 2 * ncell, c.vf + (long)bb * ncell, tile_bytes, &mbar[j]);
    for (int d = 0; d < ND; d++) bulk_copy(bt + 3 * ncell + d * nfb, c.tff[d] + (long)bb * nfb, face_bytes, &mbar[j]);
  };
  if (threadIdx.x == 0) {
    mbar_init(&mbar[0], 1);
    mbar_init(&mbar[1], 1);
  }
  __syncthreads();
  if (blockIdx.x >= L.n) return;
  if (threadIdx.x == 0) issue(blockIdx.x, 0);
  const long kWait = 1l << 22;
  unsigned phase[2] = {0u, 0u};
  int k = 0;
  for (int p = blockIdx.x; p < L.n; p += gridDim.x, k++) {
    const int j = k & 1;
    if (threadIdx.x == 0 && p + (int)gridDim.x < L.n) issue(p + gridDim.x, j ^ 1);
    const int *hxe = L.hx ? L.hx + (long)p * kHX : nullptr;
    const int b = hxe ? hxe[kHXBlock] : L.blocks[p];
    const uint16_t ft = hxe ? (uint16_t)(hxe[kHXInfo] & 0xffff) : L.ftypes[p];
    const long cb = (long)b * ncell, fb = (long)b * nfb;
    for (int e = threadIdx.x; e < 2 * ND * nface; e += blockDim.x) {
      const int f = e / nface, m = e - f * nface;
      const int d = f >> 1, s = f & 1;
      int ijk[3] = {0, 0, 0};
      ijk[d] = s ? nb - 1 : 0;
      const int q0 = d == 0 ? 1 : 0, q1 = d == 2 ? 1 : 2;
      ijk[q0] = m % nb;
      if (ND == 3) ijk[q1] = m / nb;
      if (((ijk[0] + ijk[1] + ijk[2]) & 1) != color) continue;
      int fx;
      if (d == 0)
        fx = ijk[0] + s + (nb + 1) * (ijk[1] + nb * ijk[2]);
      else if (d == 1)
        fx = ijk[0] + nb * (ijk[1] + s + (nb + 1) * ijk[2]);
      else
        fx = encode(ijk, nb) + s * nb * nb;
      const int ty = face_type_of(ft, f);
      T vc = 0, vk = 0, vv = 0;
      if (ty == 0) {
        vc = vk = c.tff[d][fb + fx];
        vv = same_level_ghost<T, false>(t, b, f, ijk, phi, hxe);
      } else if (ty == 1) {
        if (t.bc_type[b * 6 + f] != kBCNeumann) vc = c.tff[d][fb + fx] * (T)2.0;
      } else if (ty == 2) {
        vc = vk = cf_face<T, ND>(c, t, b, f, ijk);
        vv = fine_crse_ghost<T, ND, false>(t, b, f, ijk, phi, hxe);
      } else {
        vc = cf_face<T, ND>(c, t, b, f, ijk);
        vk = (T)1;
        vv = refined_sum<T, ND, false>(t, c, b, f, ijk, phi, hxe);
      }
      hc[e] = vc;
      hk[e] = vk;
      hv[e] = vv;
    }
    const bool ok = mbar_wait(&mbar[j], phase[j], kWait);
    phase[j] ^= 1u;
    if (__syncthreads_or(!ok)) {
      if (threadIdx.x == 0) {
        // the error word makes the solve report a CUDA error; should the
        // bounded drain below also time out, copies may still be landing in
        // shared memory this CTA released, so nothing the device computes
        // after the flag is set is trusted (the host reports the failure)
        if (t.err) atomicExch(t.err, 1);
        // let this CTA's copies land before it exits
        mbar_wait(&mbar[j], phase[j] ^ 1u, kWait);
        if (p + (int)gridDim.x < L.n) mbar_wait(&mbar[j ^ 1], phase[j ^ 1], kWait);
      }
      return;
    }
    T *tile = buf0 + j * buf_elems;
    const T *rh = tile + ncell, *vfs = tile + 2 * ncell, *tf0 = tile + 3 * ncell;
    const T dv = geom(c, b, 6);
    for (int h = threadIdx.x; h < nhalf; h += blockDim.x) {
      int ijk[3];
      color_cell_fast<ND>(h, t, color, ijk);
      const int ci = t.lnb >= 0 ? ijk[0] + ((ijk[1] + (ijk[2] << t.lnb)) << t.lnb) : encode(ijk, nb);
      T diag = c.alpha * dv;
      T off = 0;
#pragma unroll
      for (int f = 0; f < 2 * ND; f++) {
        const int d = f >> 1, s = f & 1;
        const bool bnd = s ? ijk[d] == nb - 1 : ijk[d] == 0;
        if (!bnd) {
          int fx;
          if (d == 0)
            fx = ijk[0] + s + (nb + 1) * (ijk[1] + nb * ijk[2]);
          else if (d == 1)
            fx = ijk[0] + nb * (ijk[1] + s + (nb + 1) * ijk[2]);
          else
            fx = ci + s * nb * nb;
          const T coef = tf0[d * nfb + fx];
          const int stride = d == 0 ? 1 : (d == 1 ? nb : nb * nb);
          diag += coef;
          off = fma_t(coef, tile[ci + (s ? stride : -stride)], off);
        } else {
          const int q0 = d == 0 ? 1 : 0, q1 = d == 2 ? 1 : 2;
          const int m = ijk[q0] + (ND == 3 ? nb * ijk[q1] : 0);
          const int e = f * nface + m;
          diag += hc[e];
          off = fma_t(hk[e], hv[e], off);
        }
      }
      T unew = 0;
      if (sizeof(T) == 8 && L.sa) {
        const long fo = (long)p * ncell + ci;
        unew = fma_t(rh[ci], (T)L.sa[fo], off * (T)L.ia[fo]);
        if (L.ia[fo] != 0.0) unew = relax(c.omega, unew, tile[ci]);
      } else {
        const T vfv = vfs[ci];
        if (vfv > 0 && diag > 0) unew = relax(c.omega, fast_div(fma_t(rh[ci] * dv, vfv, off), diag), tile[ci]);
      }
      tile[ci] = unew;
    }
    __syncthreads();
    if ((ncell & 3) == 0 && sizeof(T) == 4) {
      const float4 *src = reinterpret_cast<const float4 *>(tile);
      float4 *dst = reinterpret_cast<float4 *>(phi + cb);
      for (int i = threadIdx.x; i < (ncell >> 2); i += blockDim.x) dst[i] = src[i];
    } else {
      for (int i = threadIdx.x; i < ncell; i += blockDim.x) phi[cb + i] = tile[i];
    }
    __syncthreads();  // buffer j and the boundary arrays are free again
  }
}

template <typename T, int ND>
static size_t rbgs_stream_smem(const Topo &t) {
  const int nface = ND == 3 ? t.nb * t.nb : t.nb;
  return 16 + sizeof(T) * (2 * ((size_t)3 * t.ncell + (size_t)ND * t.nfb) + 3 * 2 * ND * (size_t)nface);
}

template <typename T, int ND>
static void rbgs_stream_go(const Topo &t, const Coef<T> &c, const BlockList &L, int color, T *phi, const T *rhs,
                           const int *guard, cudaStream_t s, bool pdl) {
  const size_t smem = rbgs_stream_smem<T, ND>(t);
  int dev = 0, nsm = 152;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    nsm = 152;
  }
  ensure_max_smem((const void *)k_rbgs_stream<T, ND>, 227 * 1024);
  launch_k(pdl, k_rbgs_stream<T, ND>, std::min(L.n, nsm), kStreamThreads, smem, s, t, c, L, color, phi, rhs,
           guard);
}

template <typename T, int ND>
static size_t rbgs_bulk_smem(const Topo &t) {
  const int nface = ND == 3 ? t.nb * t.nb : t.nb;
  return 16 + sizeof(T) * ((size_t)t.ncell + (size_t)ND * t.nfb + 3 * 2 * ND * (size_t)nface);
}

template <typename T, int ND>
static void rbgs_bulk_go(const Topo &t, const Coef<T> &c, const BlockList &L, int color, T *phi, const T *rhs,
                         const int *guard, cudaStream_t s, bool pdl) {
  const size_t smem = rbgs_bulk_smem<T, ND>(t);
  ensure_max_smem((const void *)k_rbgs_bulk<T, ND>, 200 * 1024);
  const int threads = std::min(kThreads, ((t.ncell >> 1) + 31) / 32 * 32);
  launch_k(pdl, k_rbgs_bulk<T, ND>, L.n, threads, smem, s, t, c, L, color, phi, rhs, guard);
}

int rbgs_bulk_error(int *err, cudaStream_t s, bool clear) {
  if (!err) return 0;
  int v = 0;
  if (cudaMemcpyAsync(&v, err, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return -1;
  if (clear && v) {
    if (cudaMemsetAsync(err, 0, sizeof(int), s) != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess) return -1;
  }
  return v;
}

// ---- prolongation of a level fused with the first (red) sweep that follows
// it: one CTA per block of the level; the block's tile is filled with its
// prolonged values (masked injection from the parent, as k_prolong), the
// red cells' same-level neighbours outside the block are prolonged on the
// fly from their own parents, coarse neighbours (FINE_CRSE) are read as they
// are; the red cells are then updated with the tiled sweep's arithmetic and
// the whole tile is written.  Same values as k_prolong + k_rbgs_tile.

// FAC: L has the FP64 smoother's factors, which need no diagonal (and leave
// registers for six CTAs per SM: 30.3 us at four, 26.5 at six; 33.5 with the
// diagonal; 32 problems, 5.4 M cells).
template <typename T, int ND, bool FAC>
__global__ void __launch_bounds__(kThreads, FAC ? 6 : 4) k_prolong_red(Topo t, Coef<T> c, BlockList L, T *__restrict__ phi,
                                                            const T *__restrict__ rhs, const int *guard,
                                                            BlockList X) {
  extern __shared__ __align__(16) unsigned char pr_smem[];
  pdl_enter();
  if (guard && *guard) return;
  const int nb = t.nb, ncell = t.ncell, nhalf = ncell >> 1;
  const int nface = ND == 3 ? nb * nb : nb;
  T *tile = reinterpret_cast<T *>(pr_smem);
  T *hc = tile + ncell;
  T *hk = hc + 2 * ND * nface;
  T *hv = hk + 2 * ND * nface;
  const ListRange lr = list_range(L), xr = list_range(X);
  const int nl = lr.b - lr.a, nx = xr.b - xr.a;
  for (int p = blockIdx.x; p < nl + nx; p += gridDim.x) {
    if (p >= nl) {
      // the red sweep of a block of X: blocks two or more levels coarser,
      // which neither read nor are read by the level being prolonged
      const int px = xr.a + p - nl;
      const long fo = factor_entry(X, px) * ncell;
      const int *e = X.hx + (long)px * kHX;
      if (block_off(X, e[kHXBlock])) continue;
      for (int h = threadIdx.x; h < nhalf; h += blockDim.x) {
        int ijk[3];
        color_cell_fast<ND>(h, t, 0, ijk);
        smooth_cell_fast<T, ND>(t, c, e[kHXBlock], (uint16_t)(e[kHXInfo] & 0xffff), ijk, phi, rhs,
                                X.sa ? X.sa + fo : nullptr, X.ia ? X.ia + fo : nullptr, e);
      }
      continue;
    }
    const int pl = lr.a + p;
    const int *hxe = L.hx ? L.hx + (long)pl * kHX : nullptr;
    const int b = hxe ? hxe[kHXBlock] : L.blocks[pl];
    if (block_off(L, b)) continue;  // uniform over the CTA
    const long f0 = factor_entry(L, pl) * ncell;
    const uint16_t ft = hxe ? (uint16_t)(hxe[kHXInfo] & 0xffff) : L.ftypes[pl];
    const long cb = (long)b * ncell;
    const long fb = (long)b * t.nfb;
    const T *u = uniform_of(c, b);  // constant coefficients: no face or vf loads
    for (int i = threadIdx.x; i < ncell; i += blockDim.x) {
      int ijk[3];
      decode<ND>(i, nb, ijk);
      tile[i] = prolonged_value<T, ND>(t, c, b, ijk, phi, hxe ? hxe[kHXPar + 6] : -1, u != nullptr);
    }
    for (int e = threadIdx.x; e < 2 * ND * nface; e += blockDim.x) {
      const int f = e / nface, m = e - f * nface;
      const int d = f >> 1, s = f & 1;
      int ijk[3] = {0, 0, 0};
      ijk[d] = s ? nb - 1 : 0;
      const int q0 = d == 0 ? 1 : 0, q1 = d == 2 ? 1 : 2;
      ijk[q0] = m % nb;
      if (ND == 3) ijk[q1] = m / nb;
      if ((ijk[0] + ijk[1] + ijk[2]) & 1) continue;  // red cells only
      int fx;
      if (d == 0)
        fx = ijk[0] + s + (nb + 1) * (ijk[1] + nb * ijk[2]);
      else if (d == 1)
        fx = ijk[0] + nb * (ijk[1] + s + (nb + 1) * ijk[2]);
      else
        fx = encode(ijk, nb) + s * nb * nb;
      const int ty = face_type_of(ft, f);
      T vc = 0, vk = 0, vv = 0;
      if (ty == 0) {
        const int n = hxe ? hxe[f] : t.neighbor[b * 6 + f];
        int ni[3] = {ijk[0], ijk[1], ijk[2]};
        ni[d] = s ? 0 : nb - 1;
        vc = vk = u ? u[d] : c.tff[d][fb + fx];
        vv = prolonged_value<T, ND>(t, c, n, ni, phi, hxe ? hxe[kHXPar + f] : -1);
      } else if (ty == 1) {
        if (!FAC && t.bc_type[b * 6 + f] != kBCNeumann) vc = (u ? u[d] : c.tff[d][fb + fx]) * (T)2.0;
      } else if (ty == 2) {
        vc = vk = cf_face<T, ND>(c, t, b, f, ijk);
        vv = fine_crse_ghost<T, ND, false>(t, b, f, ijk, phi, hxe);
      } else {  // not at the finest level of a tower
        if constexpr (!FAC) vc = cf_face<T, ND>(c, t, b, f, ijk);
        vk = (T)1;
        vv = refined_sum<T, ND, false>(t, c, b, f, ijk, phi, hxe);
      }
      if constexpr (!FAC) hc[e] = vc;
      hk[e] = vk;
      hv[e] = vv;
    }
    __syncthreads();
    const T dv = geom(c, b, 6);
    for (int h = threadIdx.x; h < nhalf; h += blockDim.x) {
      int ijk[3];
      color_cell_fast<ND>(h, t, 0, ijk);
      const int ci = t.lnb >= 0 ? ijk[0] + ((ijk[1] + (ijk[2] << t.lnb)) << t.lnb) : encode(ijk, nb);
      T diag = FAC ? (T)0 : c.alpha * dv;
      T off = 0;
#pragma unroll
      for (int f = 0; f < 2 * ND; f++) {
        const int d = f >> 1, s = f & 1;
        const bool bnd = s ? ijk[d] == nb - 1 : ijk[d] == 0;
        if (!bnd) {
          int fx;
          if (d == 0)
            fx = ijk[0] + s + (nb + 1) * (ijk[1] + nb * ijk[2]);
          else if (d == 1)
            fx = ijk[0] + nb * (ijk[1] + s + (nb + 1) * ijk[2]);
          else
            fx = ci + s * nb * nb;
          const T coef = u ? u[d] : c.tff[d][fb + fx];
          const int stride = d == 0 ? 1 : (d == 1 ? nb : nb * nb);
          if constexpr (!FAC) diag += coef;
          off = fma_t(coef, tile[ci + (s ? stride : -stride)], off);
        } else {
          const int q0 = d == 0 ? 1 : 0, q1 = d == 2 ? 1 : 2;
          const int m = ijk[q0] + (ND == 3 ? nb * ijk[q1] : 0);
          const int e = f * nface + m;
          if constexpr (!FAC) diag += hc[e];
          off = fma_t(hk[e], hv[e], off);
        }
      }
      T unew = 0;
      if constexpr (FAC) {
        bool inner = true;
#pragma unroll
        for (int q = 0; q < ND; q++) inner = inner && ijk[q] > 0 && ijk[q] < nb - 1;
        const long fo = f0 + ci;
        const bool ui = u && inner;
        const T iav = ui ? u[7] : (T)L.ia[fo];  // 0 in a solid cell
        unew = fma_t(rhs[cb + ci], ui ? u[6] : (T)L.sa[fo], off * iav);
        if (nonzero(iav)) unew = relax(c.omega, unew, tile[ci]);
      } else {
        const T vfv = u ? (T)1 : c.vf[cb + ci];
        if (vfv > 0 && diag > 0) unew = relax(c.omega, fast_div(fma_t(rhs[cb + ci] * dv, vfv, off), diag), tile[ci]);
      }
      tile[ci] = unew;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < ncell; i += blockDim.x) phi[cb + i] = tile[i];
    __syncthreads();
  }
}

template <typename T>
void launch_prolong_red(const Topo &t, const Coef<T> &c, const BlockList &L, T *phi, const T *rhs,
                        const int *guard, cudaStream_t s, bool pdl, const BlockList &X, int form) {
  if (L.n == 0) return;
  if (X.n > 0 && !X.hx) return;  // the extra sweep reads its blocks through halo descriptors
  if constexpr (sizeof(T) == 4) {
    if (form == 1 && t.ndim == 2 && t.nb == 16 && L.hx && c.cf) {
      const int g = std::min((L.n + X.n + 7) / 8, 152 * 64);
      launch_k(pdl, k_prolong_red_warp16<5>, g, kThreads, 0, s, t, c, L, phi, rhs, guard, X);
      return;
    }
  }
  if constexpr (sizeof(T) == 4) {
    if (form == 1 && t.ndim == 3 && t.nb == 8 && L.hx && c.cf) {
      const int g = std::min(L.n + X.n, 152 * 32);
      launch_k(pdl, k_prolong_red_rows8, g, 64, 0, s, t, c, L, phi, rhs, guard, X);
      return;
    }
  }
  const int nface = t.ndim == 3 ? t.nb * t.nb : t.nb;
  const size_t smem = sizeof(T) * ((size_t)t.ncell + 3 * 2 * t.ndim * (size_t)nface);
  const int threads = std::min(kThreads, ((t.ncell >> 1) + 31) / 32 * 32);
  const int grid = std::min(L.n + X.n, L.pb ? kReducedGrid : 152 * 64);
  auto go = [&](auto k) {
    ensure_max_smem((const void *)k, 200 * 1024);
    launch_k(pdl, k, grid, threads, smem, s, t, c, L, phi, rhs, guard, X);
  };
  if constexpr (sizeof(T) == 8) {
    if (L.sa) {
      t.ndim == 2 ? go(k_prolong_red<T, 2, true>) : go(k_prolong_red<T, 3, true>);
      return;
    }
  }
  t.ndim == 2 ? go(k_prolong_red<T, 2, false>) : go(k_prolong_red<T, 3, false>);
}

template <typename T, int ND>
static size_t rbgs_tile_smem(const Topo &t) {
  const int nface = ND == 3 ? t.nb * t.nb : t.nb;
  return sizeof(T) * ((size_t)t.ncell + 3 * 2 * ND * (size_t)nface);
}

template <typename T, int ND, int MINB>
static void rbgs_tile_go(const Topo &t, const Coef<T> &c, const BlockList &L, int color, T *phi, const T *rhs,
                         const int *guard, cudaStream_t s, bool pdl) {
  const size_t smem = rbgs_tile_smem<T, ND>(t);
  ensure_max_smem((const void *)k_rbgs_tile<T, ND, MINB>, 200 * 1024);
  const int threads = std::min(kThreads, ((t.ncell >> 1) + 31) / 32 * 32);
  const int grid = std::min(L.n, L.pb ? kReducedGrid : 152 * 64);
  launch_k(pdl, k_rbgs_tile<T, ND, MINB>, grid, threads, smem, s, t, c, L, color, phi, rhs, guard);
}

// variant v: launch bounds (256 threads, kRbgsMinBlocks[v] CTAs per SM), i.e.
// a register cap of 65536 / (256 * min CTAs); same arithmetic in every variant
template <typename T, int ND, int MINB>
static void rbgs_go(const Topo &t, const Coef<T> &c, const BlockList &L, int color, T *phi, const T *rhs,
                    const int *guard, cudaStream_t s, bool pdl, dim3 grid, int threads) {
  launch_k(pdl, k_rbgs<T, ND, MINB>, grid, threads, 0, s, t, c, L, color, phi, rhs, guard);
}

// variant 10: CPT = 2 cells per thread (k_rbgs_ilp), cap 64; variants 11 .. 13
// of an FP32 sweep: one warp per 16x16 block in 2D (k_rbgs_warp16, register
// caps 64, 48, 80), one thread per row of an 8^3 block in 3D (k_rbgs_rows8,
// 8, 12, 16 CTAs of 64 threads per SM); elsewhere variant 3
template <typename T, int ND, int MINB, int CPT>
static void rbgs_ilp_go(const Topo &t, const Coef<T> &c, const BlockList &L, int color, T *phi, const T *rhs,
                        const int *guard, cudaStream_t s, bool pdl, dim3 grid, int threads) {
  grid.y = std::min((L.n + CPT - 1) / CPT, L.pb ? kReducedGrid : 65535);
  if constexpr (sizeof(T) == 8) {
    if (L.sa) {
      launch_k(pdl, k_rbgs_ilp<T, ND, MINB, CPT, true>, grid, threads, 0, s, t, c, L, color, phi, rhs, guard);
      return;
    }
  }
  launch_k(pdl, k_rbgs_ilp<T, ND, MINB, CPT, false>, grid, threads, 0, s, t, c, L, color, phi, rhs, guard);
}

template <typename T, int ND>
static void rbgs_nd(int variant, const Topo &t, const Coef<T> &c, const BlockList &L, int color, T *phi,
                    const T *rhs, const int *guard, cudaStream_t s, bool pdl, dim3 grid, int threads) {
  switch (variant) {
    case 10: rbgs_ilp_go<T, ND, 4, 2>(t, c, L, color, phi, rhs, guard, s, pdl, grid, threads); return;
    case 11:
    case 12:
    case 13:
      if constexpr (ND == 2 && sizeof(T) == 4) {
        if (t.nb == 16 && L.hx && c.cf) {
          const int g = std::min((L.n + 7) / 8, 152 * 64);
          if (variant == 11)
            launch_k(pdl, k_rbgs_warp16<4>, g, kThreads, 0, s, t, c, L, color, phi, rhs, guard);
          else if (variant == 12)
            launch_k(pdl, k_rbgs_warp16<5>, g, kThreads, 0, s, t, c, L, color, phi, rhs, guard);
          else
            launch_k(pdl, k_rbgs_warp16<3>, g, kThreads, 0, s, t, c, L, color, phi, rhs, guard);
          return;
        }
      }
      if constexpr (ND == 3 && sizeof(T) == 4) {
        if (t.nb == 8 && L.hx && c.cf) {
          const int g = std::min(L.n, 152 * 32);
          const auto k = variant == 11 ? k_rbgs_rows8<8> : variant == 12 ? k_rbgs_rows8<12> : k_rbgs_rows8<16>;
          launch_k(pdl, k, g, 64, 0, s, t, c, L, color, phi, rhs, guard);
          return;
        }
      }
      rbgs_go<T, ND, 6>(t, c, L, color, phi, rhs, guard, s, pdl, grid, threads);
      return;
    default: break;
  }
  switch (variant) {
    case 0: rbgs_go<T, ND, 2>(t, c, L, color, phi, rhs, guard, s, pdl, grid, threads); break;
    case 1: rbgs_go<T, ND, 3>(t, c, L, color, phi, rhs, guard, s, pdl, grid, threads); break;
    case 2: rbgs_go<T, ND, 4>(t, c, L, color, phi, rhs, guard, s, pdl, grid, threads); break;
    case 3: rbgs_go<T, ND, 6>(t, c, L, color, phi, rhs, guard, s, pdl, grid, threads); break;
    case 4: rbgs_go<T, ND, 8>(t, c, L, color, phi, rhs, guard, s, pdl, grid, threads); break;
    case 5: rbgs_tile_go<T, ND, 2>(t, c, L, color, phi, rhs, guard, s, pdl); break;
    case 6: rbgs_tile_go<T, ND, 4>(t, c, L, color, phi, rhs, guard, s, pdl); break;
    case 7: rbgs_tile_go<T, ND, 6>(t, c, L, color, phi, rhs, guard, s, pdl); break;
    case 8: rbgs_bulk_go<T, ND>(t, c, L, color, phi, rhs, guard, s, pdl); break;
    default: rbgs_stream_go<T, ND>(t, c, L, color, phi, rhs, guard, s, pdl); break;
  }
}

template <typename T>
void launch_rbgs(const Topo &t, const Coef<T> &c, const BlockList &L, int color, T *phi, const T *rhs,
                 const int *guard, cudaStream_t s, bool pdl, int variant) {
  const int nhalf = t.ncell / 2;
  if (L.n == 0 || nhalf == 0) return;
  // the tiled variants need the tile and halo in shared memory (<= 200 KiB);
  // the bulk-copy variant also needs 16-byte multiples for the tile and the
  // face rows of a block (and L.n CTAs in one grid dimension)
  const size_t tile = t.ndim == 2 ? rbgs_tile_smem<T, 2>(t) : rbgs_tile_smem<T, 3>(t);
  if (variant >= 5 && variant <= 9 && tile > 200 * 1024) variant = 3;
  const bool aligned = (t.ncell * sizeof(T)) % 16 == 0 && (t.nfb * sizeof(T)) % 16 == 0;
  // the bulk-copy variants know no per-problem states and no reduced lists
  if ((L.stc || L.pb) && (variant == 8 || variant == 9)) variant = 7;
  if (variant == 8) {
    const size_t bulk = t.ndim == 2 ? rbgs_bulk_smem<T, 2>(t) : rbgs_bulk_smem<T, 3>(t);
    if (bulk > 200 * 1024 || !aligned) variant = 7;
  }
  if (variant == 9) {
    const size_t st = t.ndim == 2 ? rbgs_stream_smem<T, 2>(t) : rbgs_stream_smem<T, 3>(t);
    if (st > 227 * 1024 || !aligned) variant = 7;
  }
  const int threads = std::min(kThreads, (nhalf + 31) / 32 * 32);
  const dim3 grid((nhalf + threads - 1) / threads, std::min(L.n, L.pb ? kReducedGrid : 65535));
  if (t.ndim == 2)
    rbgs_nd<T, 2>(variant, t, c, L, color, phi, rhs, guard, s, pdl, grid, threads);
  else
    rbgs_nd<T, 3>(variant, t, c, L, color, phi, rhs, guard, s, pdl, grid, threads);
}

template <int NB, int MINB>
static void bhgs_rows_go(const Topo &t, const Coef<float> &c, const BlockList &L, int nsweep, const float *src,
                         float *dst, const float *rhs, const int *guard, cudaStream_t s, bool pdl, int top, int grid) {
  const auto kern = top ? k_bhgs_rows<NB, MINB, true> : k_bhgs_rows<NB, MINB, false>;
  const int smem = (int)sizeof(H3Var<NB>);
  ensure_max_smem((const void *)kern, smem);
  launch_k(pdl, kern, grid, NB * NB, smem, s, t, c, L, nsweep, src, dst, rhs, guard, top);
}

template <typename T>
bool bhgs_prolongs(const Topo &t, const Coef<T> &c, const BlockList &L) {
  return sizeof(T) == 4 && L.hx && c.cf && (t.ndim == 2 ? t.nb == 16 : t.nb == 16 || t.nb == 8);
}

template <typename T>
void launch_bhgs(const Topo &t, const Coef<T> &c, const BlockList &L, int nsweep, const T *src, T *dst,
                 const T *rhs, const int *guard, cudaStream_t s, bool pdl, int top) {
  const int nhalf = t.ncell / 2;
  if (L.n == 0 || nhalf == 0) return;
  if constexpr (sizeof(T) == 4) {
    if (t.ndim == 2 && t.nb == 16 && L.hx && c.cf) {
      const int warps = kH16Threads / 32, g = std::min((L.n + warps - 1) / warps, 152 * 64);
      launch_k(pdl, top ? k_bhgs_warp16<4, true> : k_bhgs_warp16<4, false>, g, kH16Threads, 0, s, t, c, L, nsweep, src,
               dst, rhs, guard, top);
      return;
    }
    if (t.ndim == 3 && (t.nb == 16 || t.nb == 8) && L.hx && c.cf) {
      const int g = std::min(L.n, L.pb ? kReducedGrid : 152 * 64);
      if (t.nb == 16)
        bhgs_rows_go<16, 2>(t, c, L, nsweep, src, dst, rhs, guard, s, pdl, top, g);
      else
        bhgs_rows_go<8, 8>(t, c, L, nsweep, src, dst, rhs, guard, s, pdl, top, g);
      return;
    }
  }
  const int nface = t.ndim == 3 ? t.nb * t.nb : t.nb;
  const size_t smem = sizeof(T) * ((size_t)t.ncell + 2 * 2 * t.ndim * (size_t)nface);
  const int threads = std::min(kThreads, (nhalf + 31) / 32 * 32);
  const int grid = std::min(L.n, L.pb ? kReducedGrid : 152 * 64);
  if (t.ndim == 2) {
    ensure_max_smem((const void *)k_bhgs<T, 2, 2>, 200 * 1024);
    launch_k(pdl, k_bhgs<T, 2, 2>, grid, threads, smem, s, t, c, L, nsweep, src, dst, rhs, guard);
  } else {
    ensure_max_smem((const void *)k_bhgs<T, 3, 2>, 200 * 1024);
    launch_k(pdl, k_bhgs<T, 3, 2>, grid, threads, smem, s, t, c, L, nsweep, src, dst, rhs, guard);
  }
}

template <typename T>
void launch_smooth(const Topo &t, const Coef<T> &c, const BlockList &L, int color, T *phi, const T *rhs,
                   const int *guard, cudaStream_t s, bool pdl) {
  const long work = (long)L.n * (t.ncell / 2);
  if (work == 0) return;
  if (t.ndim == 2)
    launch_k(pdl, k_smooth<T, 2>, grid_for(work), kThreads, 0, s, t, c, L, color, phi, rhs, guard);
  else
    launch_k(pdl, k_smooth<T, 3>, grid_for(work), kThreads, 0, s, t, c, L, color, phi, rhs, guard);
}

constexpr long kRestrictPairs = 1l << 17;
template <typename T>
void launch_restrict(const Topo &t, const Coef<T> &c, const BlockList &L, T *phi, const int *guard,
                     cudaStream_t s, bool pdl) {
  const long work = (long)L.n * t.ncell;
  if (work == 0) return;
  // Two cells per thread from 131,072 cells of a level on (a side that is a
  // multiple of four: rows of four fine cells are aligned).  The form reads a
  // record before it knows whether it needs vf, one more load in the chain, and
  // has half the threads to hide it: us a launch with one and with two cells, 2D
  // FP32 30 thousand cells 3.4 and 3.7, 138 thousand 5.5 and 5.7, 364 thousand
  // 7.9 and 6.4; FP64 30 thousand 5.1 and 7.3, 131 thousand 11.0 and 9.9; 3D FP64
  // 33 thousand 6.2 and 8.4, 246 thousand 17.7 and 14.8.
  if (t.nb % 4 == 0 && work >= kRestrictPairs) {
    const auto k = t.ndim == 2 ? k_restrict_pairs<T, 2> : k_restrict_pairs<T, 3>;
    launch_k(pdl, k, grid_for(work / 2), kThreads, 0, s, t, c, L, phi, guard);
    return;
  }
  if (t.ndim == 2)
    launch_k(pdl, k_restrict<T, 2>, grid_for(work), kThreads, 0, s, t, c, L, phi, guard);
  else
    launch_k(pdl, k_restrict<T, 3>, grid_for(work), kThreads, 0, s, t, c, L, phi, guard);
}

template <typename T>
void launch_prolong(const Topo &t, const Coef<T> &c, const BlockList &L, T *phi, const int *guard,
                    cudaStream_t s, bool pdl) {
  const long work = (long)L.n * t.ncell;
  if (work == 0) return;
  if (t.ndim == 2)
    launch_k(pdl, k_prolong<T, 2>, grid_for(work), kThreads, 0, s, t, c, L, phi, guard);
  else
    launch_k(pdl, k_prolong<T, 3>, grid_for(work), kThreads, 0, s, t, c, L, phi, guard);
}

void launch_flux(const Topo &t, const Coef<double> &c, const BlockList &L, int dir, const double *phi, double *flux,
                 cudaStream_t s) {
  const long work = (long)L.n * t.nfb;
  if (work == 0) return;
  if (t.ndim == 2)
    k_flux<2><<<grid_for(work), kThreads, 0, s>>>(t, c, L, dir, phi, flux);
  else
    k_flux<3><<<grid_for(work), kThreads, 0, s>>>(t, c, L, dir, phi, flux);
}

void launch_fix_bc(const Topo &t, const Coef<double> &c, const BlockList &L, const double *phig, int ng, double *rhs,
                   cudaStream_t s) {
  const long work = (long)L.n * t.ncell;
  if (work == 0) return;
  if (t.ndim == 2)
    k_fix_bc<2><<<grid_for(work), kThreads, 0, s>>>(t, c, L, phig, ng, rhs);
  else
    k_fix_bc<3><<<grid_for(work), kThreads, 0, s>>>(t, c, L, phig, ng, rhs);
}

#define SAYAKA_INST(T)                                                                                          \
  template void launch_face_coef<T>(const Topo &, const double *, const T *[3], const T *[3], double, T *[3],  \
                                    cudaStream_t);                                                              \
  template void launch_apply<T>(const Topo &, const Coef<T> &, const BlockList &, const T *, T *, const T *,   \
                                const int *, cudaStream_t, bool);                                               \
  template void launch_smooth<T>(const Topo &, const Coef<T> &, const BlockList &, int, T *, const T *,        \
                                 const int *, cudaStream_t, bool);                                              \
  template void launch_rbgs<T>(const Topo &, const Coef<T> &, const BlockList &, int, T *, const T *,          \
                               const int *, cudaStream_t, bool, int);                                           \
  template void launch_restrict<T>(const Topo &, const Coef<T> &, const BlockList &, T *, const int *,         \
                                   cudaStream_t, bool);                                                         \
  template void launch_prolong<T>(const Topo &, const Coef<T> &, const BlockList &, T *, const int *,          \
                                  cudaStream_t, bool);                                                          \
  template void launch_prolong_red<T>(const Topo &, const Coef<T> &, const BlockList &, T *, const T *,        \
                                      const int *, cudaStream_t, bool, const BlockList &, int);                 \
  template void launch_bhgs<T>(const Topo &, const Coef<T> &, const BlockList &, int, const T *, T *,          \
                               const T *, const int *, cudaStream_t, bool, int);                                \
  template bool bhgs_prolongs<T>(const Topo &, const Coef<T> &, const BlockList &);
SAYAKA_INST(double)
SAYAKA_INST(float)
#undef SAYAKA_INST

}  // namespace sayaka_gb300
