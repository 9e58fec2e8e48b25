// The smoothing of one tower in one launch (FP32 V-cycle; 2D blocks of 16 or 8
// cells, 3D blocks of 8).
//
// With a launch per colour and level parity, a red-black sweep of a tower of a
// few hundred blocks takes four launches of 3 to 5 us, most of it the launch
// and one round of dependent loads.  Here one cooperative launch holds every
// block of the tower in the registers of a warp (3D: two warps) of its own --
// values, right-hand side, diagonal -- prolongs the top level and runs all sweeps.
// What blocks exchange between half sweeps is the values along their edges:
// each is published as one 64-bit word, the value in its low half and a tag
// in its high half, and the warp that needs it polls the word until the tag
// is the one it expects.  Value and tag arrive together, so a half sweep costs
// one trip through L2 (about 1 us) and needs no fence and no barrier.
//
// Order.  The tag of a cell counts its updates.  With n sweeps the half sweeps
// h = 0 .. 2n-1 alternate red and black, and each runs over parity group 0
// (levels L, L-2, ...) and then over group 1, as the separate launches do.  At
// half sweep h a block reads
//   * a same-level neighbour (the same group) of the other colour, updated
//     (h + 1) / 2 times;
//   * a coarser or finer neighbour (the other group): from group 0 the values
//     after its half sweep h - 1, from group 1 those after half sweep h.
// No word is overwritten before its readers have seen it: an update of it
// needs a value that its readers publish after reading.  The values and
// operations are those of the separate launches in the same order.
//
// Every warp must be resident at once: the launch is cooperative and the host
// only uses it when the tower fits (flow_fits).  A poll gives up after
// `limit` tries, sets the solver's error word and lets its thread run on
// without waiting.  A launch that finds the word set leaves the blocks alone,
// and the solve's loop ends at its next test (k_set_cond) and reports a CUDA
// error, so that one lost word costs one limit and not one per launch to come.
#include <algorithm>

#include "mac_device.h"
#include "mac_flow.h"
#include "mac_stencil.cuh"

namespace sayaka_gb300 {

namespace {

using namespace stencil;
using Word = unsigned long long;

__device__ __forceinline__ void publish(Word *p, float v, unsigned tag) {
  const Word w = ((Word)tag << 32) | __float_as_uint(v);
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ Word look(const Word *p) {
  Word w;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
  return w;
}
__device__ __forceinline__ bool tagged(Word w, unsigned tag) { return (unsigned)(w >> 32) == tag; }
__device__ __forceinline__ float value(Word w) { return __uint_as_float((unsigned)w); }
// the error word of the bounded waits
struct Wait {
  int *err, limit;
};
__device__ __forceinline__ bool given_up(const Topo &t) { return *(volatile const int *)t.err != 0; }
// (unrolled, as the compiler does with a constant limit.  us of a solve of 16
// thousand cells and of one of 1.9 million, with a constant limit and here on the
// same inputs: rolled 1,002 and 1,154, 5,704 and 5,877; by four 1,109 and 1,083,
// 5,832 and 5,879; by eight 1,108 and 1,062, 5,964 and 5,983)
__device__ __forceinline__ float poll1(const Word *p, unsigned tag, Wait wt, bool &dead) {
  Word w = 0;
#pragma unroll 8
  for (int n = 0; n < wt.limit; n++) {
    w = look(p);
    if (tagged(w, tag) || dead) return value(w);
  }
  dead = true;
  atomicExch(wt.err, 1);
  return value(w);
}
// N words, on[i]: wanted (else left alone); all of a round's loads are in
// flight together.  (3D; polling the words one after another took 32 us a
// launch instead of 26, and poll1's unrolled loop in every place 28, for the
// instruction cache.)
template <int N>
__device__ __forceinline__ void poll(const Word *const (&p)[N], const unsigned (&tag)[N], const bool (&on)[N],
                                     float (&x)[N], Wait wt, bool &dead) {
  Word w[N] = {};
  for (int n = dead ? 1 : wt.limit;;) {
    bool all = true;
#pragma unroll
    for (int i = 0; i < N; i++)
      if (on[i]) w[i] = look(p[i]);
#pragma unroll
    for (int i = 0; i < N; i++) all = all && (!on[i] || tagged(w[i], tag[i]));
    if (all) break;
    if (--n > 0) continue;
    if (!dead) atomicExch(wt.err, 1);
    dead = true;
    break;
  }
#pragma unroll
  for (int i = 0; i < N; i++) x[i] = value(w[i]);
}
// the values of the 2 x 2 fine cells behind a refined 3D face, the second row
// `up` words further, times their coefficients, in order; the first has colour
// `odd`.  (Inlined: a call saves and restores the block's registers.)
__device__ __forceinline__ float poll_fine(const Word *p, const float *__restrict__ cf, int up, int odd, unsigned red,
                                           unsigned black, Wait wt, bool &dead) {
  const Word *q[4];
  unsigned tag[4];
  float f[4], v[4], x = 0.f;
  const bool on[4] = {true, true, true, true};
#pragma unroll
  for (int n = 0; n < 4; n++) {
    q[n] = p + (n & 1) + up * (n >> 1);
    f[n] = cf[(n & 1) + up * (n >> 1)];
    tag[n] = ((odd + n + (n >> 1)) & 1) ? black : red;
  }
  poll<4>(q, tag, on, v, wt, dead);
#pragma unroll
  for (int n = 0; n < 4; n++) x += f[n] * v[n];
  return x;
}

// the slots of a block's boundary face cells (16 or 8 per face)
template <int NB>
struct FlowHalo {
  float dp[4 * NB], k[4 * NB], v[4 * NB];
};

// One warp per block.  Lane l holds columns c0 .. c0 + 2Q - 1 of row j, Q of
// them red, Q black; v[colour][q].  Boundary face cells: per colour NB/2 of
// each face, one per lane (2 NB lanes).
template <int NB>
__device__ __forceinline__ void flow_block(const Topo &t, const Coef<float> &c, const int *e, int group, int level,
                                           int nsweep, float *__restrict__ phi, const float *__restrict__ rhs,
                                           Word *__restrict__ words, unsigned tag0, const int *__restrict__ alive,
                                           int limit, int lane, FlowHalo<NB> &sh) {
  constexpr int NC = NB * NB, Q = NB * NB / 64, LPR = 32 / NB;
  const int j = lane / LPR, c0 = (lane % LPR) * 2 * Q;
  const int2 ib = *reinterpret_cast<const int2 *>(e + kHXInfo);
  const int b = ib.y, ft = ib.x & 0xffff;
  const bool top = e[kHXLevel] == level;
  const long cb = (long)b * NC, fb = (long)b * t.nfb;
  const float *u = uniform_of(c, b);
  const float dv = geom(c, b, 6);
  const int pr = j & 1;  // red cells of the row: columns 2q + pr
  float pv[2 * Q], rv[2 * Q], wv[2 * Q];
  auto load = [&](const float *p, float(&a)[2 * Q]) {
    if constexpr (Q == 4) {
      const float4 x = reinterpret_cast<const float4 *>(p)[0], y = reinterpret_cast<const float4 *>(p)[1];
      a[0] = x.x, a[1] = x.y, a[2] = x.z, a[3] = x.w, a[4] = y.x, a[5] = y.y, a[6] = y.z, a[7] = y.w;
    } else {
      const float2 x = *reinterpret_cast<const float2 *>(p);
      a[0] = x.x, a[1] = x.y;
    }
  };
  load(rhs + cb + NB * j + c0, rv);
  if (top) {
    const int pw = e[kHXPar + 6], wc = pw & 7;
    const float *q = phi + (long)(pw >> 3) * NC + (NB / 2) * (wc & 1) + c0 / 2 +
                     NB * ((NB / 2) * ((wc >> 1) & 1) + (j >> 1));
#pragma unroll
    for (int n = 0; n < Q; n++) pv[2 * n] = pv[2 * n + 1] = q[n];
  } else {
    load(phi + cb + NB * j + c0, pv);
  }
  float v[2][Q], kl[2][Q], kr[2][Q], kd[2][Q], ku[2][Q], diag[2][Q], rd[2][Q], vf[2][Q];
  if (u) {
    const float T0 = u[0], T1 = u[1];
#pragma unroll
    for (int n = 0; n < 2 * Q; n++) wv[n] = 1.f;
#pragma unroll
    for (int k = 0; k < 2; k++)
#pragma unroll
      for (int q = 0; q < Q; q++) kl[k][q] = kr[k][q] = T0, kd[k][q] = ku[k][q] = T1;
  } else {
    const float *x = c.tff[0] + fb + (NB + 1) * j + c0, *y = c.tff[1] + fb + NB * j + c0;
    load(c.vf + cb + NB * j + c0, wv);
#pragma unroll
    for (int k = 0; k < 2; k++)
#pragma unroll
      for (int q = 0; q < Q; q++) {
        const int i = 2 * q + (k ? 1 - pr : pr);
        kl[k][q] = x[i], kr[k][q] = x[i + 1], kd[k][q] = y[i], ku[k][q] = y[i + NB];
      }
  }
#pragma unroll
  for (int q = 0; q < Q; q++) {
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const bool odd = k ? !pr : pr;
      vf[k][q] = odd ? wv[2 * q + 1] : wv[2 * q];
      v[k][q] = odd ? pv[2 * q + 1] : pv[2 * q];
      rd[k][q] = (odd ? rv[2 * q + 1] : rv[2 * q]) * dv;
      if (top && !(vf[k][q] > 0.f)) v[k][q] = 0.f;
    }
  }
  // this lane's boundary face cell of each colour: what to poll
  struct Slot {
    const Word *w;   // the neighbour's word (refined face: the first of two)
    float f0, f1;    // refined face: the fine cells' coefficients
    int ty, odd;     // face type (1: nothing to poll); colour of the (first) polled cell
  } slot[2];
  constexpr int HF = NB / 2;  // boundary cells of one colour per face
  const int hf = lane / HF;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    Slot &s = slot[k];
    s.ty = 1;
    s.w = nullptr;
    s.f0 = s.f1 = 0.f;
    s.odd = 0;
    if (lane >= 4 * HF) continue;
    const int d = hf >> 1, side = hf & 1, m = 2 * (lane % HF) + ((k + side) & 1), across = side ? 0 : NB - 1;
    const long cfr = ((long)b * 4 + hf) * NB + m;
    float dp = 0.f, kk = 0.f;
    s.ty = (ft >> (2 * hf)) & 3;
    if (s.ty == 0) {
      const int fx = d ? m + NB * (side * NB) : side * NB + (NB + 1) * m;
      dp = kk = u ? u[d] : (d ? c.tff[1] : c.tff[0])[fb + fx];
      s.w = words + ((long)e[hf] * 4 + (hf ^ 1)) * NB + m;
      if (alive && !alive[e[hf]]) s.ty = 1;  // a solid block is not in a reduced list: its values are 0
    } else if (s.ty == 1) {
      const int fx = d ? m + NB * (side * NB) : side * NB + (NB + 1) * m;
      if (t.bc_type[b * 6 + hf] != kBCNeumann) dp = (u ? u[d] : (d ? c.tff[1] : c.tff[0])[fb + fx]) * 2.0f;
    } else if (s.ty == 2) {
      const int tc = HF * ((ib.x >> (17 - d)) & 1) + (m >> 1);  // which_child >> (1 - d)
      dp = kk = c.cf[cfr];
      s.w = words + ((long)e[hf] * 4 + (hf ^ 1)) * NB + tc;
      s.odd = (across + tc) & 1;
      if (alive && !alive[e[hf]]) s.ty = 1;
    } else {
      const int half = m / HF, F = e[kHXKids + 4 * hf + half], t0 = 2 * (m - HF * half);
      const long r = ((long)F * 4 + (hf ^ 1)) * NB + t0;
      dp = c.cf[cfr];
      kk = 1.f;
      s.w = words + r;
      s.f0 = c.cf[r];
      s.f1 = c.cf[r + 1];
      s.odd = (across + t0) & 1;
      if (alive && !alive[F]) s.ty = 1;
    }
    sh.dp[NB * hf + m] = dp;
    sh.k[NB * hf + m] = kk;
    sh.v[NB * hf + m] = 0.f;
  }
  // the block's own words: lane's cells on the edges, after `ver` updates
  auto give = [&](int k, unsigned ver) {
    const int pk = k ? 1 - pr : pr;
#pragma unroll
    for (int q = 0; q < Q; q++) {
      const int i = c0 + 2 * q + pk;
      Word *w = words + (long)b * 4 * NB;
      if (q == 0 && i == 0) publish(w + j, v[k][q], tag0 + ver);
      if (q == Q - 1 && i == NB - 1) publish(w + NB + j, v[k][q], tag0 + ver);
      if (j == 0) publish(w + 2 * NB + i, v[k][q], tag0 + ver);
      if (j == NB - 1) publish(w + 3 * NB + i, v[k][q], tag0 + ver);
    }
  };
  give(0, 0);
  give(1, 0);
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 2; k++)
#pragma unroll
    for (int q = 0; q < Q; q++) {
      const int i = c0 + 2 * q + (k ? 1 - pr : pr);
      float dl = kl[k][q], dr = kr[k][q], dd = kd[k][q], du = ku[k][q];
      if (q == 0 && i == 0) dl = sh.dp[j], kl[k][q] = sh.k[j];
      if (q == Q - 1 && i == NB - 1) dr = sh.dp[NB + j], kr[k][q] = sh.k[NB + j];
      if (j == 0) dd = sh.dp[2 * NB + i], kd[k][q] = sh.k[2 * NB + i];
      if (j == NB - 1) du = sh.dp[3 * NB + i], ku[k][q] = sh.k[3 * NB + i];
      float g = c.alpha * dv;
      g += dl;
      g += dr;
      g += dd;
      g += du;
      diag[k][q] = vf[k][q] > 0.f ? g : 0.f;  // 0: the cell stays at 0
    }
  bool dead = false;
  const Wait wt{t.err, limit};
  for (int s = 0; s < nsweep; s++) {
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const int h = 2 * s + k;
      const Slot &sl = slot[k];
      if (sl.ty != 1) {
        // updates of the red and black cells that the other group has done
        const unsigned cross_red = group ? (h >> 1) + 1 : (h + 1) >> 1, cross_black = group ? (h + 1) >> 1 : h >> 1;
        float x;
        if (sl.ty == 0) {
          x = poll1(sl.w, tag0 + ((h + 1) >> 1), wt, dead);
        } else if (sl.ty == 2) {
          x = poll1(sl.w, tag0 + (sl.odd ? cross_black : cross_red), wt, dead);
        } else {
          const float x0 = poll1(sl.w, tag0 + (sl.odd ? cross_black : cross_red), wt, dead);
          const float x1 = poll1(sl.w + 1, tag0 + (sl.odd ? cross_red : cross_black), wt, dead);
          x = 0.f;
          x += sl.f0 * x0;
          x += sl.f1 * x1;
        }
        sh.v[NB * hf + 2 * (lane % HF) + ((k + (hf & 1)) & 1)] = x;
      }
      __syncwarp();
      const int pk = k ? 1 - pr : pr;
      const float(&o)[Q] = v[1 - k];
      const float fl = __shfl_up_sync(0xffffffffu, o[Q - 1], 1), fr = __shfl_down_sync(0xffffffffu, o[0], 1);
      float nd[Q], nu[Q];
#pragma unroll
      for (int q = 0; q < Q; q++) {
        nd[q] = __shfl_up_sync(0xffffffffu, o[q], LPR);
        nu[q] = __shfl_down_sync(0xffffffffu, o[q], LPR);
      }
#pragma unroll
      for (int q = 0; q < Q; q++) {
        const int i = c0 + 2 * q + pk;
        float vl = pk ? o[q] : (q > 0 ? o[q > 0 ? q - 1 : 0] : fl);
        float vr = pk ? (q < Q - 1 ? o[q < Q - 1 ? q + 1 : q] : fr) : o[q];
        float vd = nd[q], vu = nu[q];
        if (q == 0 && i == 0) vl = sh.v[j];
        if (q == Q - 1 && i == NB - 1) vr = sh.v[NB + j];
        if (j == 0) vd = sh.v[2 * NB + i];
        if (j == NB - 1) vu = sh.v[3 * NB + i];
        float off = 0.f;
        off = fma_t(kl[k][q], vl, off);
        off = fma_t(kr[k][q], vr, off);
        off = fma_t(kd[k][q], vd, off);
        off = fma_t(ku[k][q], vu, off);
        v[k][q] = diag[k][q] > 0.f
                      ? relax(c.omega, fast_div(fma_t(rd[k][q], vf[k][q], off), diag[k][q]), v[k][q])
                      : 0.f;
      }
      give(k, s + 1);
      __syncwarp();  // the slots are read before the next half sweep fills them
    }
  }
  float *dst = phi + cb + NB * j + c0;
#pragma unroll
  for (int q = 0; q < Q; q += 2) {
    const float a0 = v[0][q], b0 = v[1][q];
    if constexpr (Q == 1) {
      *reinterpret_cast<float2 *>(dst) = pr ? make_float2(b0, a0) : make_float2(a0, b0);
    } else {
      const float a1 = v[0][q + 1 < Q ? q + 1 : q], b1 = v[1][q + 1 < Q ? q + 1 : q];
      *reinterpret_cast<float4 *>(dst + 2 * q) = pr ? make_float4(b0, a0, b1, a1) : make_float4(a0, b0, a1, b1);
    }
  }
}

// one warp (and CTA) per entry of the tower's parity groups A and B
template <int NB>
__global__ void __launch_bounds__(32, 16) k_flow(Topo t, Coef<float> c, BlockList A, BlockList B, int level, int nsweep,
                                             float *__restrict__ phi, const float *__restrict__ rhs, const int *guard,
                                             Word *__restrict__ words, unsigned *epoch,
                                             const int *__restrict__ alive, int limit) {
  __shared__ FlowHalo<NB> sh;
  const bool gone = given_up(t);  // in flight with the loads that follow
  if (guard && *guard) return;
  const unsigned tag0 = epoch[0] * kFlowTags + 1;
  const ListRange ar = list_range(A), br = list_range(B);
  const int na = ar.b - ar.a, n = na + br.b - br.a, p = blockIdx.x;
  if (!__any_sync(0xffffffffu, gone) && p < n) {
    const bool ga = p < na;
    const BlockList &L = ga ? A : B;
    const int *e = L.hx + (long)(ga ? ar.a + p : br.a + p - na) * kHX;
    if (!(L.stc && block_off(L, e[kHXBlock])))  // a problem's blocks are off together
      flow_block<NB>(t, c, e, ga ? 0 : 1, level, nsweep, phi, rhs, words, tag0, alive, limit, threadIdx.x, sh);
  }
  // the next launch's tags: every CTA has read epoch[0] before it counts
  if (threadIdx.x == 0 && atomicAdd(&epoch[1], 1u) == gridDim.x - 1) {
    epoch[1] = 0;
    epoch[0] += 1;
  }
}

// ---- 3D blocks of 8^3 cells: one CTA of 64 threads per block, a thread per
// row of cells along x.  The tile in shared memory is split by colour and
// padded by a layer of rows for the values across the y and z faces, as in
// k_bhgs_rows; those across the x faces have their own array.  A thread polls
// three boundary face cells per colour, one per direction.
struct Flow3Halo {
  static constexpr int kRows = 100;  // (8 + 2)^2
  float4 tile[2][kRows];             // [colour][row]: the row's four cells of the colour
  float dp[6][64], k[6][64];
  float hx[2][2][64];                // [colour of the cell][side][row]: value across the x face
  static __device__ __forceinline__ int row(int j, int k) { return j + 1 + 10 * (k + 1); }
};

// a polled boundary face cell
struct Flow3Slot {
  const Word *w;    // the neighbour's word; refined face: the first of 2 x 2
  const float *cf;  // refined face: its coefficients
  int ty, odd;      // face type (1: nothing to poll); colour of the (first) polled cell
};

// boundary face cell (a0, a1) of coarse/fine face f: what to poll, its part of
// the diagonal and its factor
struct Flow3Setup {
  Flow3Slot s;
  float dp, k;
};
__device__ __forceinline__ Flow3Setup flow3_slot(const int *__restrict__ e, const float *__restrict__ cf,
                                                 const Word *words, const int *__restrict__ alive, int f, int a0,
                                                 int a1) {
  constexpr int NB = 8, NF = 64;
  const int d = f >> 1, info = e[kHXInfo], b = e[kHXBlock], m = a0 + NB * a1, across = (f & 1) ? 0 : NB - 1;
  Flow3Setup r;
  r.s.ty = (info >> (2 * f)) & 3;
  r.dp = r.k = cf[((long)b * 6 + f) * NF + m];
  int n = e[f];
  if (r.s.ty == 2) {
    const int wc = info >> 16, q0 = d == 0 ? 1 : 0, q1 = d == 2 ? 1 : 2;
    const int t0 = 4 * ((wc >> q0) & 1) + (a0 >> 1), t1 = 4 * ((wc >> q1) & 1) + (a1 >> 1);
    r.s.w = words + ((long)n * 6 + (f ^ 1)) * NF + t0 + NB * t1;
    r.s.cf = nullptr;
    r.s.odd = (across + t0 + t1) & 1;
  } else {
    const int h0 = a0 >> 2, h1 = a1 >> 2;
    n = e[kHXKids + 4 * f + h0 + 2 * h1];
    const long o = ((long)n * 6 + (f ^ 1)) * NF + 2 * (a0 - 4 * h0) + NB * 2 * (a1 - 4 * h1);
    r.k = 1.f;
    r.s.w = words + o;
    r.s.cf = cf + o;
    r.s.odd = across & 1;  // the first fine cell's transverse indices are even
  }
  if (alive && !alive[n]) r.s.ty = 1;
  return r;
}

__device__ __forceinline__ void flow3_block(const Topo &t, const Coef<float> &c, const int *e, int group, int level,
                                            int nsweep, float *__restrict__ phi, const float *__restrict__ rhs,
                                            Word *__restrict__ words, unsigned tag0, const int *__restrict__ alive,
                                            int limit, Flow3Halo &sh) {
  constexpr int NB = 8, NC = 512, NF = 64, Q = 4;
  const int tid = threadIdx.x, j = tid & 7, k3 = tid >> 3, pr = (j + k3) & 1;
  const int info = e[kHXInfo], b = e[kHXBlock];
  const bool top = e[kHXLevel] == level;
  const long cb = (long)b * NC, fb = (long)b * t.nfb;
  const float dv = geom(c, b, 6);
  const float *u = uniform_of(c, b);  // uniform over the CTA
  const bool U = u != nullptr;
  const float T0 = U ? u[0] : 0.f, T1 = U ? u[1] : 0.f, T2 = U ? u[2] : 0.f;
  const float *fx = c.tff[0] + fb + (NB + 1) * (j + NB * k3);
  const float *fy = c.tff[1] + fb + NB * (j + (NB + 1) * k3);
  const float *fz = c.tff[2] + fb + NB * (j + NB * k3);
  const float *vfp = c.vf + cb + NB * tid;
  const int r = Flow3Halo::row(j, k3);
  float v[2][Q], rd[2][Q], dg[2][Q];
  {
    const float4 a = reinterpret_cast<const float4 *>(rhs + cb + NB * tid)[0],
                 d = reinterpret_cast<const float4 *>(rhs + cb + NB * tid)[1];
    const float rv[8] = {a.x, a.y, a.z, a.w, d.x, d.y, d.z, d.w};
    float pv[8];
    if (top) {
      const int pw = e[kHXPar + 6], wc = pw & 7;
      const float4 q = *reinterpret_cast<const float4 *>(phi + (long)(pw >> 3) * NC + 4 * (wc & 1) +
                                                          NB * (4 * ((wc >> 1) & 1) + (j >> 1) +
                                                                NB * (4 * ((wc >> 2) & 1) + (k3 >> 1))));
      pv[0] = pv[1] = q.x, pv[2] = pv[3] = q.y, pv[4] = pv[5] = q.z, pv[6] = pv[7] = q.w;
      if (!U) {
#pragma unroll
        for (int n = 0; n < 8; n++)
          if (!(vfp[n] > 0.f)) pv[n] = 0.f;
      }
    } else {
      const float4 p = reinterpret_cast<const float4 *>(phi + cb + NB * tid)[0],
                   q = reinterpret_cast<const float4 *>(phi + cb + NB * tid)[1];
      pv[0] = p.x, pv[1] = p.y, pv[2] = p.z, pv[3] = p.w, pv[4] = q.x, pv[5] = q.y, pv[6] = q.z, pv[7] = q.w;
    }
#pragma unroll
    for (int q = 0; q < Q; q++) {
      v[0][q] = pr ? pv[2 * q + 1] : pv[2 * q];
      v[1][q] = pr ? pv[2 * q] : pv[2 * q + 1];
      rd[0][q] = (pr ? rv[2 * q + 1] : rv[2 * q]) * dv;
      rd[1][q] = (pr ? rv[2 * q] : rv[2 * q + 1]) * dv;
    }
  }
  // the block's own words: the row's cells of colour k on the block's faces
  auto give = [&](int k, unsigned ver) {
    const int pk = k ? 1 - pr : pr;
    Word *w = words + (long)b * 6 * NF;
    if (!pk) publish(w + tid, v[k][0], tag0 + ver);
    if (pk) publish(w + NF + tid, v[k][Q - 1], tag0 + ver);
#pragma unroll
    for (int q = 0; q < Q; q++) {
      const int i = 2 * q + pk;
      if (j == 0) publish(w + 2 * NF + i + NB * k3, v[k][q], tag0 + ver);
      if (j == NB - 1) publish(w + 3 * NF + i + NB * k3, v[k][q], tag0 + ver);
      if (k3 == 0) publish(w + 4 * NF + i + NB * j, v[k][q], tag0 + ver);
      if (k3 == NB - 1) publish(w + 5 * NF + i + NB * j, v[k][q], tag0 + ver);
    }
  };
  give(0, 0);
  give(1, 0);
#pragma unroll
  for (int k = 0; k < 2; k++) sh.tile[k][r] = make_float4(v[k][0], v[k][1], v[k][2], v[k][3]);
  // boundary face cells: thread (side, a1, n) of direction d, both colours
  const int side = tid >> 5, a1 = (tid & 31) >> 2;
  Flow3Slot slot[2][3];
#pragma unroll
  for (int k = 0; k < 2; k++)
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const int f = 2 * d + side, fixed = side ? NB - 1 : 0;
      const int a0 = 2 * (tid & 3) + ((k + fixed + a1) & 1), m = a0 + NB * a1;
      const int fidx = d == 0   ? fixed + side + (NB + 1) * m
                       : d == 1 ? a0 + NB * (fixed + side + (NB + 1) * a1)
                                : m + NB * NB * (fixed + side);
      const float T = U ? (d == 0 ? T0 : d == 1 ? T1 : T2) : c.tff[d][fb + fidx];
      const int ty = (info >> (2 * f)) & 3;
      Flow3Setup r3;
      if (ty <= 1) {
        const int n = e[f];
        r3.s = Flow3Slot{words + ((long)n * 6 + (f ^ 1)) * NF + m, nullptr, ty, 0};
        r3.dp = r3.k = T;
        if (ty == 0 && alive && !alive[n]) r3.s.ty = 1;  // a solid block is not in a reduced list: its values are 0
        if (ty == 1) {
          r3.dp = t.bc_type[b * 6 + f] != kBCNeumann ? T * 2.0f : 0.f;
          r3.k = 0.f;
        }
      } else {
        r3 = flow3_slot(e, c.cf, words, alive, f, a0, a1);
      }
      slot[k][d] = r3.s;
      sh.dp[f][m] = r3.dp;
      sh.k[f][m] = r3.k;
      // (solid and physical neighbours stay at 0)
      if (d == 0)
        sh.hx[k][side][m] = 0.f;
      else
        reinterpret_cast<float *>(&sh.tile[1 - k][d == 1 ? Flow3Halo::row(side ? NB : -1, a1)
                                                         : Flow3Halo::row(a1, side ? NB : -1)])[a0 >> 1] = 0.f;
    }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 2; k++)
#pragma unroll
    for (int q = 0; q < Q; q++) {
      const int i = 2 * q + (k ? 1 - pr : pr);
      float g = c.alpha * dv;
      g += q == 0 && i == 0 ? sh.dp[0][tid] : (U ? T0 : fx[i]);
      g += q == Q - 1 && i == NB - 1 ? sh.dp[1][tid] : (U ? T0 : fx[i + 1]);
      g += j == 0 ? sh.dp[2][i + NB * k3] : (U ? T1 : fy[i]);
      g += j == NB - 1 ? sh.dp[3][i + NB * k3] : (U ? T1 : fy[i + NB]);
      g += k3 == 0 ? sh.dp[4][i + NB * j] : (U ? T2 : fz[i]);
      g += k3 == NB - 1 ? sh.dp[5][i + NB * j] : (U ? T2 : fz[i + NB * NB]);
      if (!U && !(vfp[i] > 0.f)) g = 0.f;  // 0: the cell stays at 0
      dg[k][q] = g;
    }
  bool dead = false;
  const Wait wt{t.err, limit};
  for (int s = 0; s < nsweep; s++) {
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const int h = 2 * s + k;
      const unsigned cross_red = tag0 + (group ? (h >> 1) + 1 : (h + 1) >> 1);
      const unsigned cross_black = tag0 + (group ? (h + 1) >> 1 : h >> 1);
      const Word *p[3];
      unsigned tag[3];
      bool on[3];
      float got[3];
#pragma unroll
      for (int d = 0; d < 3; d++) {
        const Flow3Slot &sl = slot[k][d];
        p[d] = sl.w;
        on[d] = sl.ty == 0 || sl.ty == 2;
        tag[d] = sl.ty == 0 ? tag0 + ((h + 1) >> 1) : (sl.odd ? cross_black : cross_red);
      }
      poll<3>(p, tag, on, got, wt, dead);
#pragma unroll
      for (int d = 0; d < 3; d++) {
        const Flow3Slot &sl = slot[k][d];
        if (sl.ty == 1) continue;
        float x = got[d];
        if (sl.ty == 3) x = poll_fine(sl.w, sl.cf, NB, sl.odd, cross_red, cross_black, wt, dead);
        const int a0 = 2 * (tid & 3) + ((k + (side ? NB - 1 : 0) + a1) & 1), m = a0 + NB * a1;
        if (d == 0)
          sh.hx[k][side][m] = x;
        else
          reinterpret_cast<float *>(&sh.tile[1 - k][d == 1 ? Flow3Halo::row(side ? NB : -1, a1)
                                                           : Flow3Halo::row(a1, side ? NB : -1)])[a0 >> 1] = x;
      }
      __syncthreads();
      const int pk = k ? 1 - pr : pr;
      const float(&o)[Q] = v[1 - k];
      const float4 d4 = sh.tile[1 - k][r - 1], u4 = sh.tile[1 - k][r + 1];
      const float4 b4 = sh.tile[1 - k][r - 10], f4 = sh.tile[1 - k][r + 10];
      const float vd[4] = {d4.x, d4.y, d4.z, d4.w}, vu[4] = {u4.x, u4.y, u4.z, u4.w};
      const float vb[4] = {b4.x, b4.y, b4.z, b4.w}, vz[4] = {f4.x, f4.y, f4.z, f4.w};
#pragma unroll
      for (int q = 0; q < Q; q++) {
        const int i = 2 * q + pk;
        float vl = pk ? o[q] : (q > 0 ? o[q > 0 ? q - 1 : 0] : sh.hx[k][0][tid]);
        float vr = pk ? (q < Q - 1 ? o[q < Q - 1 ? q + 1 : q] : sh.hx[k][1][tid]) : o[q];
        const float kl = q == 0 && i == 0 ? sh.k[0][tid] : (U ? T0 : fx[i]);
        const float kr = q == Q - 1 && i == NB - 1 ? sh.k[1][tid] : (U ? T0 : fx[i + 1]);
        float off = 0.f;
        off = fma_t(kl, vl, off);
        off = fma_t(kr, vr, off);
        off = fma_t(j == 0 ? sh.k[2][i + NB * k3] : (U ? T1 : fy[i]), vd[q], off);
        off = fma_t(j == NB - 1 ? sh.k[3][i + NB * k3] : (U ? T1 : fy[i + NB]), vu[q], off);
        off = fma_t(k3 == 0 ? sh.k[4][i + NB * j] : (U ? T2 : fz[i]), vb[q], off);
        off = fma_t(k3 == NB - 1 ? sh.k[5][i + NB * j] : (U ? T2 : fz[i + NB * NB]), vz[q], off);
        const float g = dg[k][q];
        v[k][q] = g > 0.f ? relax(c.omega, fast_div(fma_t(rd[k][q], U ? 1.f : vfp[i], off), g), v[k][q]) : 0.f;
      }
      sh.tile[k][r] = make_float4(v[k][0], v[k][1], v[k][2], v[k][3]);
      give(k, s + 1);
    }
  }
  float4 *dst = reinterpret_cast<float4 *>(phi + cb + NB * tid);
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const float a0 = v[0][2 * h], a1_ = v[0][2 * h + 1], b0 = v[1][2 * h], b1 = v[1][2 * h + 1];
    dst[h] = pr ? make_float4(b0, a0, b1, a1_) : make_float4(a0, b0, a1_, b1);
  }
}

__global__ void __launch_bounds__(64, 8) k_flow3(Topo t, Coef<float> c, BlockList A, BlockList B, int level, int nsweep,
                                                 float *__restrict__ phi, const float *__restrict__ rhs,
                                                 const int *guard, Word *__restrict__ words, unsigned *epoch,
                                                 const int *__restrict__ alive, int limit) {
  __shared__ Flow3Halo sh;
  const bool gone = given_up(t);  // in flight with the loads that follow
  if (guard && *guard) return;
  const unsigned tag0 = epoch[0] * kFlowTags + 1;
  const ListRange ar = list_range(A), br = list_range(B);
  const int na = ar.b - ar.a, n = na + br.b - br.a, p = blockIdx.x;
  if (!__syncthreads_or(gone) && p < n) {
    const bool ga = p < na;
    const BlockList &L = ga ? A : B;
    const int *e = L.hx + (long)(ga ? ar.a + p : br.a + p - na) * kHX;
    if (!(L.stc && block_off(L, e[kHXBlock]))) {
      flow3_block(t, c, e, ga ? 0 : 1, level, nsweep, phi, rhs, words, tag0, alive, limit, sh);
    }
  }
  __syncthreads();  // every thread has read epoch[0]
  if (threadIdx.x == 0 && atomicAdd(&epoch[1], 1u) == gridDim.x - 1) {
    epoch[1] = 0;
    epoch[0] += 1;
  }
}

using FlowKernel = void (*)(Topo, Coef<float>, BlockList, BlockList, int, int, float *, const float *, const int *,
                            Word *, unsigned *, const int *, int);
struct FlowForm {
  FlowKernel kernel;
  int threads;  // per block
};
FlowForm flow_form(const Topo &t) {
  if (t.ndim == 2 && t.nb == 16) return {k_flow<16>, 32};
  if (t.ndim == 2 && t.nb == 8) return {k_flow<8>, 32};
  if (t.ndim == 3 && t.nb == 8) return {k_flow3, 64};
  return {nullptr, 0};
}

}  // namespace

int flow_capacity(const Topo &t) {
  const FlowForm f = flow_form(t);
  if (!f.kernel) return 0;
  int dev = 0, sms = 0, per = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, (const void *)f.kernel, f.threads, 0) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return sms * per;
}

size_t flow_words(const Topo &t) {
  return (size_t)t.nblocks * 2 * t.ndim * (t.ndim == 3 ? t.nb * t.nb : t.nb);
}

cudaError_t launch_flow(const Topo &t, const Coef<float> &c, const BlockList &A, const BlockList &B, int level,
                        int nsweep, int grid, float *phi, const float *rhs, const int *guard,
                        unsigned long long *words, unsigned *epoch, const int *alive, cudaStream_t s, int limit) {
  const FlowForm f = flow_form(t);
  if (!f.kernel) return cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(f.threads);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, f.kernel, t, c, A, B, level, nsweep, phi, rhs, guard, words, epoch, alive,
                            limit);
}

}  // namespace sayaka_gb300
