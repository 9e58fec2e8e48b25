// The smoothing of one tower in one launch (2D, FP32 V-cycle).
//
// With a launch per colour and level parity, a red-black sweep of a tower of a
// few hundred blocks takes four launches of 3 to 5 us, most of it the launch
// and one round of dependent loads.  Here one cooperative launch holds every
// block of the tower in the registers of a warp of its own -- values,
// coefficients, right-hand side -- prolongs the top level and runs all sweeps.
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
// kPollLimit tries, sets the solver's error word (the solve then reports a
// CUDA error) and lets the warp run on without waiting.
#include <algorithm>

#include "mac_device.h"
#include "mac_flow.h"
#include "mac_stencil.cuh"

namespace sayaka_gb300 {

namespace {

using namespace stencil;
using Word = unsigned long long;

constexpr int kPollLimit = 1 << 20;  // about half a second

__device__ __forceinline__ void publish(Word *p, float v, unsigned tag) {
  const Word w = ((Word)tag << 32) | __float_as_uint(v);
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ float poll(const Word *p, unsigned tag, int *err, bool &dead) {
  Word w = 0;
  for (int n = 0; n < kPollLimit; n++) {
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
    if ((unsigned)(w >> 32) == tag || dead) return __uint_as_float((unsigned)w);
  }
  dead = true;
  atomicExch(err, 1);
  return __uint_as_float((unsigned)w);
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
                                           int lane, FlowHalo<NB> &sh) {
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
          x = poll(sl.w, tag0 + ((h + 1) >> 1), t.err, dead);
        } else if (sl.ty == 2) {
          x = poll(sl.w, tag0 + (sl.odd ? cross_black : cross_red), t.err, dead);
        } else {
          const float x0 = poll(sl.w, tag0 + (sl.odd ? cross_black : cross_red), t.err, dead);
          const float x1 = poll(sl.w + 1, tag0 + (sl.odd ? cross_red : cross_black), t.err, dead);
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
                                             const int *__restrict__ alive) {
  __shared__ FlowHalo<NB> sh;
  if (guard && *guard) return;
  const unsigned tag0 = epoch[0] * kFlowTags + 1;
  const ListRange ar = list_range(A), br = list_range(B);
  const int na = ar.b - ar.a, n = na + br.b - br.a, p = blockIdx.x;
  if (p < n) {
    const bool ga = p < na;
    const BlockList &L = ga ? A : B;
    const int *e = L.hx + (long)(ga ? ar.a + p : br.a + p - na) * kHX;
    if (!(L.stc && block_off(L, e[kHXBlock])))  // a problem's blocks are off together
      flow_block<NB>(t, c, e, ga ? 0 : 1, level, nsweep, phi, rhs, words, tag0, alive, threadIdx.x, sh);
  }
  // the next launch's tags: every CTA has read epoch[0] before it counts
  if (threadIdx.x == 0 && atomicAdd(&epoch[1], 1u) == gridDim.x - 1) {
    epoch[1] = 0;
    epoch[0] += 1;
  }
}

const void *flow_kernel(int nb) {
  return nb == 16 ? (const void *)k_flow<16> : (const void *)k_flow<8>;
}

}  // namespace

int flow_capacity(const Topo &t) {
  if (t.ndim != 2 || (t.nb != 16 && t.nb != 8)) return 0;
  int dev = 0, sms = 0, per = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, flow_kernel(t.nb), 32, 0) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return sms * per;
}

size_t flow_words(const Topo &t) { return (size_t)t.nblocks * 4 * t.nb; }

cudaError_t launch_flow(const Topo &t, const Coef<float> &c, const BlockList &A, const BlockList &B, int level,
                        int nsweep, float *phi, const float *rhs, const int *guard, unsigned long long *words,
                        unsigned *epoch, const int *alive, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(A.n + B.n);
  cfg.blockDim = dim3(32);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (t.nb == 16) return cudaLaunchKernelEx(&cfg, k_flow<16>, t, c, A, B, level, nsweep, phi, rhs, guard, words, epoch,
                                             alive);
  return cudaLaunchKernelEx(&cfg, k_flow<8>, t, c, A, B, level, nsweep, phi, rhs, guard, words, epoch,
                                             alive);
}

}  // namespace sayaka_gb300
