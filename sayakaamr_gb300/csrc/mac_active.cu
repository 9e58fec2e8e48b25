// Active blocks of the device solve.
//
// A block whose cells are all solid (vf = 0) takes no part in a solve: the
// right-hand side is masked there, the smoother and the prolongation hold it
// at 0 and the operator gives 0, so every vector of the iteration is 0 on it
// and adds nothing to a dot product or a norm.  In a domain that is mostly
// body -- the elbow pipe in its box: 19,154 of 26,860 leaf blocks -- the
// V-cycle would spend most of its work writing those zeros again.
//
// The block lists that the captured iteration walks are therefore kept in a
// second, reduced form: the same entries in the same order without the solid
// blocks, with the number of entries before every place of the full list
// (pre), so that any segment [a, b) of a list is [pre[a], pre[b]) of the
// reduced one.  Kernels read the two bounds from device memory, so the lists
// follow a moving body by one scan and one copy per coefficient change and
// the captured graph stays valid.
//
// The reduced lists are used when at least a quarter of the finest tower's
// blocks are solid (kActiveShare): a launch pays one dependent load for the
// bounds, about 0.4 us, which a launch-bound solve without solid blocks would
// lose.  Their memory, about 170 bytes an entry of every list, is allocated
// when that share is first reached; where it cannot be had, the solve walks the
// full lists.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "cuda_check.h"
#include "dev_alloc.h"
#include "mac_solver.h"

namespace sayaka_gb300 {

namespace {

constexpr int kScanThreads = 1024;
// reduced lists from a share of 1/kActiveShare solid blocks on
constexpr int kActiveShare = 4;

// one warp per block: does any cell hold fluid
__global__ void __launch_bounds__(256) k_block_active(int nblocks, int ncell, const double *__restrict__ vf,
                                                     int *__restrict__ flag) {
  const int lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
  for (int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < nblocks; b += warps) {
    bool any = false;
    for (int i = lane; i < ncell; i += 32) any = any || vf[(long)b * ncell + i] > 0;
    any = __any_sync(0xffffffffu, any);
    if (lane == 0) flag[b] = any;
  }
}

// one CTA per list: pre[p] = active entries before p (p <= n), orig[k] = full
// place of the k-th active entry; order kept
__global__ void __launch_bounds__(kScanThreads) k_active_scan(const ActiveList *__restrict__ lists,
                                                             const int *__restrict__ flag) {
  __shared__ int warp_sum[kScanThreads / 32];
  __shared__ int base;
  const ActiveList l = lists[blockIdx.x];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x == 0) base = 0;
  __syncthreads();
  for (int p0 = 0; p0 < l.n; p0 += kScanThreads) {
    const int p = p0 + threadIdx.x;
    const bool on = p < l.n && flag[l.blocks[p]] != 0;
    const unsigned m = __ballot_sync(0xffffffffu, on);
    if (lane == 0) warp_sum[w] = __popc(m);
    __syncthreads();
    int before = base;
    for (int q = 0; q < w; q++) before += warp_sum[q];
    const int k = before + __popc(m & ((1u << lane) - 1u));
    if (p < l.n) l.pre[p] = k;
    if (on) l.orig[k] = p;
    __syncthreads();
    if (threadIdx.x == kScanThreads - 1) base = k + (on ? 1 : 0);
    __syncthreads();
  }
  if (threadIdx.x == 0) l.pre[l.n] = base;
}

// the active entries' block ids, face types, halo descriptors and links
__global__ void __launch_bounds__(256) k_active_copy(const ActiveList *__restrict__ lists) {
  const ActiveList l = lists[blockIdx.y];
  const int n = l.pre[l.n], step = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
  for (int k = t0; k < n; k += step) {
    const int p = l.orig[k];
    l.ablocks[k] = l.blocks[p];
    if (l.ftypes) l.aftypes[k] = l.ftypes[p];
  }
  if (l.hx)
    for (long i = t0; i < (long)n * kHX; i += step) l.ahx[i] = l.hx[(long)l.orig[i / kHX] * kHX + i % kHX];
  if (l.links)
    for (long i = t0; i < (long)n * l.nlinks; i += step)
      l.alinks[i] = l.links[(long)l.orig[i / l.nlinks] * l.nlinks + i % l.nlinks];
}

// count[0], count[1]: the active blocks of the finest tower, and those of them
// with one face coefficient (see k_iso); zeroed by the caller
__global__ void __launch_bounds__(kScanThreads) k_active_count(int n, const int *__restrict__ blocks,
                                                              const int *__restrict__ flag,
                                                              const double *__restrict__ iso, int *count) {
  for (int i0 = blockIdx.x * kScanThreads; i0 < n; i0 += gridDim.x * kScanThreads) {
    const int i = i0 + threadIdx.x;
    const bool on = i < n && flag[blocks[i]] != 0;
    const int a = __syncthreads_count(on), k = __syncthreads_count(on && iso[blocks[i]] != 0.0);
    if (threadIdx.x == 0 && a) {
      atomicAdd(&count[0], a);
      atomicAdd(&count[1], k);
    }
  }
}

// head[i]: active entries of list i
__global__ void __launch_bounds__(kScanThreads) k_active_head(int *head, const ActiveList *__restrict__ lists,
                                                             int nlists) {
  for (int i = threadIdx.x; i < nlists; i += blockDim.x) head[i] = lists[i].pre[lists[i].n];
}

// zeros on the solid blocks of up to four vectors
template <typename T>
__global__ void __launch_bounds__(256) k_zero_solid(int nblocks, int ncell, const int *__restrict__ flag, T *a, T *b,
                                                   T *c, T *d) {
  const int lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
  for (int blk = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; blk < nblocks; blk += warps) {
    if (flag[blk]) continue;
    for (int i = lane; i < ncell; i += 32) {
      const long q = (long)blk * ncell + i;
      if (a) a[q] = (T)0;
      if (b) b[q] = (T)0;
      if (c) c[q] = (T)0;
      if (d) d[q] = (T)0;
    }
  }
}

}  // namespace

// device memory that a solve can do without: null where it cannot be had
bool MacGpu::optional_malloc(char **p, size_t bytes) {
  if (!deny_optional_ && dev_malloc(p, bytes) == cudaSuccess) return true;
  cudaGetLastError();
  *p = nullptr;
  return false;
}

// the counts (and the entries of the reduced lists) as the launches before left
// them; one copy and one wait
bool MacGpu::read_active(bool lists) {
  std::vector<int> h(2 + (lists ? n_act_lists_ : 0), 0);
  CKR_(cudaMemcpyAsync(h.data(), d_act_head_, h.size() * sizeof(int), cudaMemcpyDeviceToHost, stream_), false);
  CKR_(cudaStreamSynchronize(stream_), false);
  n_act_ = h[0];
  n_iso_ = h[1];
  if (!lists) return true;
  // active entries of every tower's parity-grouped list
  n_act_par_.assign(towers_.size(), 0);
  for (size_t i = 0, q = 2; i < towers_.size(); i++) {
    if (towers_[i].all.n) q++;
    if (towers_[i].par.n) n_act_par_[i] = h[q++];
  }
  act_lists_version_ = coef_version_;
  return true;
}

// the blocks that hold fluid, by the current volume fractions, and the lists
// reduced to them where they exist
bool MacGpu::count_active() {
  const int nbk = tt_.num_blocks;
  const DevList &top = towers_[finest_].all;
  n_act_ = top.n;
  n_iso_ = 0;
  if (top.n == 0) return true;
  char *mem = nullptr;
  const size_t nhead = 2 + 2 * towers_.size() + levels_.size() + nonleaf_.size();
  if (!d_active_ && !optional_malloc(&mem, (nbk + nhead) * sizeof(int))) return false;
  if (mem) d_active_ = reinterpret_cast<int *>(mem);
  d_act_head_ = d_active_ + nbk;
  CKR_(cudaMemsetAsync(d_act_head_, 0, 2 * sizeof(int), stream_), false);
  k_block_active<<<std::min((nbk + 7) / 8, 152 * 8), 256, 0, stream_>>>(nbk, ncell_, d_vf_, d_active_);
  k_active_count<<<std::min((top.n + kScanThreads - 1) / kScanThreads, 152), kScanThreads, 0, stream_>>>(
      top.n, top.blocks, d_active_, d_iso_, d_act_head_);
  CKR_(cudaGetLastError(), false);
  if (d_act_lists_) reduce_lists();
  return read_active(d_act_lists_ != nullptr);
}

// the reduced lists of these blocks
void MacGpu::reduce_lists() {
  k_active_scan<<<n_act_lists_, kScanThreads, 0, stream_>>>(d_act_lists_, d_active_);
  k_active_copy<<<dim3(152, n_act_lists_), 256, 0, stream_>>>(d_act_lists_);
  k_active_head<<<1, kScanThreads, 0, stream_>>>(d_act_head_ + 2, d_act_lists_, n_act_lists_);
  CK(cudaGetLastError());
}

// the same for the first time; their arrays lie in one allocation
bool MacGpu::build_active() {
  std::vector<ActiveList> h;
  size_t used = 0;
  char *base = nullptr;
  auto take = [&](auto *&p, size_t n) {
    p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(base ? base + used : nullptr);
    used += (n * sizeof(*p) + 15) / 16 * 16;
  };
  ActiveList *lists = nullptr;
  auto lay = [&] {  // sizes first, then places
    used = 0;
    h.clear();
    auto reduce = [&](DevList &d, int nlinks) {
      if (d.n == 0) return;
      take(d.act.blocks, d.n);
      take(d.act.pre, d.n + 1);
      take(d.act.orig, d.n);
      if (d.ftypes) take(d.act.ftypes, d.n);
      if (d.hx) take(d.act.hx, (size_t)d.n * kHX);
      if (d.links) take(d.act.links, (size_t)d.n * nlinks);
      h.push_back(ActiveList{d.blocks, d.ftypes, d.hx, d.links, nlinks, d.n, d.act.blocks, d.act.ftypes, d.act.hx,
                             d.act.links, d.act.pre, d.act.orig});
    };
    for (DevTower &t : towers_) {
      reduce(t.all, 0);
      reduce(t.par, 0);
    }
    for (DevList &l : levels_) reduce(l, 1);
    for (DevList &l : nonleaf_) reduce(l, 8);
    take(lists, h.size());
  };
  lay();
  if (!optional_malloc(&base, used)) return false;
  d_active_mem_ = base;
  lay();
  n_act_lists_ = (int)h.size();
  CKR_(cudaMemcpyAsync(lists, h.data(), h.size() * sizeof(ActiveList), cudaMemcpyHostToDevice, stream_), false);
  CKR_(cudaStreamSynchronize(stream_), false);
  d_act_lists_ = lists;
  reduce_lists();
  return read_active(true);
}

// whether the next solve walks the reduced lists: one shared BiCGSTAB state,
// no learned correction (its kernels walk the full ones), enough solid blocks
void MacGpu::choose_active() {
  act_on_ = false;
  if (multi() || learned_active()) return;
  if (act_version_ != coef_version_) {
    if (!count_active()) return;
    act_version_ = coef_version_;
  }
  const long n = towers_[finest_].all.n;
  if (n_act_ == 0 || (n - n_act_) * kActiveShare < n) return;
  if (act_lists_version_ != coef_version_ && !build_active()) return;
  act_on_ = true;
}

// the solid blocks of the vectors whose neighbours read them are 0 before a
// solve that does not write them
void MacGpu::zero_solid() {
  const int nbk = tt_.num_blocks, g = std::min((nbk + 7) / 8, 152 * 8);
  if (prm_.precision == 1) {
    k_zero_solid<float><<<g, 256, 0, stream_>>>(nbk, ncell_, d_active_, d_resid32_, d_corr32_, d_corr32b_, nullptr);
    k_zero_solid<double><<<g, 256, 0, stream_>>>(nbk, ncell_, d_active_, vec_[kPHAT], vec_[kSHAT], nullptr, nullptr);
  } else {
    k_zero_solid<double><<<g, 256, 0, stream_>>>(nbk, ncell_, d_active_, vec_[kRESID], vec_[kCORR], d_corr64b_,
                                                 nullptr);
  }
  CK_(cudaGetLastError());
}

// list r = entries [a, b) of d, reduced to the active blocks while a solve
// that walks the reduced lists is recorded
BlockList MacGpu::active(BlockList r, const DevList &d, int a, int b) const {
  if (!(solve_lists_ && reduced()) || d.n == 0) return r;
  r.blocks = d.act.blocks;
  r.ftypes = d.act.ftypes;
  r.hx = d.act.hx;
  r.links = d.act.links;
  r.orig = d.act.orig;
  r.pa = d.act.pre + a;
  r.pb = d.act.pre + b;
  return r;
}

}  // namespace sayaka_gb300
