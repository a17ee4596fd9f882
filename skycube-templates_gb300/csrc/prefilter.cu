// Pruner prefilter ahead of the full-space skyline: the suite's priority-queue
// filter (PQFilter::ExecuteExtended, src/utilities/pq_filter.h:140-231,
// applied by MDMC<D>::Init when n > 2 * pq_size, src/mdmc/MDMC.cu:251-252).
// The pq_size points of smallest norm become pruners and every point that a
// pruner strictly dominates is dropped.
//
// Why it is exact: if r is dropped (a pruner t is < r on every attribute)
// and r dominates a point s (<= everywhere), then t is < s everywhere and s
// is dropped as well. So every point that dominates or strictly dominates a
// survivor is a survivor, and the skyline / extended-skyline status of each
// survivor over the survivors equals its status over all points; dropped
// points are strictly dominated, status 2. A point that no other can strictly
// dominate (it holds an attribute's minimum) and that a pruner dominates has
// status 1; what it dominates, strictly or not, a skyline point below it
// dominates as well, so it is not needed as a dominator either and leaves
// the list too.
//
// GB300 form. The norm is the cell sum over S (rank space, so attributes of
// different scales weigh alike; the suite sums raw values). The K smallest
// are picked without a sort: a 2048-bin histogram of cell sums (for the full
// space the cells kernel makes it), a collection pass that finds the
// threshold bin first, and a one-block rank by (sum, id) so the strongest
// pruners are tried first.
// The filter looks a point's cells up in bit tables of the ranked pruners
// (k_prefilter); floats are read only where cells tie.
#include <algorithm>

#include "kernels.cuh"

namespace skc {

__device__ __forceinline__ uint32_t cell_sum(const uint4& c, uint32_t S, int d) {
  uint32_t s = 0;
  for (int k = 0; k < d; ++k)
    if ((S >> k) & 1u) s += (word_of(c, k >> 2) >> (8 * (k & 3))) & 0x7fu;
  return s;
}

__global__ void __launch_bounds__(256) k_pruner_hist(const uint4* __restrict__ cells,
                                                     const uint32_t* __restrict__ ids,
                                                     const uint32_t* __restrict__ m_ptr,
                                                     uint32_t S, int d,
                                                     uint32_t* __restrict__ hist) {
  __shared__ uint32_t h[kSumBins];
  for (uint32_t b = threadIdx.x; b < kSumBins; b += blockDim.x) h[b] = 0;
  __syncthreads();
  const uint32_t m = *m_ptr;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    const uint32_t id = ids ? ids[i] : i;
    atomicAdd(&h[cell_sum(cells[id], S, d)], 1u);
  }
  __syncthreads();
  for (uint32_t b = threadIdx.x; b < kSumBins; b += blockDim.x)
    if (h[b]) atomicAdd(&hist[b], h[b]);
}

// Collects the K points of smallest cell sum. The threshold bin (the first
// whose inclusive count reaches Kp = min(K, m)) comes from the histogram, and
// every CTA finds it for itself (a launch less than a select kernel). sel[2]
// = Kp; sel[3] and sel[4] are the collection cursors, zero before the launch.
__global__ void __launch_bounds__(256) k_pruner_collect(const uint4* __restrict__ cells,
                                                        const uint32_t* __restrict__ ids,
                                                        const uint32_t* __restrict__ m_ptr,
                                                        uint32_t S, int d, uint32_t K,
                                                        const uint32_t* __restrict__ hist,
                                                        uint32_t* __restrict__ sel,
                                                        uint32_t* __restrict__ pr_ids,
                                                        uint32_t* __restrict__ pr_key) {
  __shared__ uint32_t wsum[8];
  __shared__ uint32_t s_thr, s_below;
  const uint32_t m = *m_ptr;
  const uint32_t Kp = min(K, m);
  if (blockIdx.x == 0 && threadIdx.x == 0) sel[2] = Kp;
  if (Kp == 0) return;
  {
    const int t = threadIdx.x, ln = t & 31, wid = t >> 5;
    uint32_t h[8], c = 0;  // this thread's bins 8t .. 8t + 7
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      h[j] = hist[8 * t + j];
      c += h[j];
    }
    uint32_t inc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
      if (ln >= o) inc += u;
    }
    if (ln == 31) wsum[wid] = inc;
    __syncthreads();
    uint32_t e = inc - c;  // points in the bins before this thread's
    for (int j = 0; j < wid; ++j) e += wsum[j];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (e < Kp && e + h[j] >= Kp) {
        s_thr = 8 * t + j;
        s_below = e;
      }
      e += h[j];
    }
    __syncthreads();
  }
  const uint32_t thr = s_thr, below = s_below;
  const int lane = threadIdx.x & 31;
  const uint32_t warp0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t base = warp0; base < m; base += stride) {
    const uint32_t i = base + lane;
    uint32_t id = 0, s = 0xffffffffu;
    if (i < m) {
      id = ids ? ids[i] : i;
      s = cell_sum(cells[id], S, d);
    }
    // Warp-aggregated cursors: one atomic per warp and class.
    const uint32_t lo = __ballot_sync(0xffffffffu, s < thr);
    const uint32_t eq = __ballot_sync(0xffffffffu, s == thr);
    uint32_t lo_base = 0, eq_base = 0;
    if (lane == 0) {
      if (lo) lo_base = atomicAdd(&sel[3], (uint32_t)__popc(lo));
      if (eq) eq_base = atomicAdd(&sel[4], (uint32_t)__popc(eq));
    }
    lo_base = __shfl_sync(0xffffffffu, lo_base, 0);
    eq_base = __shfl_sync(0xffffffffu, eq_base, 0);
    const uint32_t before = (1u << lane) - 1u;
    uint32_t slot = 0xffffffffu;
    if (s < thr) {
      slot = lo_base + __popc(lo & before);
    } else if (s == thr) {
      const uint32_t t = eq_base + __popc(eq & before);
      if (t < Kp - below) slot = below + t;
    }
    if (slot < Kp) {
      pr_ids[slot] = id;
      pr_key[slot] = s;
    }
  }
}

// Ranks the Kp pruners by (sum, id) and stores their cells and floats in rank
// order: out_x[k * K + r] for attribute k. Zeroes the filter's counts.
__global__ void __launch_bounds__(1024) k_pruner_order(const uint32_t* __restrict__ pr_ids,
                                                       const uint32_t* __restrict__ pr_key,
                                                       const uint32_t* __restrict__ sel,
                                                       const uint4* __restrict__ cells,
                                                       const float* __restrict__ x,
                                                       uint64_t n_pad, int d, uint32_t K,
                                                       uint4* __restrict__ out_cells,
                                                       float* __restrict__ out_x,
                                                       uint32_t* __restrict__ blk, uint32_t nblk) {
  static_assert(kMaxPruners <= 1024, "one pruner per thread");
  __shared__ unsigned long long key[kMaxPruners];
  for (uint32_t b = threadIdx.x; b < nblk; b += blockDim.x) blk[b] = 0;
  const uint32_t Kp = sel[2];
  const uint32_t t = threadIdx.x;
  unsigned long long me = ~0ull;
  if (t < Kp) me = ((unsigned long long)pr_key[t] << 32) | pr_ids[t];
  key[t] = me;
  __syncthreads();
  if (t >= Kp) return;
  uint32_t r = 0;
#pragma unroll 8
  for (uint32_t j = 0; j < Kp; ++j) r += key[j] < me;
  const uint32_t id = (uint32_t)me;
  out_cells[r] = cells[id];
  for (int k = 0; k < d; ++k) out_x[(uint64_t)k * K + r] = x[(uint64_t)k * n_pad + id];
}

// Pruner tables. A group is 64 consecutive ranks; T[g][k][v] holds, one bit
// per pruner, those whose cell on attribute k is at most v (all of the group's
// for k outside S). The AND over a point's attributes is the group's pruners
// that may dominate it.
constexpr uint32_t kGroupPruners = 64;

static uint32_t pruner_groups(uint32_t K) { return (K + kGroupPruners - 1) / kGroupPruners; }

__global__ void __launch_bounds__(128) k_pruner_tables(const uint4* __restrict__ pr_cells,
                                                       const uint32_t* __restrict__ sel,
                                                       uint32_t S,
                                                       unsigned long long* __restrict__ tab) {
  const uint32_t g = blockIdx.x, k = blockIdx.y, v = threadIdx.x;
  const uint32_t beg = g * kGroupPruners, end = min(sel[2], beg + kGroupPruners);
  __shared__ uint8_t c[kGroupPruners];
  if (beg + v < end && v < kGroupPruners)
    c[v] = (uint8_t)(word_of(pr_cells[beg + v], k >> 2) >> (8 * (k & 3)));
  __syncthreads();
  unsigned long long b = 0;
  for (uint32_t j = 0; beg + j < end; ++j)
    if (!((S >> k) & 1u) || c[j] <= v) b |= 1ull << j;
  tab[((uint64_t)g * gridDim.y + k) * 128 + v] = b;
}

// Tests the list's points against the pruner groups [g0, g1): status 2 when
// one strictly dominates the point on S; status 1 when the point holds the
// minimum of an attribute of S (amin: nothing can strictly dominate it) and
// one dominates it; else 0. A further launch (`again`) leaves the settled
// ones. With blk, blk[b] = the entries of [1024 b, 1024 b + 1024) left at 0
// (the count pass of their compaction; zero before).
//
// The tables give the pruners whose cells are all at most the point's with D
// 8-byte loads from shared memory per 64 pruners; only those few are compared
// in the exact floats where cells tie. A walk over the pruners one by one (a
// warp as many as its last open lane), groups of eight skipped by their
// minimum cells, took 0.40 ms for the 512 pruners of 1M x 10 anticorrelated
// points and 0.29 for 1M x 12 uniform; now 0.12 and 0.12. Settling the
// points with a minimum matters on tied data: nearly every point left holds
// one there (581k x 10 ties: 24,600 of 24,600), and the skyline kernel would
// search each one's dominator. A point with every minimum is equal to the
// pruners it passes: it is left at once (500k x 8 correlated: a walk over all pruners,
// 0.090 -> 0.046 ms for the step).
//
// One pass over the list with all pruners. Two, the second over what a 16th
// of the pruners left and only when that was a quarter, take a compaction
// and two launches more, and the skyline kernel then got 20,200 points of
// 250k x 5 uniform where 2,600 are left now: prefilter and skyline kernel
// 0.130 -> 0.096 ms there, 100k x 6 0.118 -> 0.091, 1M x 10 1.25 -> 1.23.
template <int D>
__global__ void __launch_bounds__(1024) k_prefilter(
    const uint4* __restrict__ cells, const float* __restrict__ x, uint64_t n_pad,
    const uint32_t* __restrict__ ids, const uint32_t* __restrict__ m_ptr, uint32_t S,
    const uint4* __restrict__ pr_cells, const float* __restrict__ pr_x, uint32_t K,
    const unsigned long long* __restrict__ tab, uint32_t g0, uint32_t g1,
    const uint32_t* __restrict__ amin, int again,
    uint8_t* __restrict__ status, uint32_t* __restrict__ blk) {
  constexpr int NW = (D + 3) / 4;
  extern __shared__ uint4 s_tab4[];  // [groups][D][128] eight-byte masks
  const unsigned long long* s_tab = reinterpret_cast<const unsigned long long*>(s_tab4);
  const uint32_t m = *m_ptr;
  const uint32_t groups = g1 - g0;
  if ((uint64_t)blockIdx.x * 1024 >= m) return;
  const uint4* src = reinterpret_cast<const uint4*>(tab + (uint64_t)g0 * (D * 128));
  for (uint32_t t = threadIdx.x; t < groups * (D * 64); t += 1024) s_tab4[t] = src[t];
  __syncthreads();
  uint32_t hS[NW];
#pragma unroll
  for (int w = 0; w < NW; ++w) hS[w] = guard_mask(S, w);
  const int na = __popc(S);
  for (uint64_t base = (uint64_t)blockIdx.x * 1024; base < m; base += (uint64_t)gridDim.x * 1024) {
    const uint32_t i = (uint32_t)base + threadIdx.x;
    bool keep = false;
    if (i < m) {
      if (again && status[i]) {
        keep = false;
      } else {
        const uint32_t id = ids ? ids[i] : i;
        const uint4 c4 = cells[id];
        uint32_t found = 0;  // the status a pruner gives
        int n_min = -1;  // attributes of S on which the point holds the minimum (-1: not counted)
        for (uint32_t g = 0; g < groups && !found && n_min != na; ++g) {
          const unsigned long long* T = s_tab + g * (D * 128);
          unsigned long long b = ~0ull;
#pragma unroll
          for (int k = 0; k < D; ++k)
            b &= T[128 * k + ((word_of(c4, k >> 2) >> (8 * (k & 3))) & 0x7fu)];
          for (; b && !found; b &= b - 1) {
            const uint32_t t = (g0 + g) * kGroupPruners + __ffsll(b) - 1;
            const uint4 q = pr_cells[t];
            uint32_t Z = 0;  // attributes of S with equal cells
#pragma unroll
            for (int w = 0; w < NW; ++w)
              Z |= pack_guards(ge_bytes(word_of(q, w) | kGuard, word_of(c4, w)) & hS[w]) << (4 * w);
            if (n_min < 0) {  // a minimum's cell is 0, and so is the pruner's there
              uint32_t zero = 0;
#pragma unroll
              for (int w = 0; w < NW; ++w)
                zero |= pack_guards((kGuard - word_of(c4, w)) & hS[w]) << (4 * w);
              n_min = 0;
              for (; zero; zero &= zero - 1) {
                const int k = __ffs(zero) - 1;
                n_min += ordered_u32(x[(uint64_t)k * n_pad + id]) == amin[k];
              }
              if (n_min == na) break;  // nothing dominates it
            }
            const bool at_min = n_min > 0;
            bool le = true, all_lt = true, any_lt = Z != S;
            for (; Z && le && (all_lt || at_min); Z &= Z - 1) {
              const int k = __ffs(Z) - 1;
              const float a = pr_x[(uint64_t)k * K + t], p = x[(uint64_t)k * n_pad + id];
              le = a <= p;
              if (a < p) any_lt = true; else all_lt = false;
            }
            if (at_min) found = (le && any_lt) ? 1u : 0u;
            else found = (le && all_lt) ? 2u : 0u;
          }
        }
        keep = !found;
        status[i] = (uint8_t)found;
      }
    }
    const int kept = __syncthreads_count(keep);
    if (blk && threadIdx.x == 0) blk[base >> 10] = kept;
  }
}

size_t prefilter_table_bytes(int d, uint32_t K) {
  return (size_t)pruner_groups(K) * d * 128 * sizeof(unsigned long long);
}

// Groups of one launch: their tables have to fit the shared memory.
constexpr size_t kMaxTableSmem = 200 * 1024;

template <int D>
static int launch_prefilter_d(cudaStream_t s, int num_sms, const PrefilterArgs& a) {
  constexpr size_t kGroupBytes = D * 128 * sizeof(unsigned long long);
  constexpr uint32_t kMost = (uint32_t)(kMaxTableSmem / kGroupBytes);
  const uint32_t G = pruner_groups(a.K);
  SKC_CUDA(cudaFuncSetAttribute(k_prefilter<D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(kMost * kGroupBytes)));
  const uint64_t want = (a.m_max + 1023) / 1024;
  for (uint32_t g = 0; g < G; g += kMost) {
    const uint32_t e = std::min(G, g + kMost);
    const size_t smem = (e - g) * kGroupBytes;
    const uint64_t per_sm = smem > 110 * 1024 ? 1 : 2;
    const unsigned grid =
        (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(want, (uint64_t)num_sms * per_sm));
    k_prefilter<D><<<grid, 1024, smem, s>>>(a.cells, a.x, a.n_pad, a.ids, a.m_ptr, a.S,
                                            a.ps.pr_cells, a.ps.pr_x, a.K, a.ps.tab, g, e, a.amin,
                                            g > 0, a.status, e == G ? a.ps.blk : nullptr);
    SKC_LAUNCH_CHECK();
  }
  return SKC_OK;
}

int launch_prefilter(cudaStream_t s, int d, int num_sms, const PrefilterArgs& a,
                     uint32_t* out, uint32_t* out_count) {
  if (a.K < 1 || a.K > (uint32_t)kMaxPruners)
    return set_error(SKC_ERR_INVALID, "pruner count %u outside [1, %d]", a.K, kMaxPruners);
  const PrefilterScratch& p = a.ps;
  const uint64_t want = (a.m_max + 255) / 256;
  const unsigned grid =
      (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(want, (uint64_t)num_sms * 8));
  if (!a.hist_ready) {
    SKC_CUDA(cudaMemsetAsync(p.hist, 0, (kSumBins + 8) * sizeof(uint32_t), s));
    k_pruner_hist<<<grid, 256, 0, s>>>(a.cells, a.ids, a.m_ptr, a.S, d, p.hist);
    SKC_LAUNCH_CHECK();
  }
  uint32_t* sel = p.hist + kSumBins;
  k_pruner_collect<<<grid, 256, 0, s>>>(a.cells, a.ids, a.m_ptr, a.S, d, a.K, p.hist, sel,
                                        p.pr_ids, p.pr_key);
  SKC_LAUNCH_CHECK();
  k_pruner_order<<<1, 1024, 0, s>>>(p.pr_ids, p.pr_key, sel, a.cells, a.x, a.n_pad, d, a.K,
                                    p.pr_cells, p.pr_x, p.blk,
                                    (uint32_t)((a.m_max + 1023) / 1024));
  SKC_LAUNCH_CHECK();
  k_pruner_tables<<<dim3(pruner_groups(a.K), d), 128, 0, s>>>(p.pr_cells, sel, a.S, p.tab);
  SKC_LAUNCH_CHECK();
  switch (d) {
#define SKC_PF_CASE(D) \
  case D: SKC_TRY(launch_prefilter_d<D>(s, num_sms, a)); break;
    SKC_PF_CASE(2) SKC_PF_CASE(3) SKC_PF_CASE(4) SKC_PF_CASE(5) SKC_PF_CASE(6)
    SKC_PF_CASE(7) SKC_PF_CASE(8) SKC_PF_CASE(9) SKC_PF_CASE(10) SKC_PF_CASE(11)
    SKC_PF_CASE(12) SKC_PF_CASE(13) SKC_PF_CASE(14) SKC_PF_CASE(15) SKC_PF_CASE(16)
#undef SKC_PF_CASE
    default:
      return set_error(SKC_ERR_INVALID, "unsupported d=%d", d);
  }
  return launch_status_keep(s, a.status, a.m_ptr, a.m_max, p.blk, out, out_count);
}

}  // namespace skc
