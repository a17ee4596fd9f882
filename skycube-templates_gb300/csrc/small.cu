// Skyline of a short list (at most kSmallList points) on one subspace, in one
// launch: statuses by comparing every pair's floats, then the compaction into
// id lists by the last CTA to finish.
//
// The median-partition pipeline (partition.cu) takes eight launches and a
// grid of cells before it compares anything, 60 to 90 us on one GB300 however
// short the list. Up to a few thousand points all pairs are less work than
// that: the full space of 1,000 x 4 uniform 20 us against 71, 5,003 x 8
// correlated 45 against 95, 4,000 x 16 anticorrelated 47 against 110. At
// 8,192 points it is even (ties x 10 110 against 105, anticorrelated x 16 143
// against 150), so the limit lies below. Bound by the shared-memory broadcasts
// and compares of the pairs. The suite has no counterpart (SkyAlign runs on
// every list, src/sdsc/skyAlign.cu:9-53).
#include "kernels.cuh"

namespace skc {

constexpr uint32_t kAllLanes = 0xffffffffu;
constexpr int kSmallThreads = 1024;
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr uint32_t kSmallUnroll = 4;  // q's tested side by side: a warp's chain of compares is its latency
static_assert(kSmallList % 32 == 0 && kSmallList / 32 <= kSmallThreads,
              "the last CTA scans one 32-point mask per thread");

struct SmallArgs {
  const float* x;            // attribute-major points
  uint64_t n_pad;
  unsigned long long attrs;  // attribute t of S in bits 4t .. 4t + 3
  const uint32_t* sub;       // the list positions to compare (nullptr: all)
  const uint32_t* ids;       // list position -> point id (nullptr: identity)
  const uint32_t* m_ptr;     // list length, at most kSmallList (nullptr: m)
  uint32_t m;
  uint32_t nblk;             // CTAs of this list
  uint32_t* masks;           // [2 * kSmallList / 32] skyline, extended skyline bits
  uint32_t* ticket;          // CTAs done, 0 before the launch
  SplitOut out;
};

// The largest float below v (finite): q < v exactly when q <= float_below(v).
__device__ __forceinline__ float float_below(float v) {
  const uint32_t u = __float_as_uint(v);
  return __uint_as_float(v > 0.f ? u - 1u : v < 0.f ? u + 1u : 0x80000001u);
}

// A CTA owns 32 list entries (a lane each, in every warp); its warps share the
// q's, staged a tile at a time, and read them by broadcast. Once a point is dominated
// only strict domination matters, so its values become their predecessors and
// the same <= test decides it (tied points else pass it again and again).
// Thread 0 .. 31 (a lane per entry) return the entry's flags: 1 dominated, 2
// strictly so (2 also past the end).
template <int NA>
__device__ __forceinline__ uint32_t small_pairs(const SmallArgs& a, uint32_t m, uint32_t blk) {
  constexpr int NV = (NA + 3) / 4;
  constexpr uint32_t TQ = NV <= 2 ? 1024 : 512;  // q's per tile (at most 32 KB)
  __shared__ float4 s_q[TQ * NV];  // [q][its NA values]
  __shared__ uint32_t s_dom, s_strict;
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t i = blk * 32 + lane;
  float pv[NA];
  uint32_t id = 0;
  if (i < m) {
    id = a.sub ? a.sub[i] : i;
    if (a.ids) id = a.ids[id];
  }
#pragma unroll
  for (int t = 0; t < NA; ++t)
    pv[t] = i < m ? a.x[((a.attrs >> (4 * t)) & 15u) * a.n_pad + id] : 0.f;
  const uint32_t none = __ballot_sync(kAllLanes, i >= m);
  if (threadIdx.x == 0) {
    s_dom = 0;
    s_strict = none;  // lanes without a point count as settled
  }
  bool dom = false, strict = i >= m;
  for (uint32_t base = 0; base < m; base += TQ) {
    const uint32_t j = base + threadIdx.x;
    if (threadIdx.x < TQ && j < m) {
      uint32_t qid = a.sub ? a.sub[j] : j;
      if (a.ids) qid = a.ids[qid];
      float v[4 * NV];
#pragma unroll
      for (int t = 0; t < 4 * NV; ++t)
        v[t] = t < NA ? a.x[((a.attrs >> (4 * t)) & 15u) * a.n_pad + qid] : 0.f;
#pragma unroll
      for (int t = 0; t < NV; ++t)
        s_q[threadIdx.x * NV + t] = make_float4(v[4 * t], v[4 * t + 1], v[4 * t + 2], v[4 * t + 3]);
    }
    __syncthreads();
    constexpr uint32_t QW = TQ / kSmallWarps;  // q's of a warp
    const uint32_t end = min(QW, m - min(m, base + wid * QW));
    for (uint32_t t0 = 0; t0 < end; t0 += kSmallUnroll) {
      bool le[kSmallUnroll];
      bool some = false;
#pragma unroll
      for (uint32_t u = 0; u < kSmallUnroll; ++u) {
        // past the end the last q again: a q tested twice changes nothing
        const float4* q = s_q + (wid * QW + min(t0 + u, end - 1)) * NV;
        le[u] = !strict;
#pragma unroll
        for (int g = 0; g < NV; ++g) {
          const float4 v = q[g];
          le[u] &= v.x <= pv[4 * g];
          if (4 * g + 1 < NA) le[u] &= v.y <= pv[4 * g + 1 < NA ? 4 * g + 1 : 0];
          if (4 * g + 2 < NA) le[u] &= v.z <= pv[4 * g + 2 < NA ? 4 * g + 2 : 0];
          if (4 * g + 3 < NA) le[u] &= v.w <= pv[4 * g + 3 < NA ? 4 * g + 3 : 0];
        }
        some |= le[u];
      }
      if (!__any_sync(kAllLanes, some)) continue;
      for (uint32_t u = 0; u < kSmallUnroll; ++u) {
        const float* qf = reinterpret_cast<const float*>(
            s_q + (wid * QW + min(t0 + u, end - 1)) * NV);
        // pv may have changed since the test above: compare again
        bool lt_all = !strict, le_all = !strict, any = false;
#pragma unroll
        for (int k = 0; k < NA; ++k) {
          const bool lt = qf[k] < pv[k];
          le_all &= qf[k] <= pv[k];
          lt_all &= lt;
          any |= lt;
        }
        if (!le_all) continue;
        if (dom || lt_all) {  // with dom, pv holds the predecessors
          dom = true;
          strict = true;
        } else if (any) {
          dom = true;
#pragma unroll
          for (int k = 0; k < NA; ++k) pv[k] = float_below(pv[k]);
        }
      }
      if (__all_sync(kAllLanes, strict)) break;
    }
    const uint32_t sm = __ballot_sync(kAllLanes, strict);
    if (lane == 0) atomicOr(&s_strict, sm);
    __syncthreads();
    const uint32_t settled = s_strict;
    strict = strict || ((settled >> lane) & 1u);
    if (settled == kAllLanes) break;  // the same for every warp
  }
  const uint32_t dm = __ballot_sync(kAllLanes, dom);
  if (lane == 0) atomicOr(&s_dom, dm);
  __syncthreads();
  return ((s_dom >> lane) & 1u) | ((s_strict >> lane) & 1u) << 1;
}

template <int NA>
__device__ __forceinline__ void small_skyline(const SmallArgs& a, uint32_t blk) {
  __shared__ uint32_t s_last;
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t m = a.m_ptr ? *a.m_ptr : a.m;
  if (blk * 32 < m) {
    const uint32_t f = small_pairs<NA>(a, m, blk);
    if (wid == 0) {
      const uint32_t sky = __ballot_sync(kAllLanes, f == 0), ext = __ballot_sync(kAllLanes, f == 1);
      if (lane == 0) {
        a.masks[blk] = sky;
        a.masks[kSmallList / 32 + blk] = ext;
      }
    }
  }
  // The last CTA compacts; the masks are read past L1.
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(a.ticket, 1u) == a.nblk - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  __shared__ uint32_t s_m0[kSmallList / 32], s_m1[kSmallList / 32];
  __shared__ uint32_t s_o0[kSmallList / 32], s_o1[kSmallList / 32];
  __shared__ uint32_t s_w0[kSmallWarps], s_w1[kSmallWarps], s_n0;
  const uint32_t nw = (m + 31) / 32;
  const uint32_t t = threadIdx.x;
  uint32_t m0 = 0, m1 = 0;
  if (t < nw) {
    m0 = __ldcg(a.masks + t);
    m1 = __ldcg(a.masks + kSmallList / 32 + t);
  }
  uint32_t i0 = __popc(m0), i1 = __popc(m1);
  const uint32_t c0 = i0, c1 = i1;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(kAllLanes, i0, o), v = __shfl_up_sync(kAllLanes, i1, o);
    if (lane >= (uint32_t)o) {
      i0 += u;
      i1 += v;
    }
  }
  if (lane == 31) {
    s_w0[wid] = i0;
    s_w1[wid] = i1;
  }
  __syncthreads();
  for (uint32_t w = 0; w < wid; ++w) {
    i0 += s_w0[w];
    i1 += s_w1[w];
  }
  if (t < kSmallList / 32) {
    s_m0[t] = m0;
    s_m1[t] = m1;
    s_o0[t] = i0 - c0;
    s_o1[t] = i1 - c1;
  }
  if (t == kSmallThreads - 1) {
    *a.ticket = 0;  // for the next launch
    s_n0 = i0;
    a.out.n[0] = i0;
    a.out.n[1] = i1;
    a.out.n[2] = i0 + i1;
  }
  __syncthreads();
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t* ext_out = a.out.ext ? a.out.ext : a.out.sky + s_n0;
#pragma unroll 4
  for (uint32_t w = wid; w < nw; w += kSmallWarps) {
    const uint32_t b0 = s_m0[w], b1 = s_m1[w];
    const bool sky = (b0 >> lane) & 1u, ext = (b1 >> lane) & 1u;
    if (!sky && !ext) continue;
    const uint32_t at = w * 32 + lane;
    const uint32_t pid = a.ids ? a.ids[at] : at;
    const uint32_t k0 = s_o0[w] + __popc(b0 & lt), k1 = s_o1[w] + __popc(b1 & lt);
    if (sky) a.out.sky[k0] = pid;
    else ext_out[k1] = pid;
    if (a.out.both) {
      a.out.both[k0 + k1] = pid;
      if (a.out.both_st) {
        a.out.both_st[k0 + k1] = sky ? 0 : 2;
        if (sky) a.out.pos0[k0] = k0 + k1;
      }
    }
  }
}

template <int NA>
__global__ void __launch_bounds__(kSmallThreads) k_small_skyline(SmallArgs a) {
  small_skyline<NA>(a, blockIdx.x);
}

// The lists of up to kSmallJobs subspaces of NA attributes each (cuboids of
// one lattice level), their CTAs side by side: a list alone fills a few SMs.
// One after the other, with the host's reads, the 62 cuboids of 100k x 6
// uniform (2,239 candidates) took 1.76 ms, a launch per level 0.20.
struct SmallBatch {
  const float* x;
  uint64_t n_pad;
  uint32_t* masks;   // [kSmallJobs][2 * kSmallList / 32]
  uint32_t* ticket;  // [kSmallJobs]
  uint32_t nj;
  SmallJob job[kSmallJobs];
};
static_assert(sizeof(SmallBatch) <= 4096, "kernel parameters");

template <int NA>
__global__ void __launch_bounds__(kSmallThreads)
    k_small_batch(const __grid_constant__ SmallBatch b) {
  uint32_t lo = 0, hi = b.nj - 1;  // the last job that begins at or before this CTA
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1) >> 1;
    if (b.job[mid].first <= blockIdx.x) lo = mid; else hi = mid - 1;
  }
  const SmallJob& J = b.job[lo];
  const SmallArgs a{b.x, b.n_pad, J.attrs, nullptr, J.ids, nullptr, J.m, (J.m + 31) / 32,
                    b.masks + lo * (2 * kSmallList / 32), b.ticket + lo,
                    {J.lists, nullptr, J.both, nullptr, nullptr, J.n}};
  small_skyline<NA>(a, blockIdx.x - J.first);
}

template <int NA>
static int launch_small_na(cudaStream_t s, unsigned grid, const SmallArgs& a) {
  k_small_skyline<NA><<<grid, kSmallThreads, 0, s>>>(a);
  SKC_LAUNCH_CHECK();
  return SKC_OK;
}

// Attributes of S, four bits each; returns their number.
static int small_attrs(uint32_t S, int d, unsigned long long* attrs) {
  int na = 0;
  *attrs = 0;
  for (int k = 0; k < d; ++k)
    if (S & (1u << k)) *attrs |= (unsigned long long)k << (4 * na++);
  return na;
}

int launch_small_skyline(cudaStream_t s, const float* x, uint64_t n_pad, int d,
                         const uint32_t* ids, const uint32_t* m_ptr, uint64_t m_max, uint32_t S,
                         uint32_t* masks, uint32_t* ticket, const SplitOut& out) {
  if (m_max > kSmallList)
    return set_error(SKC_ERR_INVALID, "list of %llu points for the short-list skyline",
                     (unsigned long long)m_max);
  unsigned long long attrs;
  const int na = small_attrs(S, d, &attrs);
  const unsigned grid = (unsigned)(m_max ? (m_max + 31) / 32 : 1);
  const SmallArgs a{x, n_pad, attrs, nullptr, ids, m_ptr, 0, grid, masks, ticket, out};
  switch (na) {
#define SKC_SMALL_CASE(N) \
  case N: return launch_small_na<N>(s, grid, a);
    SKC_SMALL_CASE(1) SKC_SMALL_CASE(2) SKC_SMALL_CASE(3) SKC_SMALL_CASE(4)
    SKC_SMALL_CASE(5) SKC_SMALL_CASE(6) SKC_SMALL_CASE(7) SKC_SMALL_CASE(8)
    SKC_SMALL_CASE(9) SKC_SMALL_CASE(10) SKC_SMALL_CASE(11) SKC_SMALL_CASE(12)
    SKC_SMALL_CASE(13) SKC_SMALL_CASE(14) SKC_SMALL_CASE(15) SKC_SMALL_CASE(16)
#undef SKC_SMALL_CASE
    default:
      return set_error(SKC_ERR_INVALID, "subspace with %d attributes", na);
  }
}

template <int NA>
static int launch_batch_na(cudaStream_t s, unsigned grid, const SmallBatch& b) {
  k_small_batch<NA><<<grid, kSmallThreads, 0, s>>>(b);
  SKC_LAUNCH_CHECK();
  return SKC_OK;
}

int launch_small_batch(cudaStream_t s, const float* x, uint64_t n_pad, int d, SmallJob* jobs,
                       uint32_t nj, uint32_t* masks, uint32_t* tickets) {
  if (nj == 0) return SKC_OK;
  SmallBatch b;
  b.x = x;
  b.n_pad = n_pad;
  b.masks = masks;
  b.ticket = tickets;
  b.nj = nj;
  const int na = __builtin_popcount(jobs[0].S);
  uint32_t grid = 0;
  for (uint32_t j = 0; j < nj; ++j) {
    SmallJob& J = jobs[j];
    if (nj > kSmallJobs || J.m == 0 || J.m > kSmallList || __builtin_popcount(J.S) != na)
      return set_error(SKC_ERR_INVALID, "short-list batch: job %u of %u, %u points", j, nj, J.m);
    small_attrs(J.S, d, &J.attrs);
    J.first = grid;
    grid += (J.m + 31) / 32;
    b.job[j] = J;
  }
  switch (na) {
#define SKC_BATCH_CASE(N) \
  case N: return launch_batch_na<N>(s, grid, b);
    SKC_BATCH_CASE(1) SKC_BATCH_CASE(2) SKC_BATCH_CASE(3) SKC_BATCH_CASE(4)
    SKC_BATCH_CASE(5) SKC_BATCH_CASE(6) SKC_BATCH_CASE(7) SKC_BATCH_CASE(8)
    SKC_BATCH_CASE(9) SKC_BATCH_CASE(10) SKC_BATCH_CASE(11) SKC_BATCH_CASE(12)
    SKC_BATCH_CASE(13) SKC_BATCH_CASE(14) SKC_BATCH_CASE(15)
#undef SKC_BATCH_CASE
    default:
      return set_error(SKC_ERR_INVALID, "short-list batch over %d attributes", na);
  }
}

// Statuses of the points a prefilter leaves open, when they are few: their
// number is known on the device only, so this kernel is launched before the
// partition pipeline and leaves that no points (`rest` 0) when it takes the
// list itself. The step on one GB300, pipeline alone / with this kernel: 2,600
// points left of 250k x 5 uniform 100 / 53 us, 1,000 of 204k x 4 78 / 43; 6,000
// points of 4 attributes 187 / 74, of 8 121 / 101, of 16 109 / 152, 5,000 of
// 16 113 / 136: hence the limits, by attributes. With longer lists it adds 2 us.
template <int NA>
constexpr uint32_t kSmallOpen = NA <= 8 ? kSmallList : 4096;

template <int NA>
__global__ void __launch_bounds__(kSmallThreads)
    k_small_status(SmallArgs a, uint8_t* __restrict__ status, uint32_t* __restrict__ rest) {
  const uint32_t m = *a.m_ptr;
  const bool few = m <= kSmallOpen<NA>;
  if (blockIdx.x == 0 && threadIdx.x == 0) *rest = few ? 0 : m;
  if (!few || blockIdx.x * 32 >= m) return;
  const uint32_t f = small_pairs<NA>(a, m, blockIdx.x);
  const uint32_t i = blockIdx.x * 32 + threadIdx.x;
  if (threadIdx.x < 32 && i < m && f) status[a.sub ? a.sub[i] : i] |= (uint8_t)f;
}

template <int NA>
static int launch_status_na(cudaStream_t s, const SmallArgs& a, uint8_t* status, uint32_t* rest) {
  k_small_status<NA><<<kSmallOpen<NA> / 32, kSmallThreads, 0, s>>>(a, status, rest);
  SKC_LAUNCH_CHECK();
  return SKC_OK;
}

int launch_small_status(cudaStream_t s, int d, const PartitionSkylineArgs& a, uint32_t* rest) {
  unsigned long long attrs;
  const int na = small_attrs(a.S, d, &attrs);
  const SmallArgs k{a.x, a.n_pad, attrs, a.sub, a.ids, a.m_ptr, 0, 0, nullptr, nullptr, {}};
  switch (na) {
#define SKC_STATUS_CASE(N) \
  case N: return launch_status_na<N>(s, k, a.status, rest);
    SKC_STATUS_CASE(1) SKC_STATUS_CASE(2) SKC_STATUS_CASE(3) SKC_STATUS_CASE(4)
    SKC_STATUS_CASE(5) SKC_STATUS_CASE(6) SKC_STATUS_CASE(7) SKC_STATUS_CASE(8)
    SKC_STATUS_CASE(9) SKC_STATUS_CASE(10) SKC_STATUS_CASE(11) SKC_STATUS_CASE(12)
    SKC_STATUS_CASE(13) SKC_STATUS_CASE(14) SKC_STATUS_CASE(15) SKC_STATUS_CASE(16)
#undef SKC_STATUS_CASE
    default:
      return set_error(SKC_ERR_INVALID, "subspace with %d attributes", na);
  }
}

// The bitmap kernel's inputs for at most kSmallCandidates candidates, one per
// thread of one CTA: cells, floats in candidate order, and the skyline points
// as q's in candidate order with their box minima, one partition. The cells
// come from an even grid between the attribute's least and greatest value
// (any monotone cells are exact). Quantile pivots, the sort by partition and
// the box pass are seven launches, some 35 us on one GB300, where the q's fill
// 32 blocks at most; this one takes 7. Quantiles are better where an attribute
// has a far outlier, which leaves the others in one cell and every pair to the
// floats. Whole call through the seven launches / through this one, ms, and
// the same with one such outlier per attribute: 5,003 x 8 correlated 0.154 /
// 0.131, 0.152 / 0.137; 800 x 10 uniform 0.160 / 0.124, 0.161 / 0.162; 1,000 x
// 10 anticorrelated 0.162 / 0.138, 0.162 / 0.189; 1,000 x 16 cap 4 0.366 /
// 0.340, 0.361 / 0.434.
template <int D>
__global__ void __launch_bounds__(kSmallCandidates) k_small_prep(
    const float* __restrict__ x, uint64_t n_pad, const uint32_t* __restrict__ cand,
    const uint8_t* __restrict__ cand_st, const uint32_t* __restrict__ m_ptr, int depth,
    uint64_t pitch, uint4* __restrict__ cells, float* __restrict__ px, uint4* __restrict__ qcells,
    float* __restrict__ qx, uint4* __restrict__ bmin, uint4* __restrict__ smin,
    uint4* __restrict__ hmin, uint32_t* __restrict__ boff, uint32_t* __restrict__ work) {
  __shared__ uint32_t s_lo[D], s_hi[D], s_w[32];
  const uint32_t t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const uint32_t m = *m_ptr;
  if (t < D) {
    s_lo[t] = 0xffffffffu;
    s_hi[t] = 0;
  }
  __syncthreads();
  float v[D];
  const bool in = t < m;
  const uint32_t id = in ? cand[t] : 0u;
#pragma unroll
  for (int k = 0; k < D; ++k) v[k] = in ? x[(uint64_t)k * n_pad + id] : 0.f;
#pragma unroll
  for (int k = 0; k < D; ++k) {
    const uint32_t u = ordered_u32(v[k]);
    const uint32_t lo = __reduce_min_sync(kAllLanes, in ? u : 0xffffffffu);
    const uint32_t hi = __reduce_max_sync(kAllLanes, in ? u : 0u);
    if (lane == 0) {
      atomicMin(&s_lo[k], lo);
      atomicMax(&s_hi[k], hi);
    }
  }
  const bool sky = in && cand_st[t] == 0;
  const uint32_t ball = __ballot_sync(kAllLanes, sky);
  if (lane == 0) s_w[wid] = __popc(ball);
  __syncthreads();
  uint32_t j = __popc(ball & ((1u << lane) - 1u)), mq = 0;
  for (uint32_t w = 0; w < 32; ++w) {
    if (w < wid) j += s_w[w];
    mq += s_w[w];
  }
  if (in) {
    uint32_t w[4] = {0, 0, 0, 0};
    const float top = (float)((1u << depth) - 1u);
#pragma unroll
    for (int k = 0; k < D; ++k) {
      const uint32_t a = s_lo[k], b = s_hi[k];
      const float lo = __uint_as_float((a & 0x80000000u) ? (a & 0x7fffffffu) : ~a);
      const float hi = __uint_as_float((b & 0x80000000u) ? (b & 0x7fffffffu) : ~b);
      const float scale = (top + 1.0f) / (hi - lo);
      // a degenerate range (one value, overflow) has one cell
      const float c = scale < 3.0e38f && hi - lo < 3.0e38f ? (v[k] - lo) * scale : 0.f;
      w[k >> 2] |= (uint32_t)fminf(c, top) << (8 * (k & 3));
      px[(uint64_t)k * pitch + t] = v[k];
    }
    const uint4 c4 = make_uint4(w[0], w[1], w[2], w[3]);
    cells[t] = c4;
    if (sky) {
      qcells[j] = c4;
#pragma unroll
      for (int k = 0; k < D; ++k) qx[(uint64_t)k * pitch + j] = v[k];
    }
  }
  const uint32_t pad = (mq + 31) & ~31u;
  if (t >= mq && t < pad) {  // entries that add nothing (k_q_scatter)
    qcells[t] = make_uint4(0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu);
#pragma unroll
    for (int k = 0; k < D; ++k) qx[(uint64_t)k * pitch + t] = __int_as_float(0x7f800000);
  }
  if (t == 0) {
    boff[0] = 0;
    boff[1] = mq;
    *work = 0;
  }
  __syncthreads();
  if (wid * 32 >= pad) return;
  uint4 c = qcells[t];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    c.x = __vminu4(c.x, __shfl_xor_sync(kAllLanes, c.x, o));
    c.y = __vminu4(c.y, __shfl_xor_sync(kAllLanes, c.y, o));
    c.z = __vminu4(c.z, __shfl_xor_sync(kAllLanes, c.z, o));
    c.w = __vminu4(c.w, __shfl_xor_sync(kAllLanes, c.w, o));
    if (o == 2 && (lane & 3) == 0) hmin[wid * 8 + (lane >> 2)] = c;
    if (o == 4 && (lane & 7) == 0) smin[wid * 4 + (lane >> 3)] = c;
  }
  if (lane == 0) bmin[wid] = c;
}

int launch_small_prep(cudaStream_t s, int d, const float* x, uint64_t n_pad, const uint32_t* cand,
                      const uint8_t* cand_st, const uint32_t* m_ptr, uint64_t m_max, int depth,
                      uint64_t pitch, uint4* cells, float* px, uint4* qcells, float* qx,
                      uint4* bmin, uint4* smin, uint4* hmin, uint32_t* boff, uint32_t* work) {
  if (m_max > kSmallCandidates)
    return set_error(SKC_ERR_INVALID, "%llu candidates for the one-CTA preparation",
                     (unsigned long long)m_max);
  switch (d) {
#define SKC_PREP_CASE(D)                                                                        \
  case D:                                                                                       \
    k_small_prep<D><<<1, kSmallCandidates, 0, s>>>(x, n_pad, cand, cand_st, m_ptr, depth, pitch, \
                                                   cells, px, qcells, qx, bmin, smin, hmin, boff, \
                                                   work);                                       \
    break;
    SKC_PREP_CASE(2) SKC_PREP_CASE(3) SKC_PREP_CASE(4) SKC_PREP_CASE(5) SKC_PREP_CASE(6)
    SKC_PREP_CASE(7) SKC_PREP_CASE(8) SKC_PREP_CASE(9) SKC_PREP_CASE(10) SKC_PREP_CASE(11)
    SKC_PREP_CASE(12) SKC_PREP_CASE(13) SKC_PREP_CASE(14) SKC_PREP_CASE(15) SKC_PREP_CASE(16)
#undef SKC_PREP_CASE
    default:
      return set_error(SKC_ERR_INVALID, "unsupported d=%d", d);
  }
  SKC_LAUNCH_CHECK();
  return SKC_OK;
}

// Offsets of a result that holds one cuboid, S, for both of its lists:
// off[c] = 0 up to S and the list's count above.
__global__ void k_single_offsets(const uint32_t* __restrict__ n, uint32_t S, uint32_t nsub,
                                 uint64_t* __restrict__ sky_off, uint64_t* __restrict__ ext_off) {
  const uint64_t n0 = n[0], n1 = n[1];
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c <= nsub;
       c += gridDim.x * blockDim.x) {
    sky_off[c] = c > S ? n0 : 0;
    ext_off[c] = c > S ? n1 : 0;
  }
}

int launch_single_offsets(cudaStream_t s, const uint32_t* n, uint32_t S, uint32_t nsub,
                          uint64_t* sky_off, uint64_t* ext_off) {
  k_single_offsets<<<(nsub + 256) / 256, 256, 0, s>>>(n, S, nsub, sky_off, ext_off);
  SKC_LAUNCH_CHECK();
  return SKC_OK;
}

}  // namespace skc
