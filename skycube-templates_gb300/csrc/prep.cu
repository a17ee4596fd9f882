// Data-preparation kernels of the skycube engine: upload into attribute-major
// layout, Manhattan-norm scores and bucket keys, a counting sort by bucket,
// grid pivots and cells, order-preserving compaction and scans.
//
// Every kernel that works on a point list reads the list length from device
// memory (m_ptr), so a whole pipeline can be enqueued, or captured in a CUDA
// graph, before any length is known on the host.
#include <algorithm>
#include <cfloat>
#include <cstdio>

#include "kernels.cuh"

namespace skc {

// --------------------------------------------------------------------------
// Upload: row-major n x d -> attribute-major x[k * n_pad + i]. Counts
// non-finite values into *bad (NaN would break every ordering below).
__global__ void k_rows_to_soa(const float* __restrict__ rows, uint64_t n, int d,
                              uint64_t n_pad, float* __restrict__ x,
                              uint32_t* __restrict__ bad) {
  const uint64_t total = n * (uint64_t)d;
  uint32_t nbad = 0;
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < total;
       t += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t i = t / d;
    const int k = (int)(t - i * d);
    const float v = rows[t];
    nbad += !isfinite(v);
    x[(uint64_t)k * n_pad + i] = v;
  }
  if (nbad) atomicAdd(bad, nbad);
}

__device__ __forceinline__ float u2f_ordered(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// f[i] = sum of the attributes in S of point ids[i], in increasing attribute
// order. Summing in a fixed order makes f monotone: q <= p on S implies
// f(q) <= f(p) (float addition is monotone in each operand).
// minmax[0] / minmax[1] receive the ordered-uint min / max of f.
__global__ void k_score(const float* __restrict__ x, uint64_t n_pad,
                        const uint32_t* __restrict__ ids,
                        const uint32_t* __restrict__ m_ptr, uint32_t S, int d,
                        float* __restrict__ f, uint32_t* __restrict__ minmax) {
  const uint32_t m = *m_ptr;
  uint32_t lo = 0xffffffffu, hi = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += gridDim.x * blockDim.x) {
    const uint32_t id = ids ? ids[i] : i;
    float s = 0.f;
    for (int k = 0; k < d; ++k)
      if (S & (1u << k)) s += x[(uint64_t)k * n_pad + id];
    f[i] = s;
    const uint32_t u = ordered_u32(s);
    lo = min(lo, u);
    hi = max(hi, u);
  }
  for (int o = 16; o; o >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMin(&minmax[0], lo);
    atomicMax(&minmax[1], hi);
  }
}

// key = floor((f - fmin) * (K - 1) / (fmax - fmin)), clamped to [0, K-1].
// Each step is monotone in f, so f(q) <= f(p) implies key(q) <= key(p).
__global__ void k_fkeys(const float* __restrict__ f,
                        const uint32_t* __restrict__ m_ptr,
                        const uint32_t* __restrict__ minmax, uint32_t K,
                        uint32_t* __restrict__ keys) {
  const uint32_t m = *m_ptr;
  const float fmin = u2f_ordered(minmax[0]), fmax = u2f_ordered(minmax[1]);
  const float range = fmax - fmin;
  const float scale = (range > 0.f && isfinite(range)) ? (float)(K - 1) / range : 0.f;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += gridDim.x * blockDim.x) {
    float t = (f[i] - fmin) * scale;
    uint32_t k = t <= 0.f ? 0u : (t >= (float)(K - 1) ? K - 1 : (uint32_t)t);
    keys[i] = k;
  }
}

__global__ void k_hist(const uint32_t* __restrict__ keys,
                       const uint32_t* __restrict__ m_ptr,
                       uint32_t* __restrict__ counts) {
  const uint32_t m = *m_ptr;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += gridDim.x * blockDim.x)
    atomicAdd(&counts[keys[i]], 1u);
}

// In-place exclusive scan of a[0 .. len) with one CTA of 1024 threads;
// a[len] receives the total. len + 1 entries must be allocated. The array is
// walked in tiles of 4096 (4 consecutive entries per thread, so each warp
// reads and writes 512 contiguous bytes), each tile scanned in the block and
// offset by the running total of the tiles before it.
template <typename T>
__global__ void __launch_bounds__(1024) k_scan_single(T* __restrict__ a,
                                                      uint32_t len) {
  __shared__ T warp_excl[32];
  __shared__ T tile_tot;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  T carry = 0;  // total of the tiles before this one (same in every thread)
  for (uint32_t base = 0; base < len; base += 4096) {
    T v[4];
    T local = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t i = base + 4 * threadIdx.x + j;
      v[j] = i < len ? a[i] : T(0);
      local += v[j];
    }
    T incl = local;
    for (int o = 1; o < 32; o <<= 1) {
      const T u = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += u;
    }
    if (lane == 31) warp_excl[wid] = incl;  // warp totals for now
    __syncthreads();
    if (wid == 0) {
      const T w = warp_excl[lane];
      T sw = w;
      for (int o = 1; o < 32; o <<= 1) {
        const T u = __shfl_up_sync(0xffffffffu, sw, o);
        if (lane >= o) sw += u;
      }
      warp_excl[lane] = sw - w;
      if (lane == 31) tile_tot = sw;
    }
    __syncthreads();
    T run = carry + warp_excl[wid] + incl - local;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t i = base + 4 * threadIdx.x + j;
      if (i < len) a[i] = run;
      run += v[j];
    }
    carry += tile_tot;
    __syncthreads();  // warp_excl and tile_tot are reused by the next tile
  }
  if (threadIdx.x == 0) a[len] = carry;
}

// Scatters item i to its bucket. sorted[pos] = i; hi[pos] = end of i's
// bucket in sorted order. Order inside a bucket is unspecified; every user
// of the order is insensitive to it.
__global__ void k_scatter(const uint32_t* __restrict__ keys,
                          const uint32_t* __restrict__ m_ptr,
                          const uint32_t* __restrict__ offsets,
                          uint32_t* __restrict__ cursor,
                          uint32_t* __restrict__ sorted,
                          uint32_t* __restrict__ hi) {
  const uint32_t m = *m_ptr;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += gridDim.x * blockDim.x) {
    const uint32_t k = keys[i];
    const uint32_t pos = offsets[k] + atomicAdd(&cursor[k], 1u);
    sorted[pos] = i;
    if (hi) hi[pos] = offsets[k + 1];
  }
}

// --------------------------------------------------------------------------
// Pivots: one CTA per attribute samples up to kPivotSample values of the
// list (evenly strided), sorts them in shared memory and keeps
// 2^depth - 1 evenly spaced order statistics. Any pivot set is correct;
// quantiles only make the cells informative.
constexpr int kPivotSample = 4096;

// One compare-exchange stage of the bitonic sort below on a thread's four
// consecutive elements e, e + 1, e + 2, e + 3 (e = 4 * thread): stride 1 and
// 2 stay in the thread, strides 4 .. 64 meet lane ^ (stride / 4).
template <int STRIDE>
__device__ __forceinline__ void sort_stage(float (&v)[4], int e, int size) {
  const bool up = (e & size) == 0;  // size >= 4: the same for all four
  if constexpr (STRIDE >= 4) {
    const bool take_min = ((e & STRIDE) == 0) == up;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float o = __shfl_xor_sync(0xffffffffu, v[j], STRIDE / 4);
      v[j] = take_min ? fminf(v[j], o) : fmaxf(v[j], o);
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (j & STRIDE) continue;
      const float lo = fminf(v[j], v[j | STRIDE]), hi = fmaxf(v[j], v[j | STRIDE]);
      v[j] = up ? lo : hi;
      v[j | STRIDE] = up ? hi : lo;
    }
  }
}

// Ascending bitonic sort of s[0 .. 4096) by 1,024 threads; s[cnt ..) holds
// FLT_MAX, so only the smallest power of two >= cnt is sorted. A thread owns
// four consecutive elements: strides up to 64 are exchanged in registers and
// by shuffles inside the warp's 128 elements, only strides of 128 and more go
// through shared memory (15 exchanges of the 78 stages, which a barrier per
// stage made a chain of 78 barriers). k_pivots on one GB300: 26 -> 8.5 us.
__device__ __forceinline__ void sort_sample(float* s, uint32_t cnt) {
  const int e = 4 * threadIdx.x;
  float v[4];
  const float4 in = *reinterpret_cast<const float4*>(s + e);
  v[0] = in.x; v[1] = in.y; v[2] = in.z; v[3] = in.w;
  // size 2: pairs (0, 1) ascending, (2, 3) descending
  {
    const float a = fminf(v[0], v[1]), b = fmaxf(v[0], v[1]);
    const float c = fmaxf(v[2], v[3]), d = fminf(v[2], v[3]);
    v[0] = a; v[1] = b; v[2] = c; v[3] = d;
  }
  for (int size = 4; size <= kPivotSample && (uint32_t)(size >> 1) < cnt; size <<= 1) {
    if (size > 128) {
      for (int stride = size >> 1; stride >= 128; stride >>= 1) {
        *reinterpret_cast<float4*>(s + e) = make_float4(v[0], v[1], v[2], v[3]);
        __syncthreads();
        const float4 o = *reinterpret_cast<const float4*>(s + (e ^ stride));
        const bool take_min = ((e & stride) == 0) == ((e & size) == 0);
        v[0] = take_min ? fminf(v[0], o.x) : fmaxf(v[0], o.x);
        v[1] = take_min ? fminf(v[1], o.y) : fmaxf(v[1], o.y);
        v[2] = take_min ? fminf(v[2], o.z) : fmaxf(v[2], o.z);
        v[3] = take_min ? fminf(v[3], o.w) : fmaxf(v[3], o.w);
        __syncthreads();
      }
    }
    if (size >= 128) sort_stage<64>(v, e, size);
    if (size >= 64) sort_stage<32>(v, e, size);
    if (size >= 32) sort_stage<16>(v, e, size);
    if (size >= 16) sort_stage<8>(v, e, size);
    if (size >= 8) sort_stage<4>(v, e, size);
    sort_stage<2>(v, e, size);
    sort_stage<1>(v, e, size);
  }
  *reinterpret_cast<float4*>(s + e) = make_float4(v[0], v[1], v[2], v[3]);
  __syncthreads();
}

__global__ void __launch_bounds__(1024) k_pivots(
    const float* __restrict__ x, uint64_t n_pad, const uint32_t* __restrict__ ids,
    const uint32_t* __restrict__ m_ptr, int depth, float* __restrict__ pivots,
    uint32_t* __restrict__ amin, uint32_t* __restrict__ hist, int low) {
  __shared__ __align__(16) float s[kPivotSample];
  const int k = blockIdx.x;
  if (amin && threadIdx.x == 0) amin[k] = 0xffffffffu;  // k_cells lowers it
  if (hist && k == 0)
    for (uint32_t t = threadIdx.x; t < kSumBins + 8; t += blockDim.x) hist[t] = 0;
  const uint32_t m = *m_ptr;
  const uint32_t cnt = m < kPivotSample ? m : kPivotSample;
  for (int t = threadIdx.x; t < kPivotSample; t += blockDim.x) {
    float v = FLT_MAX;
    if ((uint32_t)t < cnt) {
      const uint32_t i = (uint32_t)(((uint64_t)t * m) / cnt);
      const uint32_t id = ids ? ids[i] : i;
      v = x[(uint64_t)k * n_pad + id];
    }
    s[t] = v;
  }
  __syncthreads();
  sort_sample(s, cnt);
  // `low`: quadratic ranks, cells finer towards the minimum.
  const int P = (1 << depth) - 1;
  for (int r = threadIdx.x; r < kMaxPivots; r += blockDim.x) {
    float v = FLT_MAX;
    if (r < P && cnt > 0) {
      const uint64_t at = (uint64_t)(r + 1) * cnt;
      v = s[low ? at * (r + 1) / ((uint64_t)(P + 1) * (P + 1)) : at / (P + 1)];
    }
    pivots[k * kMaxPivots + r] = v;
  }
}

// cells[i] = grid cells of point ids[i] (see common.cuh). With `amin`, also
// lowers amin[k] to the ordered-uint minimum of attribute k over the list;
// with `hist` (and amin), the histogram of the points' cell sums for the
// prefilter; with `xout`, the list's floats in list order (xout[k * out_pad
// + i]). What a later kernel would read the points again for is written here.
// The D values are loaded before any search, and a search is `depth`
// branch-free steps, so a thread has D independent chains in flight. The
// pivots lie in shared memory level by level: up to 32 nodes of one level
// are 32 consecutive words, so a step has no bank conflicts until the last
// level (in sorted order a level's nodes share a few banks).
template <int D>
__global__ void __launch_bounds__(256) k_cells(
    const float* __restrict__ x, uint64_t n_pad, const uint32_t* __restrict__ ids,
    const uint32_t* __restrict__ m_ptr, int depth, const float* __restrict__ pivots,
    uint4* __restrict__ cells, uint32_t* __restrict__ amin, uint32_t* __restrict__ hist,
    float* __restrict__ xout, uint64_t out_pad) {
  __shared__ float piv[D * (kMaxPivots + 1)];
  __shared__ uint32_t s_min[D];
  __shared__ uint32_t s_hist[kSumBins];
  if (hist)
    for (uint32_t t = threadIdx.x; t < kSumBins; t += blockDim.x) s_hist[t] = 0;
  // Node i of the search tree (its levels one after the other).
  for (int t = threadIdx.x; t < D * (kMaxPivots + 1); t += blockDim.x) {
    const int k = t / (kMaxPivots + 1), i = t % (kMaxPivots + 1);
    const int l = 31 - __clz(i + 1);
    if (l < depth)
      piv[t] = pivots[k * kMaxPivots + ((2 * (i + 1 - (1 << l)) + 1) << (depth - 1 - l)) - 1];
  }
  if (threadIdx.x < D) s_min[threadIdx.x] = 0xffffffffu;
  __syncthreads();
  const uint32_t m = *m_ptr;
  float mn[D];
#pragma unroll
  for (int k = 0; k < D; ++k) mn[k] = FLT_MAX;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += gridDim.x * blockDim.x) {
    const uint32_t id = ids ? ids[i] : i;
    float v[D];
#pragma unroll
    for (int k = 0; k < D; ++k) v[k] = x[(uint64_t)k * n_pad + id];
    uint32_t lo[D];
#pragma unroll
    for (int k = 0; k < D; ++k) {
      lo[k] = 0;
      mn[k] = fminf(mn[k], v[k]);
    }
    for (int l = 0; l < depth; ++l) {
#pragma unroll
      for (int k = 0; k < D; ++k)
        lo[k] = 2 * lo[k] + 1 + (piv[k * (kMaxPivots + 1) + lo[k]] < v[k] ? 1u : 0u);
    }
#pragma unroll
    for (int k = 0; k < D; ++k) lo[k] -= (1u << depth) - 1u;  // pivots below v
    uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
    for (int k = 0; k < D; ++k) w[k >> 2] |= lo[k] << (8 * (k & 3));
    cells[i] = make_uint4(w[0], w[1], w[2], w[3]);
    if (xout) {
#pragma unroll
      for (int k = 0; k < D; ++k) xout[(uint64_t)k * out_pad + i] = v[k];
    }
    if (hist) {
      uint32_t sum = 0;
#pragma unroll
      for (int k = 0; k < D; ++k) sum += lo[k];
      atomicAdd(&s_hist[sum], 1u);
    }
  }
  if (!amin) return;
#pragma unroll
  for (int k = 0; k < D; ++k) {
    const uint32_t u = __reduce_min_sync(0xffffffffu, ordered_u32(mn[k]));
    if ((threadIdx.x & 31) == 0) atomicMin(&s_min[k], u);
  }
  __syncthreads();
  if (threadIdx.x < D) atomicMin(&amin[threadIdx.x], s_min[threadIdx.x]);
  if (hist)
    for (uint32_t t = threadIdx.x; t < kSumBins; t += blockDim.x)
      if (s_hist[t]) atomicAdd(&hist[t], s_hist[t]);
}

// --------------------------------------------------------------------------
// Order-preserving compaction of a status array in blocks of 1024 entries:
// entries with status 0 go to out0, with status 1 to out1, both together to
// both_out (status 2 and above is dropped). k_status_count counts a block's
// entries per status; k_status_write places them. A block adds up the counts
// of the blocks before it itself: at most kSelfScanBlocks of them, four loads
// a thread, instead of a scan launch per output (a compaction took four
// launches, and the union of two outputs four more). Longer lists scan first.
constexpr uint32_t kSelfScanBlocks = 4096;

__global__ void __launch_bounds__(1024) k_status_count(
    const uint8_t* __restrict__ st, const uint32_t* __restrict__ m_ptr,
    uint32_t* __restrict__ c0, uint32_t* __restrict__ c1) {
  __shared__ uint32_t s0[32], s1[32];
  const uint32_t m = *m_ptr;
  const uint32_t nblk = (m + 1023) / 1024;
  if (blockIdx.x >= nblk) {  // the scan of a longer list reads these
    if (threadIdx.x == 0) { c0[blockIdx.x] = 0; c1[blockIdx.x] = 0; }
    return;
  }
  const uint32_t i = blockIdx.x * 1024 + threadIdx.x;
  const uint8_t v = i < m ? st[i] : 2;
  const uint32_t b0 = __ballot_sync(0xffffffffu, v == 0);
  const uint32_t b1 = __ballot_sync(0xffffffffu, v == 1);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) { s0[wid] = __popc(b0); s1[wid] = __popc(b1); }
  __syncthreads();
  if (wid == 0) {
    const uint32_t a = __reduce_add_sync(0xffffffffu, s0[lane]);
    const uint32_t b = __reduce_add_sync(0xffffffffu, s1[lane]);
    if (lane == 0) { c0[blockIdx.x] = a; c1[blockIdx.x] = b; }
  }
}

struct StatusOut {
  uint32_t* out0;      // ids with status 0
  uint32_t* out1;      // ids with status 1, or nullptr
  uint32_t* both;      // ids with status 0 or 1, or nullptr
  uint8_t* both_st;    // per entry of `both`: 0 for status 0, else 2
  uint32_t* pos0;      // per entry of out0: its position in `both`
  uint32_t* n;         // [0] entries of out0, and with out1 [1] of out1, [2] of both
};

__global__ void __launch_bounds__(1024) k_status_write(
    const uint8_t* __restrict__ st, const uint32_t* __restrict__ ids,
    const uint32_t* __restrict__ m_ptr, const uint32_t* __restrict__ c0,
    const uint32_t* __restrict__ c1, int scanned, StatusOut o) {
  __shared__ uint32_t s0[32], s1[32], p0[32], p1[32];
  const uint32_t m = *m_ptr;
  const uint32_t nblk = (m + 1023) / 1024;
  const uint32_t b = blockIdx.x;
  if (nblk == 0) {
    if (b == 0 && threadIdx.x == 0) {
      o.n[0] = 0;
      if (o.out1) o.n[1] = o.n[2] = 0;
    }
    return;
  }
  if (b >= nblk) return;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t i = b * 1024 + threadIdx.x;
  const uint8_t v = i < m ? st[i] : 2;
  const uint32_t b0 = __ballot_sync(0xffffffffu, v == 0);
  const uint32_t b1 = __ballot_sync(0xffffffffu, v == 1);
  uint32_t f0 = 0, f1 = 0;  // entries of the blocks before this one
  if (scanned) {
    if (threadIdx.x == 0) { f0 = c0[b]; if (o.out1) f1 = c1[b]; }
  } else {
    for (uint32_t j = threadIdx.x; j < b; j += 1024) {
      f0 += c0[j];
      if (o.out1) f1 += c1[j];
    }
  }
  f0 = __reduce_add_sync(0xffffffffu, f0);
  f1 = __reduce_add_sync(0xffffffffu, f1);
  if (lane == 0) {
    s0[wid] = __popc(b0);
    s1[wid] = __popc(b1);
    p0[wid] = f0;
    p1[wid] = f1;
  }
  __syncthreads();
  if (wid == 0) {
    const uint32_t a = s0[lane], c = s1[lane];
    uint32_t ia = a, ic = c;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, ia, k);
      const uint32_t w = __shfl_up_sync(0xffffffffu, ic, k);
      if (lane >= k) { ia += u; ic += w; }
    }
    const uint32_t q0 = __reduce_add_sync(0xffffffffu, p0[lane]);
    const uint32_t q1 = __reduce_add_sync(0xffffffffu, p1[lane]);
    s0[lane] = q0 + ia - a;
    s1[lane] = q1 + ic - c;
    if (lane == 31 && b == nblk - 1) {
      o.n[0] = q0 + ia;
      if (o.out1) {
        o.n[1] = q1 + ic;
        o.n[2] = q0 + ia + q1 + ic;
      }
    }
  }
  __syncthreads();
  const uint32_t lt = (1u << lane) - 1u;
  if (v > 1) return;
  const uint32_t id = ids ? ids[i] : i;
  const uint32_t k0 = s0[wid] + __popc(b0 & lt), k1 = s1[wid] + __popc(b1 & lt);
  if (v == 0) o.out0[k0] = id;
  else if (o.out1) o.out1[k1] = id;
  if (o.both) {  // statuses 0 and 1 in list order
    o.both[k0 + k1] = id;
    o.both_st[k0 + k1] = v == 0 ? 0 : 2;
    if (v == 0) o.pos0[k0] = k0 + k1;
  }
}

// --------------------------------------------------------------------------
// Multi-block exclusive scan of uint32 counts into uint64 offsets:
// out[i] = sum(in[0..i)), out[len] = total. Three phases.
constexpr int kScanBlock = 4096;

__global__ void __launch_bounds__(1024) k_scan_partials(
    const uint32_t* __restrict__ in, uint64_t len, uint64_t* __restrict__ bsum) {
  __shared__ uint64_t red[32];
  const uint64_t beg = (uint64_t)blockIdx.x * kScanBlock;
  uint64_t s = 0;
  for (int t = threadIdx.x; t < kScanBlock; t += 1024) {
    const uint64_t i = beg + t;
    if (i < len) s += in[i];
  }
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = red[threadIdx.x];
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) bsum[blockIdx.x] = s;
  }
}

// A CTA adds up the block sums before its own itself (`scanned` 0; at most
// kSelfScanBlocks of them), or reads their scan. With csr_off, out[c * T] goes
// to csr_off[c] for c <= nsub as well.
__global__ void __launch_bounds__(1024) k_scan_apply(
    const uint32_t* __restrict__ in, uint64_t len, const uint64_t* __restrict__ bsum,
    int scanned, uint64_t* __restrict__ out, uint32_t T, uint32_t nsub,
    uint64_t* __restrict__ csr_off) {
  __shared__ uint64_t wt[32], pre[32];
  const uint64_t beg = (uint64_t)blockIdx.x * kScanBlock;
  constexpr int per = kScanBlock / 1024;  // 4 consecutive items per thread
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint64_t before = 0;
  if (scanned) {
    if (threadIdx.x == 0) before = bsum[blockIdx.x];
  } else {
    for (uint32_t j = threadIdx.x; j < blockIdx.x; j += 1024) before += bsum[j];
  }
  uint32_t v[per];
  uint64_t local = 0;
  const uint64_t at = beg + threadIdx.x * per;
#pragma unroll
  for (int j = 0; j < per; ++j) {
    v[j] = at + j < len ? in[at + j] : 0;
    local += v[j];
  }
  uint64_t incl = local;
  for (int o = 1; o < 32; o <<= 1) {
    uint64_t u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
    before += __shfl_xor_sync(0xffffffffu, before, o);
  }
  if (lane == 31) {
    wt[wid] = incl;
    pre[wid] = before;
  }
  __syncthreads();
  if (wid == 0) {
    uint64_t a = wt[lane], s = a, p = pre[lane];
    for (int o = 1; o < 32; o <<= 1) {
      uint64_t u = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += u;
      p += __shfl_xor_sync(0xffffffffu, p, o);
    }
    wt[lane] = p + s - a;
  }
  __syncthreads();
  uint64_t run = wt[wid] + incl - local;
  uint64_t c = at / T;  // column of the next item that starts one
  if (c * T < at) ++c;
#pragma unroll
  for (int j = 0; j < per; ++j) {
    const uint64_t i = at + j;
    if (i < len) {
      out[i] = run;
      if (i == c * T) {
        if (c <= nsub) csr_off[c] = run;
        ++c;
      }
      run += v[j];
      if (i == len - 1) {
        out[len] = run;
        if (len == (uint64_t)nsub * T) csr_off[nsub] = run;
      }
    }
  }
}

// --------------------------------------------------------------------------
// Per block of 32 consecutive q's, per 8-q quarter and per 4-q half of a
// quarter: byte-wise
// minimum of their cells. Padding entries (index >= m) get cell 127 so they
// never lower the minimum.
__global__ void k_block_min(const uint4* __restrict__ cells,
                            const uint32_t* __restrict__ m_ptr,
                            uint4* __restrict__ bmin, uint4* __restrict__ smin,
                            uint4* __restrict__ hmin) {
  const uint32_t m = *m_ptr;
  const uint32_t nblk = (m + 31) / 32;
  const int lane = threadIdx.x & 31;
  for (uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < nblk;
       b += (gridDim.x * blockDim.x) >> 5) {
    const uint32_t i = b * 32 + lane;
    uint4 c = i < m ? cells[i] : make_uint4(0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu);
    for (int o = 1; o < 32; o <<= 1) {
      c.x = __vminu4(c.x, __shfl_xor_sync(0xffffffffu, c.x, o));
      c.y = __vminu4(c.y, __shfl_xor_sync(0xffffffffu, c.y, o));
      c.z = __vminu4(c.z, __shfl_xor_sync(0xffffffffu, c.z, o));
      c.w = __vminu4(c.w, __shfl_xor_sync(0xffffffffu, c.w, o));
      if (o == 2 && (lane & 3) == 0) hmin[(uint64_t)b * 8 + (lane >> 2)] = c;
      if (o == 4 && (lane & 7) == 0) smin[(uint64_t)b * 4 + (lane >> 3)] = c;
    }
    if (lane == 0) bmin[b] = c;
  }
}

// Gathers per-cuboid lists held in separate buffers into one CSR:
// cuboid c's list srcs[c] goes to dst[dst_off[c] .. dst_off[c+1]).
__global__ void k_csr_gather(const uint32_t* const* __restrict__ srcs,
                             const uint64_t* __restrict__ dst_off,
                             uint32_t* __restrict__ dst) {
  const uint32_t c = blockIdx.x;
  const uint32_t* src = srcs[c];
  const uint64_t n = dst_off[c + 1] - dst_off[c];
  if (!src) return;
  const uint64_t o = dst_off[c];
  for (uint64_t i = threadIdx.x; i < n; i += blockDim.x) dst[o + i] = src[i];
}

__global__ void k_set_u32(uint32_t* p, uint32_t v, uint32_t zeros) {
  p[0] = v;
  for (uint32_t i = 1; i <= zeros; ++i) p[i] = 0;
}

// Merges two ascending, disjoint id lists a[0..na) and b[0..nb) into
// out[0..na+nb) (ascending): every element finds its rank in the other list
// by binary search.
__global__ void k_merge_disjoint(const uint32_t* __restrict__ a, uint32_t na,
                                 const uint32_t* __restrict__ b, uint32_t nb,
                                 uint32_t* __restrict__ out, uint32_t* __restrict__ n) {
  const uint32_t total = na + nb;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    n[0] = total;
    n[1] = 0;
  }
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += gridDim.x * blockDim.x) {
    const bool from_a = i < na;
    const uint32_t v = from_a ? a[i] : b[i - na];
    const uint32_t* o = from_a ? b : a;
    uint32_t lo = 0, hi = from_a ? nb : na;
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (o[mid] < v) lo = mid + 1; else hi = mid;
    }
    out[(from_a ? i : i - na) + lo] = v;
  }
}

// ==========================================================================
// Host-side launch helpers.
static inline unsigned grid_for(uint64_t items, int threads, int max_blocks) {
  uint64_t b = (items + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > (uint64_t)max_blocks) b = max_blocks;
  return (unsigned)b;
}

int launch_rows_to_soa(cudaStream_t s, const float* rows, uint64_t n, int d,
                       uint64_t n_pad, float* x, uint32_t* bad) {
  k_rows_to_soa<<<grid_for(n * d, 256, 152 * 32), 256, 0, s>>>(rows, n, d, n_pad, x, bad);
  SKC_LAUNCH_CHECK();
  return SKC_OK;
}

int launch_bucket_order(cudaStream_t s, const float* x, uint64_t n_pad, int d,
                        const uint32_t* ids, const uint32_t* m_ptr,
                        uint64_t m_max, uint32_t S, uint32_t K,
                        const BucketScratch& b, uint32_t* sorted, uint32_t* hi) {
  SKC_CUDA(cudaMemsetAsync(b.minmax, 0, 2 * sizeof(uint32_t), s));
  SKC_CUDA(cudaMemsetAsync(b.minmax, 0xff, sizeof(uint32_t), s));
  const unsigned g = grid_for(m_max, 256, 152 * 8);
  k_score<<<g, 256, 0, s>>>(x, n_pad, ids, m_ptr, S, d, b.f, b.minmax);
  SKC_LAUNCH_CHECK();
  k_fkeys<<<g, 256, 0, s>>>(b.f, m_ptr, b.minmax, K, b.keys);
  SKC_LAUNCH_CHECK();
  return launch_counting_sort(s, b.keys, m_ptr, m_max, K, b, sorted, hi);
}

int launch_counting_sort(cudaStream_t s, const uint32_t* keys,
                         const uint32_t* m_ptr, uint64_t m_max, uint32_t K,
                         const BucketScratch& b, uint32_t* sorted, uint32_t* hi) {
  SKC_CUDA(cudaMemsetAsync(b.counts, 0, (K + 1) * sizeof(uint32_t), s));
  SKC_CUDA(cudaMemsetAsync(b.cursor, 0, (K + 1) * sizeof(uint32_t), s));
  const unsigned g = grid_for(m_max, 256, 152 * 8);
  k_hist<<<g, 256, 0, s>>>(keys, m_ptr, b.counts);
  SKC_LAUNCH_CHECK();
  k_scan_single<uint32_t><<<1, 1024, 0, s>>>(b.counts, K);
  SKC_LAUNCH_CHECK();
  k_scatter<<<g, 256, 0, s>>>(keys, m_ptr, b.counts, b.cursor, sorted, hi);
  SKC_LAUNCH_CHECK();
  return SKC_OK;
}

template <int D>
static int launch_cells(cudaStream_t s, const float* x, uint64_t n_pad, const uint32_t* ids,
                        const uint32_t* m_ptr, uint64_t m_max, int depth, const float* pivots,
                        uint4* cells, uint32_t* amin, uint32_t* hist, float* xout,
                        uint64_t out_pad) {
  k_cells<D><<<grid_for(m_max, 256, 152 * 6), 256, 0, s>>>(x, n_pad, ids, m_ptr, depth, pivots,
                                                            cells, amin, hist, xout, out_pad);
  SKC_LAUNCH_CHECK();
  return SKC_OK;
}

int launch_pivots_cells(cudaStream_t s, const float* x, uint64_t n_pad, int d,
                        const uint32_t* ids, const uint32_t* m_ptr,
                        uint64_t m_max, int depth, float* pivots, uint4* cells, uint32_t* amin,
                        uint32_t* hist, float* xout, uint64_t out_pad, int low) {
  k_pivots<<<d, 1024, 0, s>>>(x, n_pad, ids, m_ptr, depth, pivots, amin, hist, low);
  SKC_LAUNCH_CHECK();
  switch (d) {
#define SKC_CELLS_CASE(D) \
  case D:                                                                               \
    return launch_cells<D>(s, x, n_pad, ids, m_ptr, m_max, depth, pivots, cells, amin, hist, \
                           xout, out_pad);
    SKC_CELLS_CASE(2) SKC_CELLS_CASE(3) SKC_CELLS_CASE(4) SKC_CELLS_CASE(5) SKC_CELLS_CASE(6)
    SKC_CELLS_CASE(7) SKC_CELLS_CASE(8) SKC_CELLS_CASE(9) SKC_CELLS_CASE(10) SKC_CELLS_CASE(11)
    SKC_CELLS_CASE(12) SKC_CELLS_CASE(13) SKC_CELLS_CASE(14) SKC_CELLS_CASE(15)
    SKC_CELLS_CASE(16)
#undef SKC_CELLS_CASE
    default:
      return set_error(SKC_ERR_INVALID, "unsupported d=%d", d);
  }
}

// Statuses whose block counts c0 / c1 are already there (c1 unused without
// out1) into the outputs.
static int status_write(cudaStream_t s, const uint8_t* st, const uint32_t* ids,
                        const uint32_t* m_ptr, uint64_t m_max, uint32_t* c0, uint32_t* c1,
                        const StatusOut& o) {
  const uint32_t g = (uint32_t)std::max<uint64_t>(1, (m_max + 1023) / 1024);
  const int scan = g > kSelfScanBlocks;
  if (scan) {
    k_scan_single<uint32_t><<<1, 1024, 0, s>>>(c0, g);
    SKC_LAUNCH_CHECK();
    if (o.out1) {
      k_scan_single<uint32_t><<<1, 1024, 0, s>>>(c1, g);
      SKC_LAUNCH_CHECK();
    }
  }
  k_status_write<<<g, 1024, 0, s>>>(st, ids, m_ptr, c0, c1, scan, o);
  SKC_LAUNCH_CHECK();
  return SKC_OK;
}

int launch_status_split(cudaStream_t s, const uint8_t* st, const uint32_t* ids,
                        const uint32_t* m_ptr, uint64_t m_max, uint32_t* blk0, uint32_t* blk1,
                        uint32_t* sky, uint32_t* ext, uint32_t* n, uint32_t* both,
                        uint8_t* both_st, uint32_t* pos0) {
  const uint32_t g = (uint32_t)std::max<uint64_t>(1, (m_max + 1023) / 1024);
  k_status_count<<<g, 1024, 0, s>>>(st, m_ptr, blk0, blk1);
  SKC_LAUNCH_CHECK();
  return status_write(s, st, ids, m_ptr, m_max, blk0, blk1,
                      StatusOut{sky, ext, both, both_st, pos0, n});
}

int launch_status_keep(cudaStream_t s, const uint8_t* st, const uint32_t* m_ptr, uint64_t m_max,
                       uint32_t* blk0, uint32_t* out, uint32_t* n) {
  return status_write(s, st, nullptr, m_ptr, m_max, blk0, nullptr,
                      StatusOut{out, nullptr, nullptr, nullptr, nullptr, n});
}

int launch_scan_counts(cudaStream_t s, const uint32_t* in, uint64_t len, uint64_t* bsum,
                       uint64_t* out, uint32_t T, uint32_t nsub, uint64_t* csr_off) {
  const uint32_t g = (uint32_t)((len + kScanBlock - 1) / kScanBlock);  // len >= 1
  const int scan = g > kSelfScanBlocks;
  if (g > 1) {
    k_scan_partials<<<g, 1024, 0, s>>>(in, len, bsum);
    SKC_LAUNCH_CHECK();
  }
  if (scan) {
    k_scan_single<uint64_t><<<1, 1024, 0, s>>>(bsum, g);
    SKC_LAUNCH_CHECK();
  }
  k_scan_apply<<<g, 1024, 0, s>>>(in, len, bsum, scan, out, T, nsub, csr_off);
  SKC_LAUNCH_CHECK();
  return SKC_OK;
}

uint64_t scan_bsum_entries(uint64_t len) {
  return (len + kScanBlock - 1) / kScanBlock + 1;
}

int launch_block_min(cudaStream_t s, const uint4* cells, const uint32_t* m_ptr,
                     uint64_t m_max, uint4* bmin, uint4* smin, uint4* hmin) {
  k_block_min<<<grid_for(m_max, 256, 152 * 8), 256, 0, s>>>(cells, m_ptr, bmin, smin, hmin);
  SKC_LAUNCH_CHECK();
  return SKC_OK;
}

int launch_csr_gather(cudaStream_t s, const uint32_t* const* srcs,
                      const uint64_t* dst_off, uint32_t ncub, uint32_t* dst) {
  if (ncub == 0) return SKC_OK;
  k_csr_gather<<<ncub, 256, 0, s>>>(srcs, dst_off, dst);
  SKC_LAUNCH_CHECK();
  return SKC_OK;
}

int launch_merge_disjoint(cudaStream_t s, const uint32_t* a, uint32_t na,
                          const uint32_t* b, uint32_t nb, uint32_t* out, uint32_t* n) {
  k_merge_disjoint<<<grid_for((uint64_t)na + nb, 256, 152 * 8), 256, 0, s>>>(a, na, b, nb, out, n);
  SKC_LAUNCH_CHECK();
  return SKC_OK;
}

int launch_set_u32(cudaStream_t s, uint32_t* p, uint32_t v, uint32_t zeros) {
  k_set_u32<<<1, 1, 0, s>>>(p, v, zeros);
  SKC_LAUNCH_CHECK();
  return SKC_OK;
}

// Distribution signature of a dataset from a strided sample of up to
// kSignatureSamples points: out[0] = sample points on the sample's own
// full-space skyline, out[1] = sample points that share an attribute value
// with another sample point, out[2] = sample size. It keys the autotuner's
// table (correlated, independent and anticorrelated data differ by orders
// of magnitude in the first; tie-heavy data shows in the second).
constexpr uint32_t kSignatureSamples = 512;

__global__ void __launch_bounds__(kSignatureSamples) k_sample_signature(
    const float* __restrict__ x, uint64_t n_pad, uint64_t n, int d,
    uint32_t* __restrict__ out) {
  __shared__ float xs[kMaxDims][kSignatureSamples];
  __shared__ uint32_t cnt[2];
  const uint32_t ns = (uint32_t)(n < kSignatureSamples ? n : kSignatureSamples);
  const uint32_t t = threadIdx.x;
  if (t < 2) cnt[t] = 0;
  if (t < ns) {
    const uint64_t id = (uint64_t)t * n / ns;
    for (int k = 0; k < d; ++k) xs[k][t] = x[(uint64_t)k * n_pad + id];
  }
  __syncthreads();
  if (t < ns) {
    bool dominated = false, tied = false;
    for (uint32_t j = 0; j < ns; ++j) {
      if (j == t) continue;
      bool le = true, lt = false;
      for (int k = 0; k < d; ++k) {
        const float a = xs[k][j], b = xs[k][t];
        le &= a <= b;
        lt |= a < b;
        tied |= a == b;
      }
      dominated |= le && lt;
    }
    if (!dominated) atomicAdd(&cnt[0], 1u);
    if (tied) atomicAdd(&cnt[1], 1u);
  }
  __syncthreads();
  if (t == 0) {
    out[0] = cnt[0];
    out[1] = cnt[1];
    out[2] = ns;
  }
}

int launch_sample_signature(cudaStream_t s, const float* x, uint64_t n_pad, uint64_t n, int d,
                            uint32_t* out) {
  if (d < 1 || d > kMaxDims) return set_error(SKC_ERR_INVALID, "unsupported d=%d", d);
  k_sample_signature<<<1, kSignatureSamples, 0, s>>>(x, n_pad, n, d, out);
  SKC_LAUNCH_CHECK();
  return SKC_OK;
}

// Plan helpers (graph-captured launch sequences, api.cu). k_cap_count
// records the true candidate count in stats[slot]; when it is over the plan's
// capacity the device counts become 0 (candidates and skyline points), so
// every later kernel stays inside the buffers; the host sees the overflow and
// re-plans. k_stat_u64 copies one device total.
__global__ void k_cap_count(uint32_t* m_ptr, uint32_t* nsky_ptr, uint32_t cap, uint64_t* stats,
                            int slot) {
  const uint32_t m = *m_ptr;
  stats[slot] = m;
  if (m > cap) {
    *m_ptr = 0;
    *nsky_ptr = 0;
  }
}

__global__ void k_stat_u64(const uint64_t* src, uint64_t* stats, int slot) {
  stats[slot] = *src;
}

int launch_cap_count(cudaStream_t s, uint32_t* m_ptr, uint32_t* nsky_ptr, uint32_t cap,
                     uint64_t* stats, int slot) {
  k_cap_count<<<1, 1, 0, s>>>(m_ptr, nsky_ptr, cap, stats, slot);
  SKC_LAUNCH_CHECK();
  return SKC_OK;
}

int launch_stat_u64(cudaStream_t s, const uint64_t* src, uint64_t* stats, int slot) {
  k_stat_u64<<<1, 1, 0, s>>>(src, stats, slot);
  SKC_LAUNCH_CHECK();
  return SKC_OK;
}

}  // namespace skc
