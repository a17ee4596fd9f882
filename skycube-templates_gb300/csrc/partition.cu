// Median-partition skyline of a point list on one subspace S.
//
// Points are grouped by their median mask over the first B <= 10 attributes
// of S (bit j set when the point is worse than the median on that attribute:
// the top bit of its grid cell). A point q can only dominate p when q's mask
// is a subset of p's: on an attribute where q is above the median and p is
// not, q is strictly worse. This is the partition test of the suite's
// SkyAlign and Hybrid skylines (distribute_pitch_two_level_median,
// src/utilities/kernels.cu:99-125; canskip_partition, src/utilities/
// SubTuple.h:69-73), applied here to whole partitions at once.
//
// Layout. A counting sort groups the list by the lattice-level rank of the
// mask (popcount, then value), so partitions of stronger points come first;
// inside a partition points follow a Gray order of their quartile (then
// finer) cell bits, so any run of them shares its quartile on most
// attributes. The byte-wise minimum cells of every 32-point block, 8-point
// quarter and 4-point half form a box tree over the sorted list.
//
// k_skyline_tree gives a warp up to 32 points of ONE partition (a work item)
// and walks the tree under the submask partitions: a box whose minimum lies
// above p's cell on some attribute holds no q that dominates p. See there.
#include <algorithm>

#include "kernels.cuh"

namespace skc {

static inline unsigned blocks_for(uint64_t items, int threads, int cap) {
  uint64_t b = (items + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > (uint64_t)cap) b = cap;
  return (unsigned)b;
}

// key[i] = rank of the median mask of list entry sub[i] (sub nullptr: i) over the first B
// attributes of S, times 2^sub_bits, plus a sub-key: the cell bits below the
// median bit, quartile bits of S's attributes first, then the next finer
// ones, sub_bits in all, as a Gray code (a point's pattern is ranked by its
// position in the reflected binary sequence, the prefix XOR of its bits, the
// first bit most significant, so consecutive patterns differ in one bit and
// any run of them varies in few). Consecutive points then share their
// quartile on most attributes, which keeps the minimum-cell boxes of the
// blocks tight. A grid of two cells (depth 1) has no such bits: the sub-key is
// the cell sum over S scaled to sub_bits, strong points first (bitmap kernel,
// 300k x 10 uniform 8.95 -> 6.97 ms, with one partition attribute 21.8 -> 17.0).
// Only the partition part matters for correctness.
// With `counts`, also the histogram of the keys (zeroed by the caller); with
// `status`, zeroes the list's statuses.
__global__ void k_mask_keys(const uint4* __restrict__ cells,
                            const uint32_t* __restrict__ sub,
                            const uint32_t* __restrict__ ids,
                            const uint32_t* __restrict__ m_ptr, uint32_t S,
                            int d, int B, int depth, int sub_bits,
                            const uint32_t* __restrict__ rank,
                            uint32_t* __restrict__ keys, uint32_t* __restrict__ counts,
                            uint8_t* __restrict__ status) {
  const uint32_t m = *m_ptr;
  const int sh = depth - 1;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += gridDim.x * blockDim.x) {
    const uint32_t at = sub ? sub[i] : i;
    const uint4 c = cells[ids ? ids[at] : at];
    uint32_t cm = 0, g = 0;
    int j = 0;
    for (int k = 0; k < d && j < B; ++k) {
      if (!(S & (1u << k))) continue;
      const uint32_t cell = (word_of(c, k >> 2) >> (8 * (k & 3))) & 0x7fu;
      cm |= ((cell >> sh) & 1u) << j;
      ++j;
    }
    if (sh == 0) {
      for (int k = 0; k < d; ++k)
        if (S & (1u << k)) g += (word_of(c, k >> 2) >> (8 * (k & 3))) & 0x7fu;
      g = g * ((1u << sub_bits) - 1u) / (uint32_t)__popc(S);
    }
    int t = sub_bits;
    for (int lv = sh - 1; lv >= 0 && t > 0; --lv) {
      for (int k = 0; k < d && t > 0; ++k) {
        if (!(S & (1u << k))) continue;
        --t;
        g |= ((word_of(c, k >> 2) >> (8 * (k & 3) + lv)) & 1u) << t;
      }
    }
    if (sh > 0)
      for (int s2 = 1; s2 < 32; s2 <<= 1) g ^= g >> s2;  // rank in the Gray sequence
    const uint32_t key = (rank[cm] << sub_bits) | g;
    keys[i] = key;
    if (counts) atomicAdd(&counts[key], 1u);
    if (status) status[i] = 0;
  }
}

// Exclusive scan of the bucket counts in two launches: a CTA per 4,096
// buckets adds them up, then every CTA adds the sums before it (at most 64)
// and scans its own 4,096 in place. The former single-CTA scan walked 2^18
// buckets in 64 dependent tiles: 115 us on one GB300; these two: 5.
// boff[b] = offset of bucket b << sub_bits, boff[K] = the total. With m_ptr, a
// list of length 0 is left alone (nothing reads its offsets).
constexpr uint32_t kScanTile = 4096;

__global__ void __launch_bounds__(1024) k_bucket_sums(const uint32_t* __restrict__ counts,
                                                      uint32_t* __restrict__ sums,
                                                      const uint32_t* __restrict__ m_ptr) {
  if (m_ptr && *m_ptr == 0) return;
  __shared__ uint32_t red[32];
  const uint4 v = reinterpret_cast<const uint4*>(counts)[(size_t)blockIdx.x * 1024 + threadIdx.x];
  const uint32_t s = __reduce_add_sync(0xffffffffu, v.x + v.y + v.z + v.w);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    const uint32_t t = __reduce_add_sync(0xffffffffu, red[threadIdx.x]);
    if (threadIdx.x == 0) sums[blockIdx.x] = t;
  }
}

__global__ void __launch_bounds__(1024) k_bucket_scan(uint32_t* __restrict__ counts, uint32_t len,
                                                      const uint32_t* __restrict__ sums,
                                                      int sub_bits, uint32_t* __restrict__ boff,
                                                      const uint32_t* __restrict__ m_ptr) {
  if (m_ptr && *m_ptr == 0) return;
  __shared__ uint32_t wsum[32];
  __shared__ uint32_t s_base;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (wid == 0) {  // the CTAs before this one: at most kMaxSortBuckets / kScanTile = 64
    uint32_t b = 0;
    for (uint32_t j = lane; j < blockIdx.x; j += 32) b += sums[j];
    b = __reduce_add_sync(0xffffffffu, b);
    if (lane == 0) s_base = b;
  }
  const uint32_t base = blockIdx.x * kScanTile + 4 * threadIdx.x;
  uint32_t v[4], local = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    v[j] = base + j < len ? counts[base + j] : 0u;
    local += v[j];
  }
  uint32_t incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  if (lane == 31) wsum[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    const uint32_t w = wsum[lane];
    uint32_t sw = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, sw, o);
      if (lane >= o) sw += u;
    }
    wsum[lane] = sw - w;
  }
  __syncthreads();
  uint32_t run = s_base + wsum[wid] + incl - local;
  const uint32_t smask = (1u << sub_bits) - 1u;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t i = base + j;
    if (i < len) {
      counts[i] = run;
      if ((i & smask) == 0u) boff[i >> sub_bits] = run;
      run += v[j];
      if (i == len - 1) boff[len >> sub_bits] = run;
    }
  }
}

int launch_bucket_scan(cudaStream_t s, uint32_t* counts, uint32_t len, uint32_t* sums,
                       int sub_bits, uint32_t* boff, const uint32_t* m_ptr) {
  const uint32_t g = (len + kScanTile - 1) / kScanTile;
  if (g > 1) {  // then len is a multiple of the tile (both are powers of two)
    k_bucket_sums<<<g, 1024, 0, s>>>(counts, sums, m_ptr);
    SKC_LAUNCH_CHECK();
  }
  k_bucket_scan<<<g, 1024, 0, s>>>(counts, len, sums, sub_bits, boff, m_ptr);
  SKC_LAUNCH_CHECK();
  return SKC_OK;
}

// Places list entry sub[i] (sub nullptr: i) in its bucket (the scanned offsets
// are the cursors): its list position, its point id and its cells restricted
// to S's attributes, attribute t of S in byte t % 4 of word t / 4. The order
// inside a bucket is unspecified; nothing depends on it. The last block is
// filled up with cells of 127.
__global__ void k_part_scatter(const uint32_t* __restrict__ keys,
                               const uint32_t* __restrict__ m_ptr,
                               uint32_t* __restrict__ cursor, const uint4* __restrict__ cells,
                               const uint32_t* __restrict__ sub,
                               const uint32_t* __restrict__ ids, uint32_t S, int d,
                               uint32_t* __restrict__ sorted, uint32_t* __restrict__ sorted_id,
                               uint4* __restrict__ out_cells) {
  const uint32_t m = *m_ptr;
  if (blockIdx.x == 0 && threadIdx.x < 32) {
    const uint32_t i = m + threadIdx.x;
    if (i < ((m + 31) & ~31u))
      out_cells[i] = make_uint4(0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu);
  }
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += gridDim.x * blockDim.x) {
    const uint32_t pos = atomicAdd(&cursor[keys[i]], 1u);
    const uint32_t at = sub ? sub[i] : i;
    const uint32_t id = ids ? ids[at] : at;
    const uint4 c = cells[id];
    uint32_t w[4] = {0, 0, 0, 0};
    int t = 0;
    for (int k = 0; k < d; ++k) {
      if (!(S & (1u << k))) continue;
      const uint32_t cell = (word_of(c, k >> 2) >> (8 * (k & 3))) & 0x7fu;
      const uint32_t sv = cell << (8 * (t & 3));
#pragma unroll
      for (int j = 0; j < 4; ++j)  // constant indexes: w stays in registers
        if ((t >> 2) == j) w[j] |= sv;
      ++t;
    }
    sorted[pos] = at;
    sorted_id[pos] = id;
    out_cells[pos] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// The bitmap kernel's q's in their order: entry i of qpos (positions in
// candidate order) goes to the next place of its bucket with its cells and
// its floats. The last 32-q block is filled up with entries that add
// nothing, so the kernel tests every lane of a block without a bounds check:
// cells 127 and floats +inf. Such a q is worse than p on every attribute
// where p's cell is below 127, and where p's cell is 127 too the float test
// +inf <= p fails (inputs are finite), so LE = LT = {} for every p.
__global__ void k_q_scatter(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ mq_ptr,
                            uint32_t* __restrict__ cursor, const uint32_t* __restrict__ qpos,
                            const uint4* __restrict__ pcells, const float* __restrict__ px,
                            uint64_t pitch, int d, uint4* __restrict__ qcells,
                            float* __restrict__ qx) {
  const uint32_t mq = *mq_ptr;
  if (blockIdx.x == 0 && threadIdx.x < 32) {
    const uint32_t i = mq + threadIdx.x;
    if (i < ((mq + 31) & ~31u)) {
      qcells[i] = make_uint4(0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu);
      for (int k = 0; k < d; ++k) qx[(uint64_t)k * pitch + i] = __int_as_float(0x7f800000);
    }
  }
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < mq; i += gridDim.x * blockDim.x) {
    const uint32_t p = qpos[i];
    const uint32_t pos = atomicAdd(&cursor[keys[i]], 1u);
    qcells[pos] = pcells[p];
    for (int k = 0; k < d; ++k) qx[(uint64_t)k * pitch + pos] = px[(uint64_t)k * pitch + p];
  }
}

__device__ __forceinline__ uint32_t cells_hash(const uint4& c) {
  return c.x * 0x9e3779b1u + c.y * 0x85ebca77u + c.z * 0xc2b2ae3du + c.w * 0x27d4eb2fu;
}

// Whether entry i = 32 b + lane of the sorted list (cells c) repeats an entry
// before it, one of its own block or of the block before it: the same floats on
// S. A repeat needs no place in the boxes: what it dominates its first copy
// dominates as well, and that one lies in the same partition, so a point that
// walks the one walks the other (a copy may itself repeat an earlier one; the
// first is never left out). Equal points share a bucket, so they are
// neighbours, but a bucket may hold several points' copies. The hash only picks
// what to compare: a block without two equal ones is done after one match, and
// only points met twice in the block are looked up in the block before.
// The walk visits every copy otherwise, reading its floats by point id.
// Points of 200k x 6 on 2 / 4 values per attribute (skyline step): 28.2 / 8.5
// ms with all copies in the boxes, 0.20 / 0.84 so.
__device__ __forceinline__ bool repeats_earlier(const uint4* __restrict__ cells, const uint4& c,
                                                uint32_t b, int lane, uint32_t m,
                                                const uint32_t* __restrict__ sorted_id,
                                                const float* __restrict__ x, uint64_t n_pad,
                                                unsigned long long attrs, int na) {
  const uint32_t h = cells_hash(c);
  const uint32_t same = __match_any_sync(0xffffffffu, h);
  int from = __ffs(same) - 1;  // lane of the earlier entry; with `before`, in the block before
  uint32_t heads = __ballot_sync(0xffffffffu, from == lane && (same & (same - 1)));
  if (!heads) return false;  // no hash twice in the block
  const uint32_t i = b * 32 + lane;
  const uint32_t id = i < m ? sorted_id[i] : 0u;
  uint32_t id_before = 0;
  bool before = false;
  if (b > 0) {
    const uint32_t hp = cells_hash(cells[i - 32]);
    id_before = sorted_id[i - 32];
    for (; heads; heads &= heads - 1) {
      const int r = __ffs(heads) - 1;
      const uint32_t hit = __ballot_sync(0xffffffffu, hp == __shfl_sync(0xffffffffu, h, r));
      if (hit && lane == r) {
        from = __ffs(hit) - 1;
        before = true;
      }
    }
  }
  const uint32_t of_own = __shfl_sync(0xffffffffu, id, from);
  const uint32_t of_before = __shfl_sync(0xffffffffu, id_before, from);
  bool equal = i < m && (before || from != lane);
  if (equal) {
    const uint32_t of = before ? of_before : of_own;
#pragma unroll 4
    for (int t = 0; t < na; ++t) {  // all loads in flight: the chain is this kernel's time
      const uint64_t row = ((attrs >> (4 * t)) & 15u) * n_pad;
      equal &= x[row + id] == x[row + of];
    }
  }
  return equal;
}

constexpr uint32_t kMaxSplits = 255;
constexpr uint64_t kMinSliceWork = 512;  // q's: below this a slice is not worth an item

// CTA 0: the work items of the skyline kernel. An item of partition b is 32
// of its points; its cost is the number of points in the partitions under
// b's mask, work[b], the same for all of b's items and spread over orders of
// magnitude. With W = max(total work / target, kMinSliceWork) every item of
// b gets ceil(work[b] / W) slices (at most kMaxSplits); item_off is the
// exclusive prefix of items * slices. The sums over the submask partitions
// are one subset-sum transform over the B mask bits in shared memory (a
// loop over each partition's submask list took 75 us at B = 10; 4 here).
// The other CTAs: byte-wise minimum cells of the 32-q blocks, 8-q quarters
// and 4-q halves of the sorted list (padded to whole blocks), repeats left out.
__global__ void __launch_bounds__(1024) k_boxes_and_plan(
    const uint4* __restrict__ cells, const uint32_t* __restrict__ m_ptr,
    uint4* __restrict__ bmin, uint4* __restrict__ smin, uint4* __restrict__ hmin,
    const uint32_t* __restrict__ boff, const uint32_t* __restrict__ rank,
    const uint32_t* __restrict__ unrank, uint32_t K, int B, uint32_t target,
    uint32_t* __restrict__ splits, uint32_t* __restrict__ item_off,
    const uint32_t* __restrict__ sorted_id, const float* __restrict__ x, uint64_t n_pad,
    unsigned long long attrs, int na) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (*m_ptr == 0) {  // an empty list has no items
    if (blockIdx.x == 0 && threadIdx.x == 0) item_off[K] = 0;
    return;
  }
  if (blockIdx.x > 0) {
    const uint32_t m = *m_ptr, nblk = (m + 31) / 32;
    for (uint32_t b = (blockIdx.x - 1) * 32 + wid; b < nblk; b += (gridDim.x - 1) * 32) {
      uint4 c = cells[(uint64_t)b * 32 + lane];
      if (repeats_earlier(cells, c, b, lane, m, sorted_id, x, n_pad, attrs, na))
        c = make_uint4(0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu);
#pragma unroll
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
    return;
  }
  __shared__ uint32_t s_work[1024];
  __shared__ unsigned long long s_total;
  __shared__ uint32_t wsum[32];
  const uint32_t t = threadIdx.x;
  if (t == 0) s_total = 0;
  if (t < K) {  // by mask
    const uint32_t r = rank[t];
    s_work[t] = boff[r + 1] - boff[r];
  }
  __syncthreads();
  for (int j = 0; j < B; ++j) {
    if (t < K && (t & (1u << j))) s_work[t] += s_work[t ^ (1u << j)];
    __syncthreads();
  }
  unsigned long long work = 0;
  uint32_t chunks = 0;
  if (t < K) {  // by rank
    work = s_work[unrank[t]];
    chunks = (boff[t + 1] - boff[t] + 31) / 32;
  }
  {  // one shared-memory atomic per warp (1,024 of them took 30 us)
    unsigned long long c = work * chunks;
#pragma unroll
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (lane == 0 && c) atomicAdd(&s_total, c);
  }
  __syncthreads();
  unsigned long long W = (s_total + target - 1) / target;
  if (W < kMinSliceWork) W = kMinSliceWork;
  uint32_t sb = 1;
  if (t < K) {
    const unsigned long long q = (work + W - 1) / W;
    sb = (uint32_t)(q < 1 ? 1 : (q > kMaxSplits ? kMaxSplits : q));
    splits[t] = sb;
  }
  const uint32_t c = chunks * sb;
  uint32_t inc = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) wsum[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    const uint32_t v = wsum[lane];
    uint32_t vi = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, vi, o);
      if (lane >= o) vi += u;
    }
    wsum[lane] = vi - v;
  }
  __syncthreads();
  const uint32_t excl = wsum[wid] + inc - c;
  if (t < K) item_off[t] = excl;
  if (t == K - 1) item_off[K] = excl + c;
}

struct TreeArgs {
  const uint32_t* sorted;    // sorted index -> list position
  const uint32_t* sorted_id; // sorted index -> point id
  const uint4* cells;        // compact cells in sorted order, padded to whole blocks
  const uint4* bmin;         // per 32-q block: byte-wise minimum cells
  const uint4* smin;         // per 8-q quarter
  const uint4* hmin;         // per 4-q half
  const float* x;            // attribute-major points
  uint64_t n_pad;
  unsigned long long attrs;  // attribute t of S in bits 4t .. 4t + 3
  const uint32_t* amin;      // per attribute: ordered-uint minimum of a superset of the list
  const uint32_t* boff;      // partition offsets in sorted order [K + 1]
  const uint32_t* unrank;    // rank -> mask
  const uint32_t* sub_off;   // mask -> range in sub_list
  const uint32_t* sub_list;  // ranks of submasks, level order
  uint32_t K;
  const uint32_t* splits;    // slices per work item of partition b [K]
  const uint32_t* item_off;  // first item of partition b [K + 1]
  uint32_t* work;            // work counter, zero
  uint8_t* status;           // list position -> status (zeroed, 4-byte padded)
};

constexpr uint32_t kAll = 0xffffffffu;
constexpr int kTreeWarps = 8;
constexpr uint32_t kBlkQ = 40, kQuarQ = 48, kHalfQ = 40;  // per-warp stacks, entries

// Guard bits where every cell of q is <= p's (pH: p's cells with the guard
// bits set): kGuard when q may dominate p. Bytes beyond NA are 0 in both.
template <int NW>
__device__ __forceinline__ bool cells_le(const uint32_t (&pH)[NW], const uint4& q) {
  uint32_t a = pH[0] - q.x;
  if constexpr (NW > 1) a &= pH[1] - q.y;
  if constexpr (NW > 2) a &= pH[2] - q.z;
  if constexpr (NW > 3) a &= pH[3] - q.w;
  return (a & kGuard) == kGuard;
}

// Skyline status of the list's points on S (NA attributes, all compared): a
// warp takes a work item (32 points of one partition, or a slice of their
// q's) from a device counter, heavy partitions first.
//
//  1. Blocks. The submask partitions' blocks form one list; 32 blocks per
//     step, a lane each, are tested against the GROUP's byte-wise maximum
//     cells. Open ones wait in a stack.
//  2. Quarters. 8 waiting blocks' 32 quarters are tested against the group
//     maximum, a lane each; for each open quarter all 32 points test its
//     minimum with their own cells, a lane each. (point, quarter) pairs wait.
//  3. Halves. 16 waiting pairs' halves, a lane each: (point, half) pairs wait.
//  4. Walk. 8 waiting pairs, a lane per q: cells, and where cells tie the
//     exact floats (read by point id: 1 to 2 q's per point get here on
//     continuous data).
//
// The tests shared by the group and the pair stacks keep the 32 lanes busy
// with tests that are open so far, where the form before (each thread its own
// point against every q of a 32-q tile staged in shared memory) visited every
// tile of the submask partitions: per point of 1M x 10 anticorrelated data
// 561 blocks lie under its mask, 75 of their quarters are open, 34 halves,
// and 2 q's pass the cell test. Bound by instruction issue. Full skyline
// step (sort, boxes, kernel) on one GB300, before -> after: 1M x 10
// anticorrelated 5.62 -> 1.15 ms, 500k x 16 anticorrelated 8.07 -> 1.33,
// 1M x 12 uniform 4.08 -> 0.82.
//
// A point that holds the list's minimum on some attribute of S cannot be
// strictly dominated, so its first dominator settles it (status 1); one that
// holds it on every attribute of S is not dominated at all. On tied data
// nearly every remaining point is of the first kind (values clipped at the
// range's end: 24,600 of 24,600 at 581k x 10 ties), and the walk over all
// its weak dominators was the skyline kernel's whole time there; quantised
// data has thousands of equal points of the second kind. amin may belong to
// a superset of the list: a point of the list equal to it is its minimum.
//
// Slices of one item combine their statuses with a byte-wise atomic OR of
// flags (1 dominated, 2 strictly dominated; 3 reads as strictly dominated).
//
// Four CTAs per SM (64 registers, no spill): the step at 1M x 10 1.15 ms; five
// (48 registers, 50 bytes spilled) 1.26, six 1.23.
template <int NA>
__global__ void __launch_bounds__(32 * kTreeWarps, 4) k_skyline_tree(TreeArgs a) {
  constexpr int NW = (NA + 3) / 4;
  __shared__ uint4 s_p[kTreeWarps][32];
  __shared__ uint32_t s_bq[kTreeWarps][kBlkQ];
  __shared__ uint2 s_sq[kTreeWarps][kQuarQ];  // (box id, point of the group)
  __shared__ uint2 s_hq[kTreeWarps][kHalfQ];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t lt_mask = (1u << lane) - 1u;
  uint4* ps = s_p[wid];
  uint32_t* bq = s_bq[wid];
  uint2* sq = s_sq[wid];
  uint2* hq = s_hq[wid];
  const uint32_t n_items = a.item_off[a.K];
  if (n_items == 0) return;
  const uint32_t m = a.boff[a.K];

  for (;;) {
    uint32_t it = 0;
    if (lane == 0) it = atomicAdd(a.work, 1u);
    it = __shfl_sync(kAll, it, 0);
    if (it >= n_items) return;
    it = n_items - 1 - it;  // the partitions with the most work first
    uint32_t b = 0;
    {
      uint32_t hi = a.K;
      while (hi - b > 1) {
        const uint32_t mid = (b + hi) >> 1;
        if (a.item_off[mid] <= it) b = mid; else hi = mid;
      }
    }
    const uint32_t splits = a.splits[b];
    const uint32_t local = it - a.item_off[b];
    const uint32_t chunk = local / splits, sp = local - chunk * splits;
    const uint32_t i = a.boff[b] + chunk * 32 + lane;
    const bool valid = i < a.boff[b + 1];
    uint4 pc = make_uint4(0, 0, 0, 0);
    uint32_t pos = 0, id = 0;
    if (valid) {
      pc = a.cells[i];
      pos = a.sorted[i];
      id = a.sorted_id[i];
    }
    uint32_t pH[NW], gH[NW];  // own cells and the group's maximum, with guard bits
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      uint32_t g = word_of(pc, w);
      pH[w] = g | kGuard;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) g = __vmaxu4(g, __shfl_xor_sync(kAll, g, o));
      gH[w] = g | kGuard;
    }
    __syncwarp();  // the previous item's readers of ps are done
    ps[lane] = pc;
    // Attributes on which the point holds the list's minimum (its cell is then 0).
    int n_min = 0;
    if (valid) {
#pragma unroll
      for (int t = 0; t < NA; ++t) {
        if (((word_of(pc, t >> 2) >> (8 * (t & 3))) & 0x7fu) == 0u) {
          const uint32_t k = (uint32_t)(a.attrs >> (4 * t)) & 15u;
          n_min += ordered_u32(a.x[(uint64_t)k * a.n_pad + id]) == a.amin[k];
        }
      }
    }
    const uint32_t no_strict = __ballot_sync(kAll, n_min > 0);
    uint32_t dom = 0, strict = 0;  // per point of the group
    uint32_t done = __ballot_sync(kAll, !valid || n_min == NA);
    if (splits > 1) {  // settled by another slice already?
      const uint32_t st = valid ? *(volatile const uint8_t*)(a.status + pos) : 0u;
      done |= __ballot_sync(kAll, st >= 2u || (st && n_min));
    }
    __syncwarp();

    uint32_t bq_n = 0, sq_n = 0, hq_n = 0;
    // Walk step over the top c (<= 8) waiting (point, half) pairs.
    auto walk = [&](uint32_t c) {
      const uint32_t slot = lane >> 2;
      const uint2 e = hq[hq_n - c + min(slot, c - 1)];
      hq_n -= c;
      const uint32_t pi = e.y;
      const uint32_t q = e.x * 4 + (lane & 3);
      bool live = slot < c && !((done >> pi) & 1u) && q < m;
      uint32_t Z = 0;  // equal cells (attribute bits)
      bool any_lt = false, all_lt = true;
      const uint4 q4 = a.cells[q];  // the cells are padded to whole blocks
      const uint4 p4 = ps[pi];
      uint32_t wH[NW];
#pragma unroll
      for (int w = 0; w < NW; ++w) wH[w] = word_of(p4, w) | kGuard;
      live = live && cells_le<NW>(wH, q4);
      const uint32_t pid = __shfl_sync(kAll, id, pi);
      if (live) {
#pragma unroll
        for (int w = 0; w < NW; ++w)
          Z |= pack_guards(ge_bytes(word_of(q4, w) | kGuard, word_of(p4, w))) << (4 * w);
        Z &= (1u << NA) - 1u;
        any_lt = Z != (1u << NA) - 1u;
        if (Z) {
          const uint32_t qid = a.sorted_id[q];
          for (uint32_t z = Z; z && live; z &= z - 1) {
            const int t = __ffs(z) - 1;
            const uint64_t row = ((a.attrs >> (4 * t)) & 15u) * a.n_pad;
            const float qv = a.x[row + qid], pv = a.x[row + pid];
            live = qv <= pv;
            if (qv < pv) any_lt = true; else all_lt = false;
          }
        }
      }
      const bool d = live && any_lt;
      if (__any_sync(kAll, d)) {
        dom |= __reduce_or_sync(kAll, d ? 1u << pi : 0u);
        strict |= __reduce_or_sync(kAll, (d && all_lt) ? 1u << pi : 0u);
        done |= strict | (dom & no_strict);
      }
      __syncwarp();  // read before a later push overwrites the entries
    };
    // Half step over the top c (<= 16) waiting (point, quarter) pairs.
    auto half_step = [&](uint32_t c) {
      const uint32_t slot = lane >> 1;
      const uint2 e = sq[sq_n - c + min(slot, c - 1)];
      sq_n -= c;
      const uint32_t pi = e.y;
      const uint32_t hid = e.x * 2 + (lane & 1);
      const uint4 hm = a.hmin[hid];
      const uint4 p4 = ps[pi];
      uint32_t wH[NW];
#pragma unroll
      for (int w = 0; w < NW; ++w) wH[w] = word_of(p4, w) | kGuard;
      const bool open = slot < c && !((done >> pi) & 1u) && cells_le<NW>(wH, hm);
      const uint32_t om = __ballot_sync(kAll, open);
      if (open) hq[hq_n + __popc(om & lt_mask)] = make_uint2(hid, pi);
      hq_n += __popc(om);
      __syncwarp();
      while (hq_n >= 8) walk(8);
    };
    // Quarter step over the top c (<= 8) waiting blocks.
    auto quarter_step = [&](uint32_t c) {
      const uint32_t slot = lane >> 2;
      const uint32_t sid = bq[bq_n - c + min(slot, c - 1)] * 4 + (lane & 3);
      bq_n -= c;
      const uint4 sm = a.smin[sid];
      uint32_t qm = __ballot_sync(kAll, slot < c && cells_le<NW>(gH, sm));
      __syncwarp();
      for (; qm; qm &= qm - 1) {
        const int src = __ffs(qm) - 1;
        uint4 q4;
        q4.x = __shfl_sync(kAll, sm.x, src);
        if constexpr (NW > 1) q4.y = __shfl_sync(kAll, sm.y, src);
        if constexpr (NW > 2) q4.z = __shfl_sync(kAll, sm.z, src);
        if constexpr (NW > 3) q4.w = __shfl_sync(kAll, sm.w, src);
        const bool open = !((done >> lane) & 1u) && cells_le<NW>(pH, q4);
        const uint32_t om = __ballot_sync(kAll, open);
        if (!om) continue;
        const uint32_t s = __shfl_sync(kAll, sid, src);
        if (open) sq[sq_n + __popc(om & lt_mask)] = make_uint2(s, (uint32_t)lane);
        sq_n += __popc(om);
        __syncwarp();
        while (sq_n >= 16) half_step(16);
      }
    };

    const uint32_t mb = a.unrank[b];
    const uint32_t s0 = a.sub_off[mb], s1 = a.sub_off[mb + 1];
    // This slice's range [s_lo, s_hi) of the concatenated submask partitions.
    uint32_t s_lo = 0, s_hi = kAll;
    if (splits > 1) {
      uint32_t part = 0;
      for (uint32_t si = s0 + lane; si < s1; si += 32) {
        const uint32_t qb = a.sub_list[si];
        part += a.boff[qb + 1] - a.boff[qb];
      }
      const uint64_t total = __reduce_add_sync(kAll, part);
      s_lo = (uint32_t)(total * sp / splits);
      s_hi = (uint32_t)(total * (sp + 1) / splits);
    }
    uint32_t acc = 0;       // q's of the partitions before this step's
    uint32_t next_blk = 0;  // blocks below this one were listed already
    // Every slice but the first starts with the list's first block (the
    // strongest points; partition 0 lies under every mask): on correlated
    // and tied data it settles the group, which would else walk its slice to
    // the end for points that the first slice settles at once.
    bool probe = sp > 0;
    for (uint32_t si = s0;;) {
      uint32_t beg = 0, end = 0;
      if (probe) {
        if (lane == 0) end = min(32u, m);
      } else {
        if (si + lane < s1) {
          const uint32_t qb = a.sub_list[si + lane];
          beg = a.boff[qb];
          end = a.boff[qb + 1];
        }
        si += 32;
        if (splits > 1) {  // cut to the slice
          const uint32_t sz = end - beg;
          uint32_t incl = sz;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kAll, incl, o);
            if (lane >= o) incl += y;
          }
          const uint32_t start = acc + incl - sz;
          const uint32_t c0 = max(s_lo, start), c1 = min(s_hi, start + sz);
          acc += __shfl_sync(kAll, incl, 31);
          end = c0 < c1 ? beg + (c1 - start) : 0u;
          beg = c0 < c1 ? beg + (c0 - start) : 0u;
        }
      }
      // The partitions' blocks laid end to end; a block shared with the
      // partition before is listed once (ranks, and so offsets, ascend).
      const bool sel = beg < end;
      const uint32_t be = (end + 31) / 32;
      const uint32_t parts = __ballot_sync(kAll, sel);
      if (parts) {
        const uint32_t lower = parts & lt_mask;
        const uint32_t prev_be = __shfl_sync(kAll, be, lower ? 31 - __clz(lower) : 0);
        const uint32_t bf = max(beg / 32, lower ? prev_be : next_blk);
        const uint32_t cnt = (sel && be > bf) ? be - bf : 0u;
        uint32_t incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(kAll, incl, o);
          if (lane >= o) incl += y;
        }
        const uint32_t total = __shfl_sync(kAll, incl, 31);
        if (!probe) next_blk = max(next_blk, __shfl_sync(kAll, be, 31 - __clz(parts)));
        const uint32_t base = bf - (incl - cnt);  // list entry g of this lane is block g + base
        for (uint32_t t0 = 0; t0 < total && done != kAll; t0 += 32) {
          const uint32_t g = t0 + lane;
          int j = 0;  // owner of list entry g: the first lane whose inclusive sum is > g
#pragma unroll
          for (int step = 16; step; step >>= 1) {
            const uint32_t v = __shfl_sync(kAll, incl, j + step - 1);
            if (v <= g) j += step;
          }
          const uint32_t kb = g + __shfl_sync(kAll, base, j);
          bool open = false;
          if (g < total) open = cells_le<NW>(gH, a.bmin[kb]);
          const uint32_t om = __ballot_sync(kAll, open);
          if (open) bq[bq_n + __popc(om & lt_mask)] = kb;
          bq_n += __popc(om);
          __syncwarp();
          while (bq_n >= 8) quarter_step(8);
        }
      }
      const bool last = !probe && (si >= s1 || acc >= s_hi);
      if ((probe || last) && done != kAll) {  // what still waits: one short step of each kind
        if (bq_n) quarter_step(bq_n);
        if (sq_n) half_step(sq_n);
        if (hq_n) walk(hq_n);
      }
      if (last || done == kAll) break;
      probe = false;
    }
    const uint32_t st = ((dom >> lane) & 1u) | (((strict >> lane) & 1u) << 1);
    if (valid && st) {
      if (splits == 1)
        a.status[pos] = (uint8_t)(st & 2u ? 2u : 1u);
      else
        atomicOr(reinterpret_cast<unsigned int*>(a.status + (pos & ~3u)), st << (8 * (pos & 3u)));
    }
  }
}

int launch_q_scatter(cudaStream_t s, const uint32_t* keys, const uint32_t* mq_ptr, uint64_t m_max,
                     uint32_t* cursor, const uint32_t* qpos, const uint4* pcells, const float* px,
                     uint64_t pitch, int d, uint4* qcells, float* qx) {
  k_q_scatter<<<blocks_for(m_max, 256, 152 * 8), 256, 0, s>>>(keys, mq_ptr, cursor, qpos, pcells,
                                                               px, pitch, d, qcells, qx);
  SKC_LAUNCH_CHECK();
  return SKC_OK;
}

int launch_mask_keys(cudaStream_t s, const uint4* cells, const uint32_t* ids,
                     const uint32_t* m_ptr, uint64_t m_max, uint32_t S, int d,
                     int B, int depth, int sub_bits, const uint32_t* rank,
                     uint32_t* keys, uint32_t* counts) {
  k_mask_keys<<<blocks_for(m_max, 256, 152 * 8), 256, 0, s>>>(cells, nullptr, ids, m_ptr, S, d, B,
                                                               depth, sub_bits, rank, keys, counts,
                                                               nullptr);
  SKC_LAUNCH_CHECK();
  return SKC_OK;
}

// Sub-key bits of a sort of up to m_max entries in K partitions: as many as
// `most`, while the buckets stay within kMaxSortBuckets and about two per
// entry (more only cost the scan).
int sort_sub_bits(uint64_t m_max, uint32_t K, int most) {
  int b = 0;
  while (b < most && ((uint64_t)K << (b + 1)) <= kMaxSortBuckets &&
         ((uint64_t)K << b) < m_max)
    ++b;
  return b;
}

template <int NA>
static int launch_tree(cudaStream_t s, int num_sms, const TreeArgs& a) {
  static_assert(NA >= 1 && NA <= kMaxDims, "attributes");
  int per_sm = 0;
  SKC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_skyline_tree<NA>,
                                                         32 * kTreeWarps, 0));
  k_skyline_tree<NA><<<std::max(1, per_sm) * num_sms, 32 * kTreeWarps, 0, s>>>(a);
  SKC_LAUNCH_CHECK();
  return SKC_OK;
}

int launch_partition_skyline(cudaStream_t s, int num_sms, int d, const LevelTables& T,
                             const PartitionSkylineArgs& args, const PartScratch& ps) {
  PartitionSkylineArgs a = args;
  if (a.sub) {  // a prefilter ran: few points may be left
    SKC_TRY(launch_small_status(s, d, args, ps.rest));
    a.m_ptr = ps.rest;
  }
  const uint32_t K = 1u << T.B;
  const int na = __builtin_popcount(a.S);
  const int sub_bits = sort_sub_bits(a.m_max, K, std::min(kMaxSubBits, na * (kMaxDepth - 1)));
  const uint32_t KB = K << sub_bits;
  uint32_t* work = ps.fine + KB;  // the skyline kernel's work counter, behind the buckets
  SKC_CUDA(cudaMemsetAsync(ps.fine, 0, (KB + 1) * sizeof(uint32_t), s));
  const unsigned grid = blocks_for(a.m_max, 256, 152 * 8);
  k_mask_keys<<<grid, 256, 0, s>>>(a.cells, a.sub, a.ids, a.m_ptr, a.S, d, T.B, kMaxDepth, sub_bits,
                                   T.rank, ps.keys, ps.fine, a.sub ? nullptr : a.status);
  SKC_LAUNCH_CHECK();
  SKC_TRY(launch_bucket_scan(s, ps.fine, KB, ps.sums, sub_bits, ps.counts, a.m_ptr));
  k_part_scatter<<<grid, 256, 0, s>>>(ps.keys, a.m_ptr, ps.fine, a.cells, a.sub, a.ids, a.S, d,
                                      ps.sorted, ps.sorted_id, ps.ccells);
  SKC_LAUNCH_CHECK();
  // Items: enough slices that a warp takes several and the last ones are
  // short (kItemsPerSm per SM, 32 warps resident).
  unsigned long long attrs = 0;
  for (int k = 0, t = 0; k < d; ++k)
    if (a.S & (1u << k)) attrs |= (unsigned long long)k << (4 * t++);
  k_boxes_and_plan<<<1 + blocks_for(a.m_max, 1024, 152 * 2), 1024, 0, s>>>(
      ps.ccells, a.m_ptr, ps.bmin, ps.smin, ps.hmin, ps.counts, T.rank, T.unrank, K, T.B,
      (uint32_t)num_sms * kItemsPerSm, ps.splits, ps.item_off, ps.sorted_id, a.x, a.n_pad, attrs,
      na);
  SKC_LAUNCH_CHECK();
  const TreeArgs k{ps.sorted, ps.sorted_id, ps.ccells, ps.bmin, ps.smin, ps.hmin, a.x, a.n_pad, attrs,
                   a.amin, ps.counts, T.unrank, T.sub_off, T.sub_list, K, ps.splits, ps.item_off,
                   work, a.status};
#define SKC_TREE_CASE(N) \
  case N: return launch_tree<N>(s, num_sms, k);
  switch (na) {
    SKC_TREE_CASE(1) SKC_TREE_CASE(2) SKC_TREE_CASE(3) SKC_TREE_CASE(4)
    SKC_TREE_CASE(5) SKC_TREE_CASE(6) SKC_TREE_CASE(7) SKC_TREE_CASE(8)
    SKC_TREE_CASE(9) SKC_TREE_CASE(10) SKC_TREE_CASE(11) SKC_TREE_CASE(12)
    SKC_TREE_CASE(13) SKC_TREE_CASE(14) SKC_TREE_CASE(15) SKC_TREE_CASE(16)
    default:
      return set_error(SKC_ERR_INVALID, "subspace with %d attributes", na);
  }
#undef SKC_TREE_CASE
}

}  // namespace skc
