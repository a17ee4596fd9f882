// Launch helpers of the skycube engine's kernels (internal).
#pragma once

#include "common.cuh"

namespace skc {

constexpr int kMaxDims = 16;
constexpr int kMaxPivots = 127;  // 2^kMaxDepth - 1

// Scratch of the counting sort by bucket (all device pointers).
struct BucketScratch {
  float* f = nullptr;        // [m_max] scores
  uint32_t* keys = nullptr;  // [m_max]
  uint32_t* counts = nullptr;  // [K + 1]
  uint32_t* cursor = nullptr;  // [K + 1]
  uint32_t* minmax = nullptr;  // [2]
};

// prep.cu
int launch_rows_to_soa(cudaStream_t s, const float* rows, uint64_t n, int d,
                       uint64_t n_pad, float* x, uint32_t* bad);
int launch_bucket_order(cudaStream_t s, const float* x, uint64_t n_pad, int d,
                        const uint32_t* ids, const uint32_t* m_ptr,
                        uint64_t m_max, uint32_t S, uint32_t K,
                        const BucketScratch& b, uint32_t* sorted, uint32_t* hi);
int launch_counting_sort(cudaStream_t s, const uint32_t* keys,
                         const uint32_t* m_ptr, uint64_t m_max, uint32_t K,
                         const BucketScratch& b, uint32_t* sorted, uint32_t* hi);
constexpr uint32_t kSumBins = 2048;  // cell sums: 127 * 16 < 2048
int launch_pivots_cells(cudaStream_t s, const float* x, uint64_t n_pad, int d,
                        const uint32_t* ids, const uint32_t* m_ptr,
                        uint64_t m_max, int depth, float* pivots, uint4* cells,
                        uint32_t* amin = nullptr, uint32_t* hist = nullptr,
                        float* xout = nullptr, uint64_t out_pad = 0, int low = 0);
// Entries of status 0 / 1 into sky / ext (ids in list order), n[0] / n[1]
// their counts, n[2] the sum; with `both`, also their union in list order,
// its entries' flags (0 for status 0, else 2) and the union positions of the
// status-0 entries. blk0, blk1: [m_max / 1024 + 2].
int launch_status_split(cudaStream_t s, const uint8_t* st, const uint32_t* ids,
                        const uint32_t* m_ptr, uint64_t m_max, uint32_t* blk0, uint32_t* blk1,
                        uint32_t* sky, uint32_t* ext, uint32_t* n, uint32_t* both = nullptr,
                        uint8_t* both_st = nullptr, uint32_t* pos0 = nullptr);
// List positions of status 0 into out, *n their count;
// blk0[b] holds the count over i in [1024 b, 1024 b + 1024) (zero past the list).
int launch_status_keep(cudaStream_t s, const uint8_t* st, const uint32_t* m_ptr, uint64_t m_max,
                       uint32_t* blk0, uint32_t* out, uint32_t* n);
// Exclusive scan of in[0 .. len) into out[0 .. len]; csr_off[c] = out[c * T]
// for c <= nsub (nsub * T <= len).
int launch_scan_counts(cudaStream_t s, const uint32_t* in, uint64_t len, uint64_t* bsum,
                       uint64_t* out, uint32_t T, uint32_t nsub, uint64_t* csr_off);
uint64_t scan_bsum_entries(uint64_t len);
int launch_block_min(cudaStream_t s, const uint4* cells, const uint32_t* m_ptr,
                     uint64_t m_max, uint4* bmin, uint4* smin, uint4* hmin);
int launch_csr_gather(cudaStream_t s, const uint32_t* const* srcs,
                      const uint64_t* dst_off, uint32_t ncub, uint32_t* dst);
// p[0] = v, p[1 .. zeros] = 0.
int launch_set_u32(cudaStream_t s, uint32_t* p, uint32_t v, uint32_t zeros = 0);
// Also n[0] = na + nb, n[1] = 0.
int launch_merge_disjoint(cudaStream_t s, const uint32_t* a, uint32_t na,
                          const uint32_t* b, uint32_t nb, uint32_t* out, uint32_t* n);
int launch_sample_signature(cudaStream_t s, const float* x, uint64_t n_pad, uint64_t n, int d,
                            uint32_t* out);
int launch_cap_count(cudaStream_t s, uint32_t* m_ptr, uint32_t* nsky_ptr, uint32_t cap,
                     uint64_t* stats, int slot);
int launch_stat_u64(cudaStream_t s, const uint64_t* src, uint64_t* stats, int slot);

// skyline.cu: status of every list entry on subspace S (0 skyline,
// 1 extended skyline, 2 strictly dominated).
struct SkylineArgs {
  const uint32_t* sorted;  // sorted index -> list position (bucket order)
  const uint32_t* hi;      // sorted index -> end of its bucket
  const uint32_t* ids;     // list position -> point id (nullptr: identity)
  const uint4* cells;      // point id -> grid cells
  const float* x;          // attribute-major points
  uint64_t n_pad;
  const uint32_t* m_ptr;   // list length (device)
  uint64_t m_max;          // upper bound of the list length (host)
  uint32_t S;              // subspace mask
  uint8_t* status;         // list position -> status
};
int launch_skyline(cudaStream_t s, int d, const SkylineArgs& a);

// partition.cu: median-partition skyline (status as above).
// Lattice-level tables over B-bit masks (B <= 10): rank (popcount, then
// value), its inverse, and for every mask the ranks of its submasks in
// level order.
constexpr int kMaxPartitionDims = 10;
constexpr uint64_t kMaxSortBuckets = 1u << 18;  // partition x strength buckets
struct LevelTables {
  int B = 0;
  const uint32_t* rank = nullptr;      // [2^B]
  const uint32_t* unrank = nullptr;    // [2^B]
  const uint32_t* sub_off = nullptr;   // [2^B + 1]
  const uint32_t* sub_list = nullptr;  // [3^B]
};
struct PartScratch {
  uint32_t* keys;      // [m_max]
  uint32_t* sorted;    // [m_max] list positions in partition order
  uint32_t* sorted_id; // [m_max] their point ids
  uint4* ccells;       // [m_max, rounded up to 32] compact cells in partition order
  uint4* bmin;         // [m_max / 32 + 1] minimum cells per 32-point block,
  uint4* smin;         // [(m_max / 32 + 1) * 4] 8-point quarter
  uint4* hmin;         // [(m_max / 32 + 1) * 8] and 4-point half
  uint32_t* counts;    // [2^B + 1] partition offsets after the sort
  uint32_t* fine;      // [kMaxSortBuckets + 1] counting-sort offsets, work counter
  uint32_t* sums;      // [kMaxScanSums]
  uint32_t* splits;    // [2^B]
  uint32_t* rest;      // points left by launch_small_status
  uint32_t* item_off;  // [2^B + 1]
};
struct PartitionSkylineArgs {
  const uint32_t* sub;  // the list's positions to settle, ascending (the prefilter's
                        // survivors, whose statuses are 0 already); nullptr: all
  const uint32_t* ids;  // list position -> point id (nullptr: identity)
  const uint4* cells;   // point id -> grid cells, kMaxDepth deep
  const float* x;
  uint64_t n_pad;
  const uint32_t* m_ptr;  // entries of `sub`, or of the list
  uint64_t m_max;
  uint32_t S;
  uint8_t* status;      // list position -> status; rounded up to 4 bytes
  const uint32_t* amin; // [d] ordered-uint minima over a superset of the list
};
constexpr uint32_t kMaxScanSums = 64;  // kMaxSortBuckets / 4096
// Skyline kernel: work items per SM the plan aims at (32 warps are resident).
constexpr uint32_t kItemsPerSm = 256;
constexpr int kMaxSubBits = 15;  // sub-key bits inside a partition
int sort_sub_bits(uint64_t m_max, uint32_t K, int most);
int launch_mask_keys(cudaStream_t s, const uint4* cells, const uint32_t* ids,
                     const uint32_t* m_ptr, uint64_t m_max, uint32_t S, int d,
                     int B, int depth, int sub_bits, const uint32_t* rank,
                     uint32_t* keys, uint32_t* counts);
// Exclusive scan of counts[0 .. len) in place (len a power of two, at most
// kMaxSortBuckets); boff[b] = offset of bucket b << sub_bits, boff[len >>
// sub_bits] = the total.
int launch_bucket_scan(cudaStream_t s, uint32_t* counts, uint32_t len, uint32_t* sums,
                       int sub_bits, uint32_t* boff, const uint32_t* m_ptr = nullptr);
int launch_q_scatter(cudaStream_t s, const uint32_t* keys, const uint32_t* mq_ptr, uint64_t m_max,
                     uint32_t* cursor, const uint32_t* qpos, const uint4* pcells, const float* px,
                     uint64_t pitch, int d, uint4* qcells, float* qx);
int launch_partition_skyline(cudaStream_t s, int num_sms, int d, const LevelTables& T,
                             const PartitionSkylineArgs& a, const PartScratch& ps);

// small.cu: skyline of a list of at most kSmallList points on subspace S,
// compaction included, in one launch. masks: [2 * kSmallList / 32], ticket: 0.
constexpr uint32_t kSmallList = 6144;
struct SplitOut {
  uint32_t* sky;      // skyline ids, list order
  uint32_t* ext;      // extended skyline ids (nullptr: behind the skyline's in `sky`)
  uint32_t* both;     // their union in list order, or nullptr
  uint8_t* both_st;   // per entry of `both`: 0 skyline, else 2 (nullptr: neither it nor pos0)
  uint32_t* pos0;     // per skyline id: its position in `both`
  uint32_t* n;        // [3] counts: sky, ext, both
};
int launch_small_skyline(cudaStream_t s, const float* x, uint64_t n_pad, int d,
                         const uint32_t* ids, const uint32_t* m_ptr, uint64_t m_max, uint32_t S,
                         uint32_t* masks, uint32_t* ticket, const SplitOut& out);
// The same for several lists and subspaces with one attribute count (below
// 16) in one launch; fills in `attrs` and `first`.
constexpr uint32_t kSmallJobs = 64;
struct SmallJob {
  const uint32_t* ids;
  uint32_t* lists;  // [m] skyline ids, then extended skyline ids
  uint32_t* both;   // [m] their union in list order, or nullptr
  uint32_t* n;      // [3] counts: sky, ext, both
  uint32_t m, S;    // list length (1 to kSmallList), subspace
  unsigned long long attrs;
  uint32_t first;   // first CTA
};
int launch_small_batch(cudaStream_t s, const float* x, uint64_t n_pad, int d, SmallJob* jobs,
                       uint32_t nj, uint32_t* masks, uint32_t* tickets);
// Statuses of a prefilter's open points by all pairs when there are few enough
// of them (small.cu); *rest = those left to the partition pipeline (all or 0).
int launch_small_status(cudaStream_t s, int d, const PartitionSkylineArgs& a, uint32_t* rest);
// The bitmap kernel's inputs for few candidates in one launch (one partition).
constexpr uint32_t kSmallCandidates = 1024;
int launch_small_prep(cudaStream_t s, int d, const float* x, uint64_t n_pad, const uint32_t* cand,
                      const uint8_t* cand_st, const uint32_t* m_ptr, uint64_t m_max, int depth,
                      uint64_t pitch, uint4* cells, float* px, uint4* qcells, float* qx,
                      uint4* bmin, uint4* smin, uint4* hmin, uint32_t* boff, uint32_t* work);
int launch_single_offsets(cudaStream_t s, const uint32_t* n, uint32_t S, uint32_t nsub,
                          uint64_t* sky_off, uint64_t* ext_off);

// prefilter.cu: pruner prefilter of a list on subspace S. Every list position
// gets a status: 2 strictly dominated by a pruner, 1 dominated by one and
// never strictly (it holds an attribute's minimum), 0 open. The open ones
// come out as list positions, ascending.
constexpr int kMaxPruners = 1024;
struct PrefilterScratch {
  uint32_t* hist;      // [kSumBins + 8] cell sums over S (see hist_ready), then counters
  uint32_t* pr_ids;    // [K]
  uint32_t* pr_key;    // [K]
  uint4* pr_cells;     // [K] pruner cells, rank order
  float* pr_x;         // [d * K] pruner floats, rank order
  unsigned long long* tab;  // [prefilter_table_bytes(d, K)] pruner tables
  uint32_t* blk;       // [m_max / 1024 + 2] kept entries per 1024
};
struct PrefilterArgs {
  const uint4* cells;    // point id -> grid cells
  const float* x;        // attribute-major points, pitch n_pad
  uint64_t n_pad;
  const uint32_t* ids;   // list position -> point id (nullptr: identity)
  const uint32_t* m_ptr;
  uint64_t m_max;
  uint32_t S;
  uint32_t K;            // pruners, 1 .. kMaxPruners
  const uint32_t* amin;  // [d] ordered-uint minima over a superset of the list
  PrefilterScratch ps;
  uint8_t* status;       // [m_max] by list position
  bool hist_ready;       // ps.hist already holds the list's cell sums, its counters are 0
};
int launch_prefilter(cudaStream_t s, int d, int num_sms, const PrefilterArgs& a,
                     uint32_t* out, uint32_t* out_count);
size_t prefilter_table_bytes(int d, uint32_t K);

// mdmc.cu: per-point dominated-subspace bitmaps over the candidate set.
struct BitmapArgs {
  const uint4* pcells;   // candidate order
  const float* px;       // candidate order, attribute-major, pitch p_pad
  uint64_t p_pad;
  const uint4* qcells;   // q order (level-sorted), padded to whole 32-q blocks
  const float* qx;       // q order, attribute-major, pitch p_pad
  const uint4* bmin;     // per block of 32 q's: byte-wise minimum cells
  const uint4* smin;     // the same per 8-q sub-block (4 per block)
  const uint4* hmin;     // the same per 4-q half of a sub-block (8 per block)
  const uint32_t* boff;  // q partitions: offsets in q order [K + 1]
  const uint32_t* unrank;  // partition rank -> median mask over B attributes
  uint32_t K;
  int B;
  int depth;
  const uint32_t* m_ptr;   // candidates (p's)
  uint32_t* work;        // work counter, must hold p_begin
  uint32_t chunk;        // candidates per work-counter grab (0: 1)
  uint32_t p_end;        // stop at min(m, p_end)
  uint32_t* out_dom;     // [m][words] dominated bitmaps
  uint32_t* out_ext;     // [m][words] extended-skyline bitmaps, or nullptr
  int grid_blocks;       // persistent grid (0: from occupancy)
  uint32_t* tie_slab;    // global tie maps (bitmap_tie_slab_words), or nullptr
  // Capped skycubes: only the bits of subspaces with at most `cap`
  // attributes and of the full space are exact (1 <= cap <= d - 2; 0: all
  // bits). The full-space bits then come from full_dom (per candidate,
  // nonzero when it is dominated on the full space).
  int cap = 0;
  const uint8_t* full_dom = nullptr;
};
int launch_bitmaps(cudaStream_t s, int d, int num_sms, const BitmapArgs& a);
int bitmap_tie_slab_words(int d, int num_sms, uint64_t* words);

struct CompactArgs {
  const uint32_t* bits;  // [m][words]
  uint32_t words;
  const uint32_t* m_ptr;
  uint64_t m_max;
  int count_set;         // 0: rows with the bit CLEAR (skyline); 1: SET
  uint32_t nsub;         // 2^d
  int max_d;
  const uint32_t* cand;  // row -> point id
  uint32_t* counts;      // [32*words * tiles]
  uint64_t* offs;        // [32*words * tiles + 1]
  uint64_t* bsum;        // scan scratch
  uint64_t* csr_off;     // [nsub + 1] output offsets per cuboid
  uint32_t* out;         // ids (sized by the caller after the count pass)
  uint64_t out_cap;      // entries of `out`; ids past it are not written
};
uint32_t compact_tiles(uint64_t m_max, uint32_t words);
int launch_bits_count(cudaStream_t s, const CompactArgs& a);
int launch_bits_write(cudaStream_t s, const CompactArgs& a);

// levels.cu: capped skycubes by lattice level (cuboids of at most
// kLvMaxDims attributes), one CTA per cuboid for the sort-filter skyline.
constexpr int kLvMaxDims = 4;
constexpr uint32_t kLvPruners = 32;    // per cuboid, from a strided sample
constexpr uint32_t kLvSample = 1024;   // sampled list entries
constexpr uint32_t kLvChunk = 8192;    // list entries per filter item (staged in shared memory)
constexpr uint32_t kLvThreads = 1024;  // sort-filter CTA, one batch per pass
constexpr uint32_t kLvWin = 2048;      // skyline points per cuboid
constexpr uint32_t kLvExt = 4096;      // extended-skyline points per cuboid
constexpr uint32_t kLvSlot = kLvWin + kLvExt;  // output ids per cuboid
constexpr uint32_t kLvSortCap = 8192;  // power of two >= kLvSlot
constexpr uint32_t kLvKeyBins = 127 * kLvMaxDims + 1;  // cell sums
// One dataset of a lattice launch.
struct LtJob {
  const float* x;            // attribute-major points, pitch n_pad
  uint64_t n_pad;
  const uint4* cells;        // point id -> cells on the candidates' quantile grid
  const uint32_t* cand;      // full-space skyline + extended skyline ids
  uint32_t n_cand;
  const uint8_t* cand_cells; // the candidates' cells: [d][cell_pitch] bytes in candidate order
  uint64_t cell_pitch;       // a multiple of 16
  const uint32_t* cub_index; // [2^d] mask -> cuboid table index (0xffffffff: none)
  int d, max_d;
};
// A lattice launch (levels.cu, k_lattice): every wanted cuboid of every job
// (cuboid table index c) from a device work queue in lattice-level order.
struct LtArgs {
  const LtJob* jobs;
  const uint32_t* c_mask;    // [ncub]
  const uint32_t* c_job;     // [ncub]
  const uint32_t* c_scr;     // [ncub] scratch index in the cuboid's group
  const uint32_t** c_list;   // [ncub] candidate list (set by phase P)
  uint32_t* c_list_n;        // [ncub]
  uint32_t* c_nsky;          // [ncub] outputs of phase S
  uint32_t* c_next;          // [ncub]
  uint32_t* c_flag;          // [ncub] 1: over a capacity; 2: skipped (job handed over)
  uint32_t* slot;            // [ncub * kLvSlot]: skyline ids, then extended
  unsigned long long* tab;   // [G * 128 * kLvMaxDims] first-level pruner tables
  uint32_t* pr_c;            // [G * kLvPruners] per scratch index
  float* pr_v;               // [G * kLvMaxDims * kLvPruners]
  uint32_t* pr_n;            // [G]
  uint32_t cap;              // survivors kept per cuboid
  uint32_t* cnt;             // [G]
  uint32_t* surv_id;         // [G * cap]
  uint16_t* surv_key;        // [G * cap]
  uint32_t* srt;             // [G * cap]
  uint32_t n_items;
  const uint32_t* it_cub;    // [n_items]
  const uint32_t* it_arg;    // [n_items] phase F: slice | slices << 16
  const uint32_t* it_phase;  // [n_items]
  const uint32_t* ph_size;   // [n_phases] items per phase
  const uint8_t* ph_kind;    // [n_phases] 0 P, 1 F, 2 S
  uint32_t* ph_done;         // [n_phases] zeroed before the launch
  uint32_t* next_item;       // zeroed before the launch
  uint32_t* job_over;        // [jobs] first-level cuboids over a capacity (zeroed)
  uint32_t max_fallbacks;    // more than this on a job's first level: job handed over
  uint32_t* status;          // 0, or 1 when a wait ran out (zeroed)
};
int launch_lv_counts(cudaStream_t s, const uint32_t* index, uint32_t nsub, uint32_t full_n,
                     const uint32_t* n_of, uint32_t* counts);
int launch_lv_lists(cudaStream_t s, const uint32_t* mask, uint32_t cub0, uint32_t ncub,
                    const uint32_t* slot, const uint32_t* skip, const uint32_t* n_of,
                    const uint64_t* off, const uint32_t* full, uint32_t full_c, uint32_t full_n,
                    uint32_t* out);
// One cooperative launch of the lattice kernel on `num_sms` SMs.
int launch_lattice(cudaStream_t s, int num_sms, const LtArgs& a);
int lattice_grid(int num_sms, int* grid);
int launch_cells_bytes(cudaStream_t s, const uint4* cells, const uint32_t* m_ptr, uint64_t m_max,
                       int d, uint64_t pitch, uint8_t* out);
int launch_scatter_u4(cudaStream_t s, const uint4* in, const uint32_t* idx, const uint32_t* m_ptr,
                      uint64_t m_max, uint4* out);

void upload_submask_table();

}  // namespace skc
