// Internal interface between the host runtime (topk_abi.cpp) and the kernels.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include <string>

namespace topk {

constexpr int kScanThreads = 256;     // threads per scan CTA
constexpr uint32_t kMaxQ = 64;        // attributes per query
constexpr uint32_t kMaxK = 4096;      // largest k of the fused path
constexpr uint32_t kLdAlign = 64;     // device column stride alignment (rows)
constexpr int kMaxLevels = 12;        // merge-tree levels (fan-in >= 2, <= 4096 CTAs)
constexpr int kScanSmemFixed = 1536;  // barriers, control block, radix histogram, weights

// Threshold epochs of a scan (ScanParams::epochs): at most kMaxEpochs; in id order after
// tiles 1, 4, 16, ... of every CTA, in partition mode, where the threshold decides how far
// the scan goes, after 1, 2, 4, 8, ...
constexpr uint32_t kMaxEpochs = 8;
constexpr uint32_t kEpochShift = 2, kPartEpochShift = 1;

// Device-side per-context scratch of the fused scan.  Zero between queries (but for
// `gen`): the kernel puts every counter back before it ends.
struct ScanScratch {
  uint32_t g_thr;           // running global threshold key (objects below it cannot win)
  uint32_t g_app;           // the same for rows still to be scanned (ScanParams::epub): at least
                            // g_thr while the scan runs
  unsigned long long g_keep;  // the last epoch's bound: objects below this (key, ~id) cannot win
  uint32_t error;           // nonzero after a device wait gave up (bit 0: stage wait)
  uint32_t acc_reductions;  // CTA block-selects during this scan
  uint32_t last_cands;      // entries merged at the root of the last scan
  uint32_t last_reductions; // block-selects of the last scan
  // Diagnostics of a TOPK_BOUNDS_CHECK build: first failed check (code, block,
  // tile, two values); the access it guarded was skipped.
  uint32_t diag[5];
  uint32_t acc_tiles;       // tiles scanned during this scan (partition mode)
  uint32_t pad0[18];
  // The words that CTAs count on or poll sit in lines of their own: hundreds of polls a
  // microsecond on one line hold up every other access to it.
  unsigned long long g_hid; // no CTA holds an unpublished entry at or above this (key, ~id)
  uint32_t pub_arrived;     // CTAs that published their best entries (ScanParams::pub)
  uint32_t pub_n;           // entries published
  uint32_t epoch_arrived[kMaxEpochs];  // CTAs that published for an epoch
  uint32_t finishers;       // merge tree: its root and the coordinator, the later resets
  uint32_t pad1[19];
  // How the scan in flight ends: twice the number of scans finished on this scratch,
  // plus one while the current scan ends through its merge tree.  It moves on by two
  // when a scan is answered, so a CTA that waits for the decision sees it however
  // late it looks.
  uint32_t gen;
  uint32_t pad2[31];
  uint32_t epoch0_ready;    // 1 once epoch 0's bound is in g_thr, g_app and g_keep
  uint32_t pad3[31];
};
static_assert(sizeof(ScanScratch) == 512, "four 128-byte lines");

// TOPK_BOUNDS_CHECK codes
enum : uint32_t {
  kDiagAppend = 4,  // candidate append past capacity
  kDiagMerge = 8,   // merge load past capacity
};

struct ScanParams {
  const float *table;   // column-major, stride ld
  uint64_t ld;
  uint64_t row_begin;   // rows [row_begin, row_end) are scanned
  uint64_t row_end;
  uint64_t tile_begin;  // row_begin rounded down to 4 (16-byte copies)
  uint64_t tile_end;    // row_end rounded up to 4 (<= ld)
  uint64_t tile_step;   // rows from one tile to the next (the tile size)
  uint32_t num_tiles;
  uint32_t qq;
  uint32_t k;
  uint32_t cap;         // entries of the shared candidate buffer
  uint32_t mcap;        // shared entries: the buffer, then a select's output (<= k, padded
                        // to a power of two); the merge reuses all of them
  uint32_t fanin;       // merge-tree fan-in G
  uint32_t levels;      // merge-tree levels below the root (level l has nslots[l] slots)
  uint32_t nslots[kMaxLevels];
  uint32_t slot_off[kMaxLevels];  // first slot of level l in `slots` (slot = k entries)
  uint32_t done_off[kMaxLevels];  // first group counter of level l in `done`
  uint64_t wait_limit;  // polls per bounded wait
  uint32_t fault_mode;  // 1: wait on a barrier nothing completes (timeout test)
  ScanScratch *scratch;
  uint2 *slots;         // merge-tree slots, k entries each (key, id)
  // May be null (then the merge tree answers).  Else block 0 of the launch coordinates and
  // scans nothing (launch_scan adds it to the plan's grid).  At its end each scanning CTA
  // publishes its best entries here (at most kPubMaxEntries per CTA, about pub_m when it
  // holds more, in partition mode its best k where pub_exact allows); the coordinator answers the query from the published entries when none
  // of the unpublished ones can belong to the result, else raises the global threshold
  // to the k-th largest published key and starts the merge tree.  The CTAs wait for that
  // decision, at most pub_wait polls; one whose wait runs out takes the decision for
  // the tree.
  uint2 *pub;
  uint32_t pub_m;
  uint32_t pub_wait;
  uint32_t tree_end;   // nothing is published at the end: the tree answers and no CTA waits
  uint32_t pub_exact;  // partition mode: most entries that every CTA can publish at once
  // Threshold epochs (needs pub): after its tile 1, then 2^epoch_shift times as many,
  // and so on (`epochs` of them) each CTA publishes the best entries it holds (epoch_keys
  // of them, at most 32) in epub[epoch] (epub_stride entries each); the
  // coordinator raises the global threshold to the k-th best of them.  A CTA whose
  // buffer fills before epoch 0's bound is there waits for it, at most epoch_wait polls.
  uint2 *epub;
  uint32_t epub_stride;
  uint32_t epochs;
  uint32_t epoch_shift;
  uint32_t epoch_keys;
  uint32_t epoch_wait;
  // Partition mode: every CTA waits for epoch 0's bound after its first tile.  On a small
  // copy the few tiles it could scan meanwhile are most of what the stop rule would skip
  // (2^20 rows in 129 partitions: 66 % of them scanned without, 54 % with the wait).
  uint32_t epoch_hold;
  uint32_t *slot_count; // entries per slot
  uint32_t *done;       // per-group arrival counters (zero between queries)
  uint64_t *out_ids;    // min(k, rows) ids, ascending by score
  float *out_scores;
  float *out_threshold; // may be null
  uint32_t *out_count;  // may be null
  uint32_t *out_stats;  // may be null: [0] entries merged at the root, [1] block-selects,
                        // [2] tiles scanned (partition mode)
  // Partition mode (part_list != null): tile t covers rows
  //   part_list[t >> part_shift] << part_rows_log2  +  (t & ((1 << part_shift) - 1)) * tile
  // instead of tile_begin + t * tile; rows stay within [row_begin, row_end).
  const uint32_t *part_list;
  // May be null.  part_key[i] = order key of an upper bound of every score in partition
  // part_list[i], non-increasing in i: a CTA stops at its first tile whose bound is
  // below its threshold (every later tile of that CTA is bounded lower still) -- the
  // reference's stop rule (cpu/VTA.h:210-216, cpu/PTA.h:636-641) per partition.
  const uint32_t *part_key;
  uint32_t part_shift;      // log2(tiles per partition)
  uint32_t part_rows_log2;  // log2(rows per partition)
  const uint32_t *row_ids;  // may be null: id of each row (a reordered table's original ids)
  uint32_t thr_seed;        // objects need key >= thr_seed from the start (0: none)
  const uint32_t *thr_seed_dev;  // may be null: a further seed read from device memory at start
  uint8_t attr[kMaxQ];
  float w[kMaxQ];       // weights[attr[m]], gathered on the host
  // Set by launch_scan: the first four queried columns (table + attr[m] * ld), the
  // rows from one tile of a CTA to its next in id order (grid * tile_step), and the
  // tiles [int_lo, int_lo + int_n) that lie wholly inside [row_begin, row_end).
  const float *colp[4];
  uint32_t ncta;        // scanning CTAs: the plan's grid
  uint64_t grid_rows;
  uint32_t int_lo;
  uint32_t int_n;
};

// Publishing (ScanParams::pub): grids of at least kPubMinGrid CTAs; the arrays need
// grid * kPubMaxEntries entries and grid * kPubMaxKeys entries per epoch.
constexpr uint32_t kPubMinGrid = 2;
// Polls of the two waits, about 1 us and 0.25 us apart (a decision wait hides behind the
// answering CTA's last microseconds; waiting longer for epoch 0 costs more than a select).
constexpr uint32_t kPubWaitPolls = 256, kPubWaitNs = 1000;
constexpr uint32_t kEpochWaitPolls = 64, kEpochWaitNs = 250;
constexpr uint32_t kPubMaxKeys = 32;     // of an epoch: 4 per warp
constexpr uint32_t kPubMaxEntries = 96;  // at the end (the list and 32 words in 1 KB)
// Entries a CTA that holds more than kPubMaxEntries aims to publish.  With the k best
// spread over the CTAs it holds lambda = k / grid of them; lambda + 3 sqrt(lambda) + 1.6
// leaves one out in under 1-3 % of queries (then the merge tree answers).  In a scan with
// epochs it holds that many only when much of the result is in it, and publishes about as
// many as it can bound (24 of the 32 best of its threads).  Where lambda is too large for
// that, grids of at least 16 CTAs publish 28 each, or all 32 where k needs them, whose k-th
// bounds what the tree carries (40,000 rows, k = 1000: 63 us a query against 104 without;
// 102,000 rows, k = 3000 and 3190: 111 and 116 us with 32, 288-373 without); below, or with
// too few CTAs for k entries, publishing is in vain (14 us of 57) and the tree answers alone: 0.
inline uint32_t pub_entries(uint32_t k, uint32_t grid, uint32_t epochs) {
  if (grid < kPubMinGrid || (uint64_t)grid * kPubMaxEntries < k) return 0;
  if (epochs) return 24;
  const double l = (double)k / grid;
  const uint32_t r = (uint32_t)__builtin_ceil(l + 3.0 * __builtin_sqrt(l) + 1.6);
  if (r <= 24) return r;
  return grid < 16 || 32u * grid < k ? 0 : 28u * grid >= k ? 28 : 32;
}
// Epochs of a scan over `tiles` tiles, after 1, m, m^2, ... tiles (m = 2^shift): each ends
// before the scan does, with every CTA still taking part.
inline uint32_t scan_epochs(uint64_t tiles, uint32_t grid, uint32_t shift) {
  uint32_t e = 0;
  for (uint64_t at = 1; at * grid < tiles && e < kMaxEpochs; at <<= shift) ++e;
  return e;
}
// Entries a CTA publishes per epoch, at least 3k / 2 in all: with k = 256 of 739 CTAs the
// k-th best of every CTA's best lies at rank ~315 of all.  More would tighten the bound
// a little and lengthen the coordinator's pass, which every CTA waits for in epoch 0
// (8 per CTA at k = 256 cost 13 us a query on 2^24 rows).  In partition mode, where the
// best objects sit close together and the bound decides how far the scan goes, 4k in all
// and 4 per CTA at least.
inline uint32_t epoch_keys(uint32_t k, uint32_t grid, bool part) {
  const uint32_t want = part ? 4u * k : 3u * k / 2u, least = part ? 4u : 1u;
  const uint32_t r = (want + grid - 1u) / grid;
  return r < least ? least : r < kPubMaxKeys ? r : kPubMaxKeys;
}

struct ScanPlan {
  uint32_t tile;     // objects per tile
  uint32_t stages;   // 1 when the request fits in shared memory, else 0
  uint32_t cap;
  uint32_t mcap;
  uint32_t fanin;
  int ctas_per_sm;
  size_t smem;       // dynamic shared memory bytes
  int grid;
};

// Plan a launch for qq attributes and top-k over `rows` rows (max_ctas_per_sm 0 =
// as many as fit).  stages == 0 means the request does not fit.
ScanPlan plan_scan(uint32_t qq, uint32_t k, uint64_t rows, int num_sms, size_t smem_optin,
                   uint32_t max_ctas_per_sm = 0, bool part = false);
// Fill the merge-tree fields of p for `grid` CTAs; returns slots and group
// counters needed (entries = slots * k).
void plan_merge_tree(ScanParams &p, uint32_t grid, uint32_t fanin, uint32_t *total_slots, uint32_t *total_groups);
cudaError_t launch_scan(const ScanPlan &plan, const ScanParams &p, cudaStream_t stream);
cudaError_t scan_set_attributes(size_t smem_optin);

// Merge of per-shard top-k lists (merge.cu): list j at lists + j * 12 * stride holds
// ids[stride] (u64) then scores[stride] (f32), counts[j] of them valid, base[j] (may
// be null: 0) added to its ids; the best min(k, sum of counts) of the union (score
// descending, then lower id) are written ascending to out_ids / out_scores, the k-th
// score to out_thr (may be null).
constexpr uint32_t kMaxMergeLists = 64;
cudaError_t launch_merge_lists(const unsigned char *lists, uint32_t nlists, uint64_t stride, const uint32_t *counts,
                               const uint32_t *base, uint32_t k, uint64_t *out_ids, float *out_scores, float *out_thr,
                               uint32_t *kept, cudaStream_t s);

// Set the calling thread's message returned by topk_last_error().
void set_last_error(const char *msg);

// Table kernels.
cudaError_t launch_generate(float *table, uint64_t ld, uint32_t d, uint64_t n, int dist, uint64_t seed,
                            cudaStream_t stream);
// Per-column min/max with std::min/std::max semantics.
cudaError_t launch_minmax(const float *table, uint64_t ld, uint32_t d, uint64_t n, uint32_t *work,
                          cudaStream_t stream);
cudaError_t launch_normalize(float *table, uint64_t ld, uint32_t d, uint64_t n, const float *mins,
                             const float *ranges, cudaStream_t stream);
// work layout for launch_minmax (uint32 words): per column
//   [0] max key, [1] min key, [2..3] first +0 index, [4..5] first -0 index; 8 words per column.
constexpr int kMinmaxWords = 8;

// Plain reference-order count of objects in [r0, r1) with score >= thr and > thr.
cudaError_t launch_count(const float *table, uint64_t ld, uint64_t r0, uint64_t r1, uint32_t qq,
                         const uint8_t *attr, const float *w, float thr, unsigned long long *out2,
                         cudaStream_t stream);
// Gather full rows for a list of ids: out[j*d + m] = table[m*ld + ids[j]].
cudaError_t launch_gather(const float *table, uint64_t ld, uint32_t d, const uint64_t *ids, uint64_t cnt,
                          float *out, cudaStream_t stream);

// Partitioned copy (partition.cu): Morton-ordered counting sort of the rows into
// ptable (same stride), perm[row] = original id.  lo/scale: per attribute (device),
// scale = 2^bits / (max - min).  keys: n entries; hist: 2^16 entries.
cudaError_t launch_partition_build(const float *table, uint64_t ld, uint32_t d, uint64_t n, const float *lo,
                                   const float *scale, uint32_t bits, uint16_t *keys, uint32_t *hist,
                                   uint32_t *perm, float *ptable, int num_sms, cudaStream_t s);
// Index orders of the reference as a row permutation: VTA's (cpu/VTA.h:121-135), the
// same over kVtaThreadRanges equal row ranges as VTA's threaded build makes it (IMP 2,
// VPARTITIONS = THREADS, cpu/VTA.h:13,78-85), PTA's (cpu/PTA.h:88-167, 203-236).
// work holds index_order_work_words(n, kind) words; temp is the radix sorts' scratch
// (first call with temp == nullptr to size it).  n < 2^31; PTA also needs n >= 2 and
// d <= 32.
// kGroups: VTA's order inside caller-given groups (device array `groups`, each value
// < 2^group_bits, group_bits <= 31), groups by number: SLA's index with the skyline
// layer as the group (cpu/SLA.h:199-251).
enum class IndexOrder { kVta, kVtaThreads, kPta, kGroups };
constexpr uint32_t kVtaThreadRanges = 16;
uint64_t index_order_work_words(uint64_t n, IndexOrder kind);
cudaError_t launch_index_order(const float *table, uint64_t ld, uint32_t d, uint64_t n, IndexOrder kind,
                               uint32_t *perm, uint32_t *work, void *temp, size_t *temp_bytes, int num_sms,
                               cudaStream_t s, const uint32_t *groups = nullptr, uint32_t group_bits = 0);
// SLA's skyline layers (skyline.cu; cpu/SLA.h:102-139): the layer of every row, 0 = the
// first skyline, with the reference's stop rule (the last <= 100 rows form one layer).
// d <= 32, n < 2^31.  layers: n entries on the host.
int skyline_layers_device(const float *table, uint64_t ld, uint32_t d, uint64_t n, int num_sms, uint32_t *layers,
                          uint64_t *num_layers, std::string *msg);
// A row-major copy of the table for an index build (n * row_stride(d) floats), which reads
// whole rows in random order; `rows` below may be null (then the columns are read).
inline uint32_t row_stride(uint32_t d) { return (d + 3u) / 4u * 4u; }
cudaError_t launch_rows(const float *table, uint64_t ld, uint32_t d, uint64_t n, float *rows, int num_sms,
                        cudaStream_t s);
cudaError_t launch_gather_rows(const float *table, uint64_t ld, uint32_t d, uint64_t n, const uint32_t *perm,
                               float *ptable, int num_sms, cudaStream_t s, const float *rows);
// kd order (partition.cu): the partitions of 2^part_log2 rows are the leaves of a
// balanced binary tree; each node is split at its middle partition boundary after its
// rows are sorted by the attribute of widest spread in it.  n < 2^31.  work:
// kd_order_work_words(n, d, P) words; temp: CUB storage (size query with temp null).
uint32_t kd_levels(uint32_t P);
uint64_t kd_order_work_words(uint64_t n, uint32_t d, uint32_t P);
cudaError_t launch_kd_order(const float *table, uint64_t ld, uint32_t d, uint64_t n, uint32_t part_log2,
                            uint32_t *perm, uint32_t *work, void *temp, size_t *temp_bytes, int num_sms,
                            cudaStream_t s, const float *rows);
// One query's attributes and gathered weights, for partition bounds.
struct PartQuery {
  uint32_t qq;
  uint8_t attr[kMaxQ];
  float w[kMaxQ];  // weights[attr[m]]
};
// Partitions in descending order of the query's bound (the reference-order FP32 sum
// over each partition's per-attribute max, or min for negative weights: an exact upper
// bound of its rows' scores): plist[i] = partition, pkey[i] = order key of an upper
// bound of its scores, non-increasing in i (0xFFFFFFFF for a NaN bound).  Up to
// kPartOrderOneBlock partitions one block orders them by a counting sort into 1024
// buckets over the range of the keys, pkey[i] = the largest key of i's bucket,
// partitions of one bucket in no set order; above, an exact radix sort (ties by the
// lower partition number) uses `temp` (part_order_temp_bytes(P) bytes).
constexpr uint32_t kPartOrderOneBlock = 16384;
size_t part_order_temp_bytes(uint32_t P);
cudaError_t launch_part_order(const float *pmin, const float *pmax, uint32_t P, uint32_t d, const PartQuery &q,
                              uint32_t *plist, uint32_t *pkey, void *temp, size_t temp_bytes, int num_sms,
                              cudaStream_t s);
// Per-partition min / max / mean of each attribute, [num_parts][d] each.
cudaError_t launch_partition_stats(const float *ptable, uint64_t ld, uint32_t d, uint64_t n, uint32_t rows_log2,
                                   uint32_t num_parts, float *mins, float *maxs, float *means, cudaStream_t s);

// Table files (loader.cu).  csv_shape: File<T>::count's n (newlines) and d (1 + commas
// of the first line).  load_csv_device: parses the first n rows of a comma-separated
// file into the column-major table on the device (FP32 correctly rounded, as fscanf's
// "%f"); stats (may be null): bytes consumed, rows found, host-converted values,
// chunks.  Both return a TOPK_* code and a message on failure.
int csv_shape(const char *path, uint64_t *n, uint64_t *d, std::string *msg);
struct LoaderState;  // the loader's pipeline buffers, kept between loads
LoaderState *loader_state_new();
void loader_state_free(LoaderState *L);
int load_csv_device(LoaderState *L, const char *path, float *table, uint64_t ld, uint32_t d, uint64_t n,
                    int num_sms, uint64_t chunk_bytes, uint64_t stats[4], std::string *msg);
int save_csv(const char *path, const float *table, uint64_t ld, uint32_t d, uint64_t n, std::string *msg);
// Binary column-major files: 64-byte header ("TOPKCOL1", version 1, element size 4, n,
// d), then d columns of n FP32 values.
int binary_shape(const char *path, uint64_t *n, uint64_t *d, std::string *msg);
int save_binary(const char *path, const float *table, uint64_t ld, uint32_t d, uint64_t n, std::string *msg);
int load_binary_device(LoaderState *L, const char *path, float *table, uint64_t ld, uint32_t d, uint64_t n,
                       std::string *msg);
// Row-major host tables (row i at host + i*row_stride) to and from the column-major
// device table, through the loader's buffers and a tiled transpose.
int upload_rowmajor_device(LoaderState *L, const float *host, uint64_t row_stride, float *table, uint64_t ld,
                           uint32_t d, uint64_t n, std::string *msg);
int download_rowmajor_device(LoaderState *L, float *host, uint64_t row_stride, const float *table, uint64_t ld,
                             uint32_t d, uint64_t n, std::string *msg);

// Threshold algorithm over sorted lists (ta.cu; cpu/TA.h).  ta_lists_build: per
// attribute the ids by value descending (ties by the lower id) and the sorted values,
// plus query scratch.  ta_query: exact top-k by walking the queried lists (results of
// the full scan); stats: depth walked, objects scored, blocks.  One query at a time
// per TaLists.
struct TaLists;
int ta_lists_build(TaLists **out, const float *table, uint64_t ld, uint32_t d, uint64_t n, int num_sms,
                   std::string *msg);
void ta_lists_free(TaLists *L);
int ta_lists_read(const TaLists *L, uint32_t m, uint32_t *ids, float *vals, std::string *msg);
int ta_query(TaLists *L, const float *table, uint64_t ld, uint64_t k, uint32_t qq, const float *weights,
             const uint8_t *attr, int num_sms, uint64_t *ids, float *scores, uint64_t *count, float *threshold,
             uint64_t *stats, std::string *msg);

}  // namespace topk
