// Fused single-query scan + exact top-k select (sm_100a).
//
// Replaces the TPAc full-table evaluation (cpu/TPAc.h:118-207 findTopKsimd,
// :257-358 findTopKthreads): the same per-object arithmetic
//     s = 0; for m in attr order: s = s + x[attr[m]] * w[attr[m]]   (RN mul, RN add)
// and the same result (the k best by score; ties here go to the lower id).
//
// Persistent CTAs of 256 threads, several per SM:
//   * Each tile is 1024 objects (4 per thread).  A thread issues one 128-bit
//     streaming load (ld.global.cs) per queried column for its 4 objects, all of
//     them before the first multiply, so each warp keeps q x 512 bytes in flight and
//     an SM with several CTAs keeps far more than the ~45 KB that HBM3e latency
//     needs.  Only the queried columns are read.  (A TMA bulk-copy ring with a
//     producer warp was measured on this GPU at 2.6-4.9 TB/s against 3.1-5.9 TB/s
//     for plain loads, so the scan uses plain loads.)  For q <= 4 a thread also keeps
//     the next tile's loads in flight while it scores, appends and synchronises on
//     the current one, and loads a partial tile's rows past its end from row 0 (in
//     bounds, masked out) instead of selecting zeros value by value (q = 2: 3.3 ->
//     3.6 TB/s; q = 4: 4.5 -> 5.5 TB/s, same-box A/B).
//   * An object passes if its score is >= the running threshold; passing objects
//     go to a shared candidate buffer (warp-aggregated append).  When the buffer
//     nears capacity (a barrier vote, so every thread decides alike) the CTA drops
//     what lies below the threshold by now, in place; only when that leaves too much
//     (equal scores, or no bound yet) does it keep its top-k by an 8-bit radix select
//     on the 64-bit (key, ~id) word.
//   * The threshold comes from the grid as a whole: after tiles 1, 4, 16, ... every CTA
//     publishes the largest keys it holds, and block 0, which scans nothing, takes the
//     k-th largest of them -- k real objects score at least that -- as the threshold of
//     all (epoch_publish, coordinate).  A CTA's own k-th best is the k-th of its share
//     only: with k = 1024 of 739 CTAs it let ~700 times too much through, and every CTA
//     ran selects and passed k entries up a merge tree.
//   * Bounds are (key, ~id) composites, so equal scores at the k-th are cut by id as well:
//     on tables with many equal rows (values clipped at 1) every CTA used to pass its k
//     ties up the merge tree.  Appending compares keys only, in id order strictly: the rows
//     a CTA still has to scan come after every published one and lose a tie.
//   * End: each CTA publishes what it still holds above the threshold, about k entries in
//     all, and the coordinator ranks them and writes the result.  Where the published
//     entries cannot hold it (the best rows side by side in one CTA, a large k over few
//     tiles) a merge tree with fan-in G answers: each CTA writes its best k to a slot; the
//     last CTA of each group of G slots (per-group arrival counter) merges them to k
//     entries in shared memory and moves up; the root sorts (bitonic) and writes the
//     result.  Counters are put back to zero for the next query.
//   Measured (us a query on a stream, independent rows, without epochs and coordinator ->
//   with): 2^20 rows q = 4 k = 16 39.0 -> 25.0, k = 256 67 -> 31; 2^24 rows q = 2 k = 16 73
//   -> 52, k = 1024 272 -> 83, q = 8 k = 1024 199 -> 127; 2^27 rows q = 4 k = 1024 482 -> 359
//   (two launches before: a threshold pass over every 64th tile first), q = 2 k = 16 238 ->
//   218.  Correlated rows, many equal: 2^24 rows q = 2 k = 1024 203 -> 71.
//   A launch's fixed cost is what is left: the first tiles' latency (~5 us), the first
//   epoch (~8 us, hidden from q = 8 on), the end (~10 us).
#include <cstdint>
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>

#include "block_select.cuh"
#include "device_common.cuh"
#include "topk_internal.h"

namespace topk {

namespace {

struct SmemCtl {
  uint32_t count;      // entries in the current candidate buffer
  uint32_t thr_local;  // min key that can still enter (k-th CTA key + 1)
  uint32_t thr_g[2];   // CTA copy of the global threshold: tile i reads [i & 1], thread 0
                       // writes [(i + 1) & 1] before tile i's barrier, so with a vote
                       // barrier every tile (partition mode, whose stop rule needs it)
                       // every thread of a tile reads the same value; with a vote every
                       // two tiles a thread may read a slot before or after an update,
                       // both valid bounds
  uint32_t reductions;
  uint32_t is_last;
  uint32_t red_g;      // threshold snapshot shared by the block
  uint32_t state;      // the end of the scan as this CTA goes on: kEndDone, kEndTree
  uint32_t gen0;       // the decision word as the scan started (it changes only after every
                       // CTA has arrived)
  uint32_t epoch0_seen;  // epoch 0's bound has been waited for
  uint32_t my_tiles;   // tiles of this CTA (read where it is rare: it holds no register)
  uint32_t epoch;      // next threshold epoch
  unsigned long long keep;  // no entry of this CTA below this composite can belong to the
                            // result (inclusive, unlike thr_g: entries that tie a bound's
                            // key may have come before it)
  SelShared sel;       // state of the block-wide selects
};

// shared layout
constexpr int kOffCtl = 0;        // SmemCtl (112 B)
constexpr int kOffNever = 112;    // test barrier (u64)
constexpr int kOffHist = 128;     // 256-bin radix histogram
constexpr int kOffWsm = 1152;     // weights of the runtime-q path (kMaxQ floats)
constexpr int kOffScnt = 1408;    // entry counts of a merge group's slots (kMaxFanin words)
constexpr int kOffCand = kScanSmemFixed;
constexpr uint32_t kMaxFanin = 32;  // merge-tree fan-in at most (small k: two levels for 592 CTAs)
static_assert(kOffWsm + 4 * (int)kMaxQ <= kOffScnt && kOffScnt + 4 * (int)kMaxFanin <= kScanSmemFixed,
              "fixed shared block");
static_assert(sizeof(SmemCtl) <= kOffNever, "control block layout");
static_assert(kScanThreads == 256, "one histogram bin per thread");

constexpr int kVec = 4;                      // objects per thread per tile
constexpr uint32_t kTile = kScanThreads * kVec;

__device__ __forceinline__ void bsync() { __syncthreads(); }

// TOPK_BOUNDS_CHECK: record the first failed check in scratch->diag and tell the
// caller to skip the guarded access.  Compiled out of the product build.
#ifdef TOPK_BOUNDS_CHECK
__device__ __forceinline__ bool check(bool ok, ScanScratch *s, uint32_t code, uint32_t i, uint32_t a, uint32_t b) {
  if (!ok && atomicCAS(&s->diag[0], 0u, code) == 0u) {
    s->diag[1] = blockIdx.x;
    s->diag[2] = i;
    s->diag[3] = a;
    s->diag[4] = b;
  }
  return ok;
}
#define TOPK_CHECK(cond, code, i, a, b) check((cond), p.scratch, (code), (i), (a), (b))
#else
#define TOPK_CHECK(cond, code, i, a, b) (true)
#endif

__device__ __forceinline__ float4 ld_stream(const float *p) { return __ldcs(reinterpret_cast<const float4 *>(p)); }

// Scores of this thread's 4 objects at rows [row0, row0+4) of one tile, reference
// order.  QQ > 0: compile-time attribute count, every load issued before the first
// multiply, weights as constant-bank operands.  QQ == 0: runtime count, weights
// from shared memory.  `guard`: partial tile, load only below tile_end.
template <int QQ>
__device__ __forceinline__ float4 score4(const ScanParams &p, const float *wsm, uint32_t qq, uint64_t row0,
                                         bool guard) {
  float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f, a3 = 0.0f;
  const bool inb = !guard || row0 < p.tile_end;  // tile_end <= ld, multiple of 4
  if constexpr (QQ > 0) {
    float4 x[QQ];
#pragma unroll
    for (int m = 0; m < QQ; ++m)
      x[m] = inb ? ld_stream(p.table + (uint64_t)p.attr[m] * p.ld + row0) : make_float4(0.f, 0.f, 0.f, 0.f);
    // every load is issued before the first multiply (the compiler may not sink them
    // below this point): QQ x 16 bytes in flight per thread
    asm volatile("" ::: "memory");
#pragma unroll
    for (int m = 0; m < QQ; ++m) {
      const float w = p.w[m];
      a0 = __fadd_rn(a0, __fmul_rn(x[m].x, w));
      a1 = __fadd_rn(a1, __fmul_rn(x[m].y, w));
      a2 = __fadd_rn(a2, __fmul_rn(x[m].z, w));
      a3 = __fadd_rn(a3, __fmul_rn(x[m].w, w));
    }
  } else {
    uint32_t m = 0;
    for (; m + 4 <= qq; m += 4) {  // four loads in flight at a time
      float4 x[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        x[u] = inb ? ld_stream(p.table + (uint64_t)p.attr[m + u] * p.ld + row0) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float w = wsm[m + u];
        a0 = __fadd_rn(a0, __fmul_rn(x[u].x, w));
        a1 = __fadd_rn(a1, __fmul_rn(x[u].y, w));
        a2 = __fadd_rn(a2, __fmul_rn(x[u].z, w));
        a3 = __fadd_rn(a3, __fmul_rn(x[u].w, w));
      }
    }
    for (; m < qq; ++m) {
      const float4 x = inb ? ld_stream(p.table + (uint64_t)p.attr[m] * p.ld + row0) : make_float4(0.f, 0.f, 0.f, 0.f);
      const float w = wsm[m];
      a0 = __fadd_rn(a0, __fmul_rn(x.x, w));
      a1 = __fadd_rn(a1, __fmul_rn(x.y, w));
      a2 = __fadd_rn(a2, __fmul_rn(x.z, w));
      a3 = __fadd_rn(a3, __fmul_rn(x.w, w));
    }
  }
  return make_float4(a0, a1, a2, a3);
}

// Loads of this thread's 4 objects at rows [row0, row0+4) in the QQ queried columns,
// and their scores in reference order.  `guard`: partial tile; a thread whose rows
// lie at or past tile_end loads row 0 instead (always in bounds) and its scores are
// meaningless — the caller's row-range mask drops them.  One select per tile, none
// per value, and the column pointers computed once by the caller.
template <int QQ>
__device__ __forceinline__ void load_cols(const ScanParams &p, const float *const *col, uint64_t row0, bool guard,
                                          float4 *x) {
  row0 = (!guard || row0 < p.tile_end) ? row0 : 0;
#pragma unroll
  for (int m = 0; m < QQ; ++m) x[m] = ld_stream(col[m] + row0);
}
template <int QQ>
__device__ __forceinline__ float4 score_cols(const ScanParams &p, const float4 *x) {
  float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f, a3 = 0.0f;
#pragma unroll
  for (int m = 0; m < QQ; ++m) {
    const float w = p.w[m];
    a0 = __fadd_rn(a0, __fmul_rn(x[m].x, w));
    a1 = __fadd_rn(a1, __fmul_rn(x[m].y, w));
    a2 = __fadd_rn(a2, __fmul_rn(x[m].z, w));
    a3 = __fadd_rn(a3, __fmul_rn(x[m].w, w));
  }
  return make_float4(a0, a1, a2, a3);
}

// Up to this many queried columns the scan keeps the next tile's loads in flight
// while it scores, appends and synchronises on the current one (few columns give a
// thread too few bytes in flight otherwise).
constexpr int kPrefetchQ = 4;

// Tiles between two votes on the buffer's fill (see scan_select_kernel).
__host__ __device__ constexpr uint32_t scan_vote_tiles(int qq, bool part) {
  return (qq >= 1 && qq <= 2 && !part) ? 2u : 1u;
}

// CTAs per SM the register budget is sized for: one queried column needs little data
// in flight and gains from more CTAs (6: 40 registers); more columns need their loads
// in flight (5: 48 registers up to 8 columns; 4: 64 above and with a run-time count, which
// took 4 % longer with 48.  8 to 32 bytes spill at q = 1, 4 and 14 to 16, 4 in partition
// mode).
// Partition mode runs at most 4 CTAs per SM, so it has their registers.  Two attributes in
// id order take 48 registers at 5 CTAs; at 6 the loop spilled (2^28 rows, independent, us
// at k = 16 / 1024 / 4096: 430 / 534 / 1110 with 6, 400 / 448 / 819 with 5).
template <int QQ, bool PART>
constexpr int scan_min_blocks() {
  return PART ? 4 : QQ == 1 ? 6 : (QQ >= 2 && QQ <= 8) ? 5 : 4;
}

// ---------------------------------------------------------------- results
// Put the scratch back to zero for the next scan (one thread, after everything else; the
// kernel's end makes it visible, a fence here would wait for the result's way to the host).
__device__ __forceinline__ void reset_scratch(ScanScratch *s) {
  s->acc_reductions = 0;
  s->acc_tiles = 0;
  s->pub_arrived = 0;
  s->pub_n = 0;
  s->g_hid = 0;
  s->g_keep = 0;
  s->finishers = 0;
  s->epoch0_ready = 0;
  for (uint32_t e = 0; e < kMaxEpochs; ++e) s->epoch_arrived[e] = 0;
  s->g_thr = 0;
  s->g_app = 0;
}

// The scan's statistics (thread 0 of the CTA that answers).
__device__ __forceinline__ void write_stats(const ScanParams &p, uint32_t merged, uint32_t res_n) {
  ScanScratch *s = p.scratch;
  if (p.out_count) *p.out_count = res_n;
  const uint32_t reds = ld_volatile_u32(&s->acc_reductions);
  const uint32_t tiles = ld_volatile_u32(&s->acc_tiles);
  s->last_cands = merged;
  s->last_reductions = reds;
  if (p.out_stats) {
    p.out_stats[0] = merged;
    p.out_stats[1] = reds;
    p.out_stats[2] = tiles;
  }
}

// res[0..res_n) descending -> the result, ascending (whole CTA).
__device__ __forceinline__ void write_sorted(const ScanParams &p, const uint2 *res, uint32_t res_n, uint32_t merged) {
  const int t = threadIdx.x;
  for (uint32_t r = t; r < res_n; r += kScanThreads) {
    const uint2 e = res[r];
    const uint32_t pos = res_n - 1 - r;  // ascending output
    p.out_ids[pos] = (uint64_t)e.y;
    p.out_scores[pos] = key2f(e.x);
  }
  if (t == 0) {
    if (p.out_threshold) *p.out_threshold = res_n ? key2f(res[res_n - 1].x) : 0.0f;
    write_stats(p, merged, res_n);
  }
}

// ---------------------------------------------------------------- publishing
constexpr uint32_t kEndDone = 0, kEndTree = 1;
// Entries ranked by counting alone, one per thread.
constexpr uint32_t kRankMax = kScanThreads;
// Up to this k a CTA bounds its own k-th best from 32 of its threads' largest keys.
constexpr uint32_t kLocalBoundK = 32;

// The r <= 4 largest of a warp's 32 keys, one per lane, each handed to put(0..r, key, id)
// on the lane that holds it (key 0: none left).
template <class Put>
__device__ __forceinline__ void warp_top(uint32_t key, uint32_t id, uint32_t r, int lane, Put put) {
#pragma unroll 1
  for (uint32_t x = 0; x < r; ++x) {
    const uint32_t w = __reduce_max_sync(0xFFFFFFFFu, key);
    if (lane == __ffs(__ballot_sync(0xFFFFFFFFu, key == w)) - 1) {
      put(x, w, id);
      key = 0;
    }
  }
}

// The next threshold epoch, after every append of the segment: this CTA publishes the
// best of its threads' best entries, epoch_keys of them, for the coordinator; nothing
// here waits for it.  In epoch 0 with k <= kLocalBoundK the CTA also takes the k-th best
// of 32 of those as a first bound of its own, so its buffer does not fill before epoch
// 0's bound is there.
__device__ __forceinline__ void epoch_publish(const ScanParams &p, const uint2 *cand, SmemCtl *ctl, uint32_t *hist) {
  const int t = threadIdx.x;
  const int lane = t & 31, warp = t >> 5;
  const uint32_t epoch = ctl->epoch;
  unsigned long long *words = reinterpret_cast<unsigned long long *>(hist);  // 4 per warp
  uint2 *mine = p.epub + (size_t)epoch * p.epub_stride + (size_t)(blockIdx.x - 1u) * p.epoch_keys;
  bsync();
  const uint32_t n = ctl->count;
  // this thread's best (of equal keys any); a short buffer is dealt over the warps entry by
  // entry
  uint2 m = make_uint2(0u, 0u);
  if (n <= (uint32_t)kScanThreads) {
    const uint32_t j = (uint32_t)lane * (kScanThreads / 32) + (uint32_t)warp;
    if (j < n) m = cand[j];
  } else {
#pragma unroll 4
    for (uint32_t j = t; j < n; j += kScanThreads) {
      const uint2 e = cand[j];
      if (e.x > m.x) m = e;
    }
  }
  // the best of each warp's lanes: enough for r of the block, or for a bound of its own
  const uint32_t r = p.epoch_keys;
  const bool local = epoch == 0 && p.k <= kLocalBoundK;
  if (lane < 4) words[4 * warp + lane] = 0ull;
  __syncwarp();
  warp_top(m.x, m.y, local || r > 8u ? 4u : r > 2u ? 2u : 1u, lane,
           [&](uint32_t x, uint32_t key, uint32_t id) { words[4 * warp + x] = key ? composite(key, id) : 0ull; });
  bsync();
  if (warp == 0) {
    const uint64_t v = warp_sort_desc<uint64_t>(words[lane], lane);
    if ((uint32_t)lane < r) mine[lane] = make_uint2((uint32_t)(v >> 32), 0xFFFFFFFFu - (uint32_t)v);
    // rows in id order lose a tie with the k-th; rows with ids of their own may win it
    if (local && lane == (int)p.k - 1 && v) {
      ctl->keep = v;
      ctl->thr_local = max(ctl->thr_local, (uint32_t)(v >> 32) + (p.row_ids ? 0u : 1u));
    }
    __threadfence();
    __syncwarp();
    if (lane == 0) {
      atomicAdd(&p.scratch->epoch_arrived[epoch], 1u);
      ctl->epoch = epoch + 1u;
    }
  }
  bsync();  // the buffer and the control block have been read and written
}

// The bounds known by now into the CTA's thresholds (thread 0; barriers around it).  With
// `wait`, epoch 0's is waited for when it is still on its way.
__device__ __forceinline__ void take_bound(const ScanParams &p, SmemCtl *ctl, bool wait) {
  ScanScratch *sc = p.scratch;
  if (p.epochs && !ctl->epoch0_seen) {
    uint32_t ready = ld_volatile_u32(&sc->epoch0_ready);
    for (uint32_t it = 0; it < p.epoch_wait && !ready && wait; ++it) {
      __nanosleep(kEpochWaitNs);
      ready = ld_volatile_u32(&sc->epoch0_ready);
    }
    ctl->epoch0_seen = (ready || wait) ? 1u : 0u;
  }
  const uint64_t g = max((uint64_t)ld_volatile_u64(&sc->g_keep), (uint64_t)ld_volatile_u32(&sc->g_thr) << 32);
  if (g > ctl->keep) ctl->keep = g;
  ctl->thr_g[0] = ctl->thr_g[1] =
      max(max(ctl->thr_g[0], ctl->thr_g[1]), max((uint32_t)(ctl->keep >> 32), ld_volatile_u32(&sc->g_app)));
}

// The end of a CTA's scan (p.pub set): it publishes its entries at or above its running
// bound when they are at most kPubMaxEntries, else those at or above the pub_m-th best of
// its threads' best, and keeps the largest such limit of any CTA in g_hid: no unpublished
// entry that could belong to the result reaches it.  Then it waits for the coordinator's
// decision; true: the merge tree answers.
// In partition mode the best rows lie together, so one CTA often holds most of the result
// and the limit fails; with k <= pub_exact such a CTA selects its best k instead, which
// hide nothing.  (Its select takes a few us, the tree 20: 758,368 x 4 rows in 93 partitions,
// k = 81: 65.1 us a query through the tree, 50.4 so.)
template <bool PART>
__device__ __forceinline__ bool publish_entries(const ScanParams &p, uint2 *cand, SmemCtl *ctl, uint32_t *hist) {
  const int t = threadIdx.x;
  const int lane = t & 31, warp = t >> 5;
  ScanScratch *sc = p.scratch;
  if (p.tree_end) {
    if (t == 0) atomicAdd(&sc->pub_arrived, 1u);
    return true;
  }
  const uint32_t n = ctl->count;
  uint32_t *keys = hist;                               // 4 per warp, before the list
  uint2 *list = reinterpret_cast<uint2 *>(hist + 64);  // kPubMaxEntries entries
  if (t == 0) {
    ctl->sel.valid = 0;
    ctl->sel.wcount = 0;
    // the last epoch's bound (a CTA of two or three tiles may be here before epoch 0's: with
    // it about k entries are published in all, without it tens of thousands)
    if (p.epochs) take_bound(p, ctl, true);
  }
  bsync();
  const uint64_t g = ctl->keep;
  const uint32_t gkey = (uint32_t)(g >> 32), glow = (uint32_t)g;
  uint32_t m = 0, v = 0;
#pragma unroll 4
  for (uint32_t j = t; j < n; j += kScanThreads) {
    const uint2 e = cand[j];
    m = max(m, e.x);
    v += e.x > gkey || (e.x == gkey && 0xFFFFFFFFu - e.y >= glow);
  }
  v = __reduce_add_sync(0xFFFFFFFFu, v);
  if (lane == 0) atomicAdd(&ctl->sel.valid, v);
  const bool exact = PART && p.k <= p.pub_exact;
  if (n > kPubMaxEntries && !exact) {
    if (lane < 4) keys[4 * warp + lane] = 0;
    __syncwarp();
    warp_top(m, 0u, 4u, lane, [&](uint32_t x, uint32_t key, uint32_t) { keys[4 * warp + x] = key; });
  }
  bsync();
  uint64_t limit = g, hid = 0;  // entries below the limit stay unpublished
  const bool many = ctl->sel.valid > kPubMaxEntries;
  if (exact && many) {
    bsync();  // every thread has `many` before the select writes its state
    list = cand + p.cap;  // the select's output area
    block_reduce<kScanThreads>(cand, n, list, p.k, gkey, hist, &ctl->sel);
  } else if (many) {
    const uint32_t x = __shfl_sync(0xFFFFFFFFu, warp_sort_desc<uint32_t>(keys[lane], lane), (int)p.pub_m - 1);
    if (x > gkey) limit = hid = (uint64_t)x << 32;  // (no entry below g belongs to the result)
  }
#pragma unroll 4
  for (uint32_t j = t; j < n && !(exact && many); j += kScanThreads) {
    const uint2 e = cand[j];
    if (composite(e.x, e.y) >= limit) {
      const uint32_t at = atomicAdd(&ctl->sel.wcount, 1u);
      if (at < kPubMaxEntries) list[at] = e;
    }
  }
  bsync();
  if (warp == 0) {
    const uint32_t most = exact && many ? p.k : kPubMaxEntries, c = min(ctl->sel.wcount, most);
    if (ctl->sel.wcount > most) hid = ~0ull;  // (equal keys at the limit)
    uint32_t base = 0;
    if (lane == 0) {
      if (c) base = atomicAdd(&sc->pub_n, c);
      if (hid) atomicMax(&sc->g_hid, (unsigned long long)hid);
    }
    base = __shfl_sync(0xFFFFFFFFu, base, 0);
    for (uint32_t j = lane; j < c; j += 32) p.pub[base + j] = list[j];
    __threadfence();
    __syncwarp();
    if (lane == 0) {
      atomicAdd(&sc->pub_arrived, 1u);
      const uint32_t gen0 = ctl->gen0;
      uint32_t gen = gen0;
      for (uint32_t it = 0; it < p.pub_wait && gen == gen0; ++it) {
        __nanosleep(kPubWaitNs);
        gen = ld_volatile_u32(&sc->gen);
      }
      if (gen == gen0) gen = atomicCAS(&sc->gen, gen0, gen0 | 1u);  // waited out: through the tree
      ctl->state = (gen == gen0 || gen == (gen0 | 1u)) ? kEndTree : kEndDone;
      __threadfence();  // a raised g_thr is read after the decision
    }
  }
  bsync();
  return ctl->state == kEndTree;
}

// The entries of comp[0..n) above `mine` (shared memory).
__device__ __forceinline__ uint32_t rank_of(const unsigned long long *comp, uint32_t n, unsigned long long mine) {
  uint32_t r = 0;
#pragma unroll 8
  for (uint32_t j = 0; j < n; ++j) r += comp[j] > mine;
  return r;
}

// The coordinator (block 0 of a launch with p.pub): scans nothing.  Per epoch, once every
// scanning CTA has published, it raises the global threshold to the k-th largest of the
// epoch's entries (k real objects reach that).  At the end it takes the k-th best
// published entry T: when g_hid <= T the published entries at or above T hold the result
// and it answers the query; else T's key becomes the global threshold and the merge tree
// answers.  A block of its own, because the CTA that arrives last -- the slowest --
// would be held up by this work in every epoch, and its code stays in the instruction
// cache from epoch to epoch.  Its waits are bounded; given up, the tree answers.
__device__ __noinline__ void coordinate(const ScanParams &p, SmemCtl *ctl, uint2 *buf, uint32_t *hist) {
  const int t = threadIdx.x;
  ScanScratch *sc = p.scratch;
  const uint32_t gen0 = ctl->gen0, ncta = gridDim.x - 1u;
  // its shared memory: keys or entries, then the linear bins
  uint32_t *stage = reinterpret_cast<uint32_t *>(buf);
  const uint32_t stage_cap = 2u * p.mcap - kLinBins;
  uint32_t *bins = stage + stage_cap;
  uint32_t epoch = 0;
  bool owner = false;  // thread 0: this block answered
#pragma unroll 1
  for (;;) {
    // wait for the epoch or the end, whichever is first
    if (t == 0) {
      uint32_t st = 2;  // given up, or decided by a CTA that waited out
      for (uint64_t it = 0; it < p.wait_limit; ++it) {
        const uint32_t ended = ld_volatile_u32(&sc->pub_arrived);
        const uint32_t ep = epoch < p.epochs ? ld_volatile_u32(&sc->epoch_arrived[epoch]) : 0u;
        if (ended == ncta) {
          st = 1;
          break;
        }
        if (ep == ncta) {
          st = 0;
          break;
        }
        if ((it & 15u) == 15u && ld_volatile_u32(&sc->gen) != gen0) break;
        __nanosleep(100);
      }
      ctl->state = st;
    }
    bsync();
    const uint32_t st = ctl->state;
    bsync();
    if (st == 2) {
      if (t == 0) atomicCAS(&sc->gen, gen0, gen0 | 1u);
      break;
    }
    __threadfence();
    if (st == 0) {
      const KthBound b = block_kth_bound<kScanThreads>(p.epub + (size_t)epoch * p.epub_stride, ncta * p.epoch_keys,
                                                       p.k, stage, stage_cap, bins, hist);
      if (t == 0) {
        if (b.key) {
          atomicMax(&sc->g_thr, b.key);
          atomicMax(&sc->g_keep, (unsigned long long)b.word());
          // in id order the rows that a CTA still has to scan when it sees this bound come
          // after every published one: they lose a tie with it
          atomicMax(&sc->g_app, b.key + (p.row_ids ? 0u : 1u));
        }
        if (epoch == 0) {
          __threadfence();
          atomicExch(&sc->epoch0_ready, 1u);
        }
      }
      ++epoch;
      continue;
    }
    if (p.tree_end) break;  // (nothing is decided: every CTA is on its way through the tree)
    const uint32_t np = ld_volatile_u32(&sc->pub_n);
    const uint64_t hid = ld_volatile_u64(&sc->g_hid);
    unsigned long long *comp = reinterpret_cast<unsigned long long *>(buf);
    const bool few = np <= kRankMax;  // ranked at once, no bound needed first
    KthBound b{0u, 0u, 0u};
    if (t == 0) {
      ctl->sel.wcount = 0;
      ctl->keep = 0;
    }
    bsync();
    if (few) {
      unsigned long long mine = 0ull;
      if (t < (int)np) {
        const uint2 e = __ldcg(p.pub + t);
        mine = composite(e.x, e.y);
        comp[t] = mine;
      }
      bsync();
      if (t < (int)np && rank_of(comp, np, mine) == p.k - 1u) ctl->keep = mine;  // the k-th
      bsync();
      b.key = (uint32_t)(ctl->keep >> 32);
      b.low = (uint32_t)ctl->keep;
    } else {
      b = block_kth_bound<kScanThreads>(p.pub, np, p.k, stage, stage_cap, bins, hist);
    }
    const uint64_t least = b.key ? b.word() : 0ull;
    // (an entry and its place in the order take 3 words; the select for many equal keys
    // below writes its k entries behind `cap`, and must not meet those it reads)
    const uint32_t room = min(stage_cap / 3u, p.cap);
    if (!few && hid != ~0ull) {  // the entries at or above the bound (no bound: all of them)
      for (uint32_t base = 0; base < np; base += kScanThreads * 8u) {  // uniform trip count
        uint2 e[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const uint32_t j = base + (uint32_t)u * kScanThreads + t;
          e[u] = j < np ? __ldcg(p.pub + j) : make_uint2(0u, 0xFFFFFFFFu);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const bool in = base + (uint32_t)u * kScanThreads + t < np && composite(e[u].x, e[u].y) >= least;
          const unsigned bal = __ballot_sync(0xFFFFFFFFu, in);
          if (!bal) continue;
          uint32_t at = 0;
          if ((t & 31) == 0) at = atomicAdd(&ctl->sel.wcount, (uint32_t)__popc(bal));
          at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(bal & ((1u << (t & 31)) - 1u));
          if (in && at < room) buf[at] = e[u];
        }
      }
      bsync();
    }
    const uint32_t cnt = few ? np : ctl->sel.wcount;
    const bool complete = hid != ~0ull && cnt <= room && (b.key ? hid <= least : hid == 0ull);
    if (!complete) {
      if (t == 0) {
        if (b.key) atomicMax(&sc->g_thr, b.key);
        __threadfence();
        atomicCAS(&sc->gen, gen0, gen0 | 1u);
      }
      break;
    }
    // (the answer is exact whoever decides: it is written while the decision is on its way)
    if (t == 0) owner = atomicCAS(&sc->gen, gen0, gen0 + 2u) == gen0;
    // rank every entry at or above the bound; the best k are the result, ascending
    const uint32_t res_n = min(cnt, p.k);
    auto emit = [&](uint32_t r, uint32_t key, uint32_t id) {
      if (r >= res_n) return;
      const uint32_t pos = res_n - 1u - r;
      p.out_ids[pos] = (uint64_t)id;
      p.out_scores[pos] = key2f(key);
      if (pos == 0 && p.out_threshold) *p.out_threshold = key2f(key);
    };
    if (cnt <= kRankMax) {  // by counting alone
      if (!few) {
        const uint2 e = t < (int)cnt ? buf[t] : make_uint2(0u, 0u);
        bsync();
        comp[t] = composite(e.x, e.y);
        bsync();
      }
      if (t < (int)cnt) {
        const unsigned long long mine = comp[t];
        emit(rank_of(comp, cnt, mine), (uint32_t)(mine >> 32), 0xFFFFFFFFu - (uint32_t)mine);
      }
    } else if (!block_rank_bins<kScanThreads>(buf, cnt, stage + 2u * cnt, bins, hist,
                                              [&](uint32_t r, uint2 e) { emit(r, e.x, e.y); })) {
      uint2 *res = buf, *selb = buf + p.cap;  // many equal keys
      if (cnt > p.k) {
        block_reduce<kScanThreads>(buf, cnt, selb, p.k, 0u, hist, &ctl->sel);
        res = selb;
      }
      block_sort_desc<kScanThreads>(res, res_n);
      for (uint32_t r = t; r < res_n; r += kScanThreads) emit(r, res[r].x, res[r].y);
    }
    bsync();
    if (t == 0) {
      if (!res_n && p.out_threshold) *p.out_threshold = 0.0f;
      write_stats(p, cnt, res_n);
    }
    break;
  }
  if (t != 0) return;
  if (owner) {
    reset_scratch(sc);
  } else {
    // through the tree: the later of this block and the tree's root resets the scratch
    __threadfence();
    if (atomicAdd(&sc->finishers, 1u) == 1u) {
      reset_scratch(sc);
      sc->gen = gen0 + 2u;
    }
  }
}

// QQ: compile-time attribute count (0 = runtime, any qq <= kMaxQ).  PART: partition
// mode (p.part_list set): tiles of listed partitions of a reordered copy.
template <int QQ, bool PART>
__global__ void __launch_bounds__(kScanThreads, scan_min_blocks<QQ, PART>())
    scan_select_kernel(const __grid_constant__ ScanParams p) {
  extern __shared__ __align__(1024) unsigned char smem[];
  SmemCtl *ctl = reinterpret_cast<SmemCtl *>(smem + kOffCtl);
  uint64_t *never = reinterpret_cast<uint64_t *>(smem + kOffNever);
  uint32_t *hist = reinterpret_cast<uint32_t *>(smem + kOffHist);
  float *wsm = reinterpret_cast<float *>(smem + kOffWsm);
  uint32_t *scnt = reinterpret_cast<uint32_t *>(smem + kOffScnt);
  // the candidate buffer (cap entries), then the select's output (the rest of mcap);
  // the merge reuses both
  uint2 *cand0 = reinterpret_cast<uint2 *>(smem + kOffCand);
  uint2 *selb = cand0 + p.cap;
  uint2 *mbuf = cand0;

  const int t = threadIdx.x;
  const int lane = t & 31;
  const uint32_t qq = QQ > 0 ? (uint32_t)QQ : p.qq;
  const uint32_t cap = p.cap;
  // scanning CTAs: all blocks, or all but block 0, the coordinator (p.pub)
  const uint32_t ncta = p.ncta, cta = blockIdx.x - (p.pub ? 1u : 0u);

  if (QQ == 0 && t < (int)kMaxQ && t < (int)qq) wsm[t] = p.w[t];
  if (t == 0) {
    mbar_init(never, 1);
    fence_barrier_init();
    ctl->count = 0;
    ctl->thr_local = 0;
    const uint32_t seed = max(p.thr_seed, p.thr_seed_dev ? *p.thr_seed_dev : 0u);
    if (seed) atomicMax(&p.scratch->g_thr, seed);  // every later read includes it
    // both slots hold a valid bound from the start: with two tiles per vote a thread
    // can read the second slot before thread 0's first copy into it
    ctl->thr_g[0] = ctl->thr_g[1] = max(ld_volatile_u32(&p.scratch->g_thr), seed);
    ctl->reductions = 0;
    // (without the tree's flag: a CTA may start after another one has waited out)
    ctl->gen0 = ld_volatile_u32(&p.scratch->gen) & ~1u;
    ctl->epoch0_seen = 0;
    ctl->keep = 0;
    ctl->epoch = 0;
    ctl->my_tiles = cta < p.num_tiles ? (p.num_tiles - cta + ncta - 1) / ncta : 0;
  }
  bsync();

  if (p.fault_mode == 1) {
    // Test hook: wait on a barrier that nothing arrives on.  The bounded wait runs
    // out and the scan reports a timeout; nothing else is in flight.
    const bool ok = mbar_wait_bounded(never, 0, p.wait_limit);
    if (__syncthreads_or(!ok)) {
      if (t == 0) atomicOr(&p.scratch->error, 1u);
      return;
    }
  }

  if (p.pub && blockIdx.x == 0) {
    coordinate(p, ctl, cand0, hist);
    return;
  }

  uint32_t g_pending = 0;  // thread 0's in-flight copy of the global threshold
  // next-tile prefetch: the loads of tile i + 1 are in flight while tile i is scored
  constexpr int kPQ = (QQ >= 1 && QQ <= kPrefetchQ) ? QQ : 1;
  constexpr bool prefetch = QQ >= 1 && QQ <= kPrefetchQ;
  // queried columns of the prefetching forms: read from the parameter block (colp), no
  // registers held
  // partition mode: the partitions (and bounds) of tiles i and i + 1 are known at the
  // start of tile i, the one of tile i + 2 is loaded during it
  const uint32_t pmask = (1u << p.part_shift) - 1u;
  uint32_t part_cur = 0, key_cur = 0xFFFFFFFFu, part_nx = 0, key_nx = 0xFFFFFFFFu;
  auto part_of = [&](uint32_t j, uint32_t &part, uint32_t &key) {
    const uint64_t x = ((uint64_t)cta + (uint64_t)j * ncta) >> p.part_shift;
    part = __ldg(p.part_list + x);
    if (p.part_key) key = __ldg(p.part_key + x);
  };
  if (PART) {
    if (ctl->my_tiles > 0) part_of(0, part_cur, key_cur);
    if (ctl->my_tiles > 1) part_of(1, part_nx, key_nx);
  }
  auto tile_row = [&](uint32_t j, uint32_t part) -> uint64_t {  // first row of tile j of this CTA
    const uint64_t tix = cta + (uint64_t)j * ncta;
    if constexpr (PART) return ((uint64_t)part << p.part_rows_log2) + (tix & pmask) * kTile;
    return p.tile_begin + tix * p.tile_step;
  };
  auto load_rows = [&](uint64_t tl, float4 *dst) {  // the tile that starts at row tl
    const float *c[kPQ];
#pragma unroll
    for (int m = 0; m < kPQ; ++m) c[m] = p.colp[m];
    load_cols<kPQ>(p, c, tl + (uint64_t)t * kVec, !(tl >= p.row_begin && tl + kTile <= p.row_end), dst);
  };
  // id order with prefetch: first row and index of the tile whose loads went out last;
  // tile j lies wholly inside [row_begin, row_end) iff j - int_lo < int_n (unsigned)
  uint64_t next_row = p.tile_begin + (uint64_t)cta * p.tile_step;
  uint32_t next_tix = cta;
  auto load_next = [&](float4 *dst) {
    const uint64_t r = next_row + (uint64_t)t * kVec;
    const bool inner = next_tix - p.int_lo < p.int_n;
    load_cols<kPQ>(p, p.colp, r, !inner, dst);
  };
  float4 xn[kPQ];
  // tiles between two select votes: 2 for q <= 2 in id order (a thread's work per tile
  // is small there and the vote's barrier was the top stall), 1 elsewhere; the buffer
  // has room for that many tiles above its select mark (plan_scan)
  constexpr uint32_t kVoteTiles = scan_vote_tiles(QQ, PART);
  uint32_t after = 0;  // fill after this thread's warp last appended, since the last vote
  // the tiles run in segments, each ended by a threshold epoch (the last by the end)
  uint32_t seg = 0, seg_len = p.epochs ? 1u : ctl->my_tiles;  // the segment's first tile and length
  // q <= 2 in id order: two tiles per loop pass, so the prefetched registers swap roles
  // instead of being copied (q = 2 on 2^28 rows: 0.420 -> 0.406 ms)
  constexpr int kUnroll = kVoteTiles == 2 ? 2 : 1;
  bool stopped = false;
  for (;;) {
    // the segment's first loads; in id order its last tile prefetches nothing, so the
    // epoch's code holds no loads in flight in registers (partition mode has the registers)
    if (prefetch && seg_len) {
      if constexpr (PART) {
        if (seg == 0) load_rows(tile_row(0, part_cur), xn);
      } else {
        next_row = p.tile_begin + ((uint64_t)cta + (uint64_t)seg * ncta) * p.tile_step;
        next_tix = cta + seg * ncta;
        load_next(xn);
      }
    }
    // i: the tile of the segment (base + i the CTA's), above eight columns the CTA's: one
    // value less beside the loads (2^28 rows, q = 14: 2183 us with base, 2150 without; at
    // q = 1, where the loop is unrolled, 426 with, 458 without)
    constexpr bool kAbs = !PART && QQ > 8;
    const uint32_t base = kAbs ? 0u : seg, end = kAbs ? seg + seg_len : seg_len;
    uint32_t i = kAbs ? seg : 0u;
    // two tiles per vote: after every odd one, and in the second segment, which starts at
    // tile 1, after every even one -- no more than two tiles ever meet an unvoted buffer
    const uint32_t vote_at = seg == 1u ? 0u : 1u;
#pragma unroll(kUnroll)
    for (; i < end; ++i) {
      // every thread reads the same thresholds in tile i (see SmemCtl::thr_g); in id
      // order they are read after the scores, so they hold no register across the loads
      uint32_t thr = 0;
      if constexpr (PART) {
        thr = max(ctl->thr_local, ctl->thr_g[i & 1u]);
        // nothing in this partition (nor in any later one of this CTA) can reach thr
        if (key_cur < thr) {
          stopped = true;
          break;
        }
      }
      const uint64_t tile0 = (prefetch && !PART) ? next_row : tile_row(base + i, part_cur);
      const uint64_t row0 = tile0 + (uint64_t)t * kVec;
      const bool interior = (prefetch && !PART) ? next_tix - p.int_lo < p.int_n
                                                : tile0 >= p.row_begin && tile0 + kTile <= p.row_end;  // uniform
      float4 s;
      if (prefetch) {
        float4 x[kPQ];
#pragma unroll
        for (int m = 0; m < kPQ; ++m) x[m] = xn[m];
        if constexpr (PART) {
          if (base + i + 1 < ctl->my_tiles) load_rows(tile_row(base + i + 1, part_nx), xn);
        } else if (i + 1 < end) {
          next_row += p.grid_rows;
          next_tix += ncta;
          load_next(xn);
        }
        s = score_cols<kPQ>(p, x);
      } else {
        s = score4<QQ>(p, wsm, qq, row0, !interior);
      }
      if constexpr (PART) {
        part_cur = part_nx;
        key_cur = key_nx;
        if (base + i + 2 < ctl->my_tiles) part_of(base + i + 2, part_nx, key_nx);
      }

      if constexpr (!PART) thr = max(ctl->thr_local, ctl->thr_g[i & 1u]);
      // key(score) >= thr  <=>  thr == 0 (everything, NaN included) or score >= thr_float(thr)
      const bool take_all = thr == 0u;
      const float thr_f = thr_float(thr);
      const float sv[4] = {s.x, s.y, s.z, s.w};
      unsigned pass_mask = 0;
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        bool pv = take_all || sv[v] >= thr_f;
        if (!interior) pv = pv && row0 + v >= p.row_begin && row0 + v < p.row_end;
        pass_mask |= (unsigned)pv << v;
      }
      // `after` = fill after this warp's append.  The warp that appends last before a
      // vote sees the final count, so OR-voting "after > cap - kVoteTiles * TILE" at the
      // barrier gives every thread the same reduce decision.  (Reading ctl->count after
      // a barrier would not: a fast warp may already be appending the next tile.)
      if (__ballot_sync(0xFFFFFFFFu, pass_mask != 0u)) {  // warp-uniform: some lane passed
        uint2 *cand = cand0;
        const uint32_t npass = __popc(pass_mask);
        uint32_t incl = npass;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
          if (lane >= o) incl += y;
        }
        const uint32_t wtotal = __shfl_sync(0xFFFFFFFFu, incl, 31);
        uint32_t base = 0;
        if (lane == 31) base = atomicAdd(&ctl->count, wtotal);
        base = __shfl_sync(0xFFFFFFFFu, base, 31);
        after = base + wtotal;
        base += incl - npass;
#pragma unroll
        for (int v = 0; v < 4; ++v)
          if (pass_mask & (1u << v)) {
            if (TOPK_CHECK(base < cap, kDiagAppend, i, base, cap))
              cand[base] = make_uint2(f2key(sv[v]), p.row_ids ? __ldg(p.row_ids + row0 + v) : (uint32_t)(row0 + v));
            ++base;
          }
      }
      // thread 0 hands the CTA its copy of the global threshold (see SmemCtl::thr_g): it
      // loads the global word every 4 tiles (8 where a tile is more than eight columns) and
      // applies it on the last of them, so the L2 round trip is never waited on (every 2 and
      // on the next in partition mode, where it ends the scan).  The new value goes to the
      // slot the next tile reads, and on the tile after into the other slot too; between
      // updates both slots agree.  One word: the larger of two would be waited for here, and
      // every warp with it at the vote (2^28 rows, q = 14, k = 16: 2183 us so, 2135 now).
      constexpr uint32_t kPoll = PART ? 1u : (QQ == 0 || QQ > 8) ? 7u : 3u;
      if (t == 0) {
        if ((i & kPoll) == kPoll) ctl->thr_g[(i + 1u) & 1u] = max(ctl->thr_g[i & 1u], g_pending);
        if ((i & kPoll) == 0u) {
          ctl->thr_g[(i + 1u) & 1u] = ctl->thr_g[i & 1u];
          g_pending = ld_volatile_u32(&p.scratch->g_app);
        }
      }
      // (uniform: every thread takes the same votes; the scan's end needs no room)
      if (kVoteTiles > 1 && (i & 1u) != vote_at) continue;
      const bool full = __syncthreads_or(after > cap - kVoteTiles * kTile);
      after = 0;
      if (full && base + i + 1 < ctl->my_tiles) {
        if (t == 0) {
          // the first fill may come before any bound: epoch 0's is on its way, and dropping
          // what lies below it costs one pass over the buffer instead of a select
          take_bound(p, ctl, ctl->keep == 0ull);
          ctl->sel.wcount = 0;
        }
        bsync();
        // what lies below the bound out of the buffer, in place; a select when much is left
        const uint32_t left = block_compact<kScanThreads>(cand0, ctl->count, ctl->keep, &ctl->sel);
        if (left <= (cap - kVoteTiles * kTile) / 2u) {
          if (t == 0) ctl->count = left;
          bsync();
          continue;
        }
        // the best k into the output area, then back to the front of the buffer
        const uint32_t kept = block_reduce<kScanThreads>(cand0, left, selb, p.k, 0u, hist, &ctl->sel);
        for (uint32_t j = t; j < kept; j += kScanThreads) cand0[j] = selb[j];
        if (t == 0) {
          ctl->count = kept;
          ctl->reductions++;
          if (kept == p.k) {  // the CTA knows a k-th key
            // Rows in id order: a later row has a larger id and loses a tie with the
            // k-th, so it must beat it strictly.  Rows carrying their own ids (a
            // reordered copy) may win the tie: the threshold stays inclusive.
            ctl->thr_local = ctl->sel.kept_min + (p.row_ids ? 0u : 1u);
            atomicMax(&p.scratch->g_thr, ctl->sel.kept_min);
            atomicMax(&p.scratch->g_app, ctl->sel.kept_min);
          }
        }
        bsync();
      }
    }
    seg = base + i;
    // (a CTA that a seed stopped before epoch 0 arrives there all the same: others wait for it)
    if (ctl->epoch >= p.epochs || (stopped && ctl->epoch != 0u)) break;
    epoch_publish(p, cand0, ctl, hist);
    if (stopped) break;
    if (PART && p.epoch_hold && ctl->epoch == 1u) {  // (a small copy: few tiles to stop before)
      if (t == 0) take_bound(p, ctl, true);
      bsync();
    }
    seg_len = (ctl->epoch < p.epochs ? seg << p.epoch_shift : ctl->my_tiles) - seg;
  }

  // ---- end of scan ----
  bsync();
  if (t == 0 && ctl->reductions) atomicAdd(&p.scratch->acc_reductions, ctl->reductions);
  if (PART && t == 0) atomicAdd(&p.scratch->acc_tiles, seg);

  if (p.pub && !publish_entries<PART>(p, cand0, ctl, hist)) return;

  // ---- merge tree: this CTA's best k first ----
  if (t == 0) {
    ctl->red_g = ld_volatile_u32(&p.scratch->g_thr);
    ctl->reductions = 0;
  }
  bsync();
  if (ctl->count > p.k) {
    const uint32_t kept = block_reduce<kScanThreads>(cand0, ctl->count, selb, p.k, ctl->red_g, hist, &ctl->sel);
    for (uint32_t j = t; j < kept; j += kScanThreads) cand0[j] = selb[j];
    if (t == 0) {
      ctl->count = kept;
      atomicAdd(&p.scratch->acc_reductions, 1u);
      if (kept == p.k) atomicMax(&p.scratch->g_thr, ctl->sel.kept_min);
    }
    bsync();
  }

  const uint32_t k = p.k;
  uint2 *res = cand0;
  uint32_t res_n = ctl->count;
  uint32_t level = 0, slot = cta, merged = res_n;
  uint32_t kpad = 1;  // k rounded up to a power of two: the kept entries and the sort's padding
  while (kpad < k) kpad <<= 1;
  uint2 *outb = mbuf + (p.mcap - kpad);
  while (p.nslots[level] > 1) {
    // publish my result into slot (level, slot), filtered by the current threshold
    if (t == 0) {
      ctl->red_g = ld_volatile_u32(&p.scratch->g_thr);
      ctl->sel.wcount = 0;
    }
    bsync();
    {
      const uint32_t g = ctl->red_g;
      uint2 *dst = p.slots + (size_t)(p.slot_off[level] + slot) * k;
      for (uint32_t j = t; j < res_n; j += kScanThreads) {
        const uint2 e = res[j];
        if (e.x >= g) dst[atomicAdd(&ctl->sel.wcount, 1u)] = e;  // <= res_n <= k entries
      }
    }
    __threadfence();  // each writer makes its slot entries visible device-wide
    bsync();
    const uint32_t grp = slot / p.fanin;
    const uint32_t first = grp * p.fanin;
    const uint32_t gsize = min(p.fanin, p.nslots[level] - first);
    if (t == 0) {
      p.slot_count[p.slot_off[level] + slot] = ctl->sel.wcount;
      __threadfence();
      const uint32_t arrived = atomicAdd(&p.done[p.done_off[level] + grp], 1u);
      ctl->is_last = (arrived == gsize - 1u) ? 1u : 0u;
      if (ctl->is_last) p.done[p.done_off[level] + grp] = 0u;  // every arrival is in: reset
    }
    bsync();
    if (!ctl->is_last) return;
    __threadfence();
    // the last arrival merges the group's slots: their counts first, then all their
    // entries as one flat index space, kMergeBatch loads per thread in flight at a
    // time, in chunks that fit the shared input area; the best k so far (in `outb`)
    // open each chunk after the first
    if (t == 0) ctl->red_g = ld_volatile_u32(&p.scratch->g_thr);
    if (t < (int)gsize) scnt[t] = __ldcg(&p.slot_count[p.slot_off[level] + first + t]);
    bsync();
    {
      const uint32_t g = ctl->red_g;
      const uint32_t in_cap = p.mcap - kpad;  // input area [0, in_cap), outb after it
      uint32_t total = 0;
      for (uint32_t si = 0; si < gsize; ++si) total += scnt[si];
      uint32_t kept = 0, done = 0;
      merged = 0;
      do {
        for (uint32_t j = t; j < kept; j += kScanThreads) mbuf[j] = outb[j];
        if (t == 0) ctl->sel.wcount = kept;
        bsync();
        const uint32_t n_load = min(total - done, in_cap - kept);
        constexpr int kMergeBatch = 2;
        for (uint32_t base = 0; base < n_load; base += kScanThreads * kMergeBatch) {
          uint2 e[kMergeBatch];
#pragma unroll
          for (int u = 0; u < kMergeBatch; ++u) {
            const uint32_t j = base + (uint32_t)u * kScanThreads + t;
            e[u] = make_uint2(0u, 0u);
            if (j < n_load) {
              uint32_t f = done + j, si = 0;
              while (f >= scnt[si]) f -= scnt[si++];  // done + j < total: ends inside a slot
              e[u] = __ldcg(p.slots + (size_t)(p.slot_off[level] + first + si) * k + f);
            }
          }
#pragma unroll
          for (int u = 0; u < kMergeBatch; ++u) {
            if (base + (uint32_t)u * kScanThreads + t < n_load && e[u].x >= g) {
              const uint32_t pos = atomicAdd(&ctl->sel.wcount, 1u);
              if (TOPK_CHECK(pos < in_cap, kDiagMerge, level, pos, in_cap)) mbuf[pos] = e[u];
            }
          }
        }
        bsync();
        const uint32_t loaded = min(ctl->sel.wcount, in_cap);
        bsync();  // every thread has `loaded` before block_reduce resets wcount
        merged += loaded - kept;
        kept = block_reduce<kScanThreads>(mbuf, loaded, outb, k, 0u, hist, &ctl->sel);
        done += n_load;
      } while (done < total);
      res_n = kept;
    }
    res = outb;
    level += 1;
    slot = grp;
  }

  // ---- root: sort and write the result (res has room for the padding) ----
  block_sort_desc<kScanThreads>(res, res_n);
  write_sorted(p, res, res_n, merged);
  if (t == 0) {
    // with a coordinator, the later of it and this CTA resets the scratch (no CTA waits for
    // the decision any more: each has published a slot)
    bool last = true;
    if (p.pub) {
      __threadfence();
      last = atomicAdd(&p.scratch->finishers, 1u) == 1u;
    }
    if (last) {
      reset_scratch(p.scratch);
      if (p.pub) p.scratch->gen = ctl->gen0 + 2u;
    }
  }
}

using ScanKernel = void (*)(ScanParams);

// [part][q] for q = 1..16; [..][0] is the runtime-q kernel used for q > 16
#define TOPK_SCAN_ROW(P)                                                                                        \
  {scan_select_kernel<0, P>,  scan_select_kernel<1, P>,  scan_select_kernel<2, P>,  scan_select_kernel<3, P>,   \
   scan_select_kernel<4, P>,  scan_select_kernel<5, P>,  scan_select_kernel<6, P>,  scan_select_kernel<7, P>,   \
   scan_select_kernel<8, P>,  scan_select_kernel<9, P>,  scan_select_kernel<10, P>, scan_select_kernel<11, P>,  \
   scan_select_kernel<12, P>, scan_select_kernel<13, P>, scan_select_kernel<14, P>, scan_select_kernel<15, P>,  \
   scan_select_kernel<16, P>}
const ScanKernel kKernels[2][17] = {TOPK_SCAN_ROW(false), TOPK_SCAN_ROW(true)};
#undef TOPK_SCAN_ROW

ScanKernel kernel_for(uint32_t qq, bool part) { return kKernels[part ? 1 : 0][qq <= 16 ? qq : 0]; }

}  // namespace

cudaError_t scan_set_attributes(size_t smem_optin) {
  for (const auto &row : kKernels)
    for (ScanKernel f : row) {
      const cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void *>(f),
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_optin);
      if (e != cudaSuccess) return e;
    }
  return cudaSuccess;
}

namespace {

// Shared memory of an SM that the unified L1 / shared memory can give (B200: 228 KB),
// the L1 the scan keeps (its 128-bit loads land in L1 while in flight: with less, the
// loads in flight per SM, and the bandwidth, shrink), and the per-CTA reserve.
constexpr size_t kSmemPerSm = 228 * 1024;
constexpr size_t kScanL1Keep = 60 * 1024;
constexpr size_t kSmemPerCtaReserve = 1024;

// The shared-memory carveout last set on each scan kernel, per device (the attribute
// is per function and device; setting it again costs a driver call).
std::mutex g_carveout_mu;
int g_carveout[64][2][17];

void set_carveout(const void *fn, bool part, uint32_t qq, int percent) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return;
  std::lock_guard<std::mutex> lk(g_carveout_mu);
  int &cur = g_carveout[dev][part ? 1 : 0][qq <= 16 ? qq : 0];
  if (cur == percent + 1) return;  // stored plus one: 0 means not set yet
  if (cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, percent) == cudaSuccess)
    cur = percent + 1;
  else
    (void)cudaGetLastError();
}

}  // namespace

namespace {

// Plans by (device, q, k, partition mode, CTA cap): the occupancy queries behind a plan
// are driver calls, a few microseconds each, on every query's critical path otherwise.
struct PlanEntry {
  ScanPlan pl;
  int carveout;
};
std::mutex g_plan_mu;
std::map<std::tuple<int, uint32_t, uint32_t, bool, uint32_t>, PlanEntry> g_plans;

}  // namespace

ScanPlan plan_scan(uint32_t qq, uint32_t k, uint64_t rows, int num_sms, size_t smem_optin, uint32_t max_ctas_per_sm,
                   bool part) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    (void)cudaGetLastError();
    dev = -1;
  }
  const auto key = std::make_tuple(dev, qq <= 16 ? qq : 0u, k, part, max_ctas_per_sm);
  const void *fn = reinterpret_cast<const void *>(kernel_for(qq, part));
  const uint64_t tiles = (rows + 3 + kTile) / kTile;
  auto finish = [&](ScanPlan pl) {
    uint64_t grid = (uint64_t)num_sms * (uint64_t)pl.ctas_per_sm - 1u;  // one place for the coordinator
    if (grid > tiles) grid = tiles;
    if (grid < 1) grid = 1;
    pl.grid = (int)grid;
    return pl;
  };
  {
    std::lock_guard<std::mutex> lk(g_plan_mu);
    const auto it = g_plans.find(key);
    if (it != g_plans.end()) {
      const PlanEntry pe = it->second;
      // the carveout is per function: another plan may have changed it since
      set_carveout(fn, part, qq, pe.carveout);
      return finish(pe.pl);
    }
  }
  ScanPlan pl{};
  pl.tile = kTile;
  uint32_t P = 1;
  while (P < k) P <<= 1;
  // after a select the buffer holds <= k entries; kVoteTiles tiles add <= that many times
  // kTile, and a select runs once the fill exceeds cap - kVoteTiles * kTile
  // (plus half a tile of slack when every tile votes; with two tiles per vote the
  // rounding below leaves some, and more would cost q <= 2 a CTA per SM)
  const uint32_t vote_tiles = scan_vote_tiles(qq <= 16 ? (int)qq : 0, part);
  uint32_t cap = k + vote_tiles * kTile + (vote_tiles == 1 ? kTile / 2 : 0u);
  // partition mode: room for two tiles more, so that no CTA waits for epoch 0's bound with a
  // full buffer (its few CTAs per SM leave the shared memory)
  if (part) cap += 2 * kTile;
  if (cap < P) cap = P;
  if (cap < 2048) cap = 2048;
  cap = (cap + kScanThreads - 1) / kScanThreads * kScanThreads;
  pl.cap = cap;
  // the select writes <= k entries (padded to P for the sort) after the buffer; the
  // merge reuses both, its input in chunks of up to cap entries, so the fan-in is not
  // bound by it: G = what two buffers of cap would hold, 4 to kMaxFanin
  uint32_t mcap = cap + P;
  uint32_t G = (2 * cap - P) / k;
  if (G > kMaxFanin) G = kMaxFanin;
  if (G < 4) G = 4;
  pl.fanin = G;
  pl.mcap = mcap;
  pl.smem = kScanSmemFixed + (size_t)mcap * 8;
  pl.stages = pl.smem <= smem_optin ? 1u : 0u;
  // CTAs per SM: as many as registers and threads allow, and as the shared memory
  // allows with kScanL1Keep left as L1 (or the caller's number); the carveout is set to
  // just fit them, so the rest of the unified memory stays L1
  set_carveout(fn, part, qq, 100);
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, kScanThreads, pl.smem) != cudaSuccess || occ < 1) {
    (void)cudaGetLastError();
    occ = 1;
  }
  const size_t per_cta = pl.smem + kSmemPerCtaReserve;
  const int by_l1 = (int)std::max<size_t>(1, (kSmemPerSm - kScanL1Keep) / per_cta);
  if (max_ctas_per_sm >= 1) occ = std::min<int>(occ, (int)max_ctas_per_sm);
  else occ = std::min(occ, by_l1);
  // the smallest shared-memory size of the SM (KB) that holds them, as a percentage
  static const size_t kSizesKb[] = {0, 8, 16, 32, 64, 100, 132, 164, 196, 228};
  size_t want = per_cta * (size_t)occ, size_kb = 228;
  for (size_t kb : kSizesKb)
    if (kb * 1024 >= want) {
      size_kb = kb;
      break;
    }
  const int carveout = (int)((size_kb * 100 + 227) / 228);
  set_carveout(fn, part, qq, carveout);
  int fit = 0;  // what the driver reports with that preference
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, fn, kScanThreads, pl.smem) == cudaSuccess && fit >= 1)
    occ = std::min(occ, fit);
  else
    (void)cudaGetLastError();
  pl.ctas_per_sm = occ;
  if (dev >= 0) {
    std::lock_guard<std::mutex> lk(g_plan_mu);
    g_plans[key] = PlanEntry{pl, carveout};
  }
  return finish(pl);
}

void plan_merge_tree(ScanParams &p, uint32_t grid, uint32_t fanin, uint32_t *total_slots, uint32_t *total_groups) {
  uint32_t l = 0, soff = 0, doff = 0;
  p.nslots[0] = grid;
  while (p.nslots[l] > 1 && l + 1 < (uint32_t)kMaxLevels) {
    const uint32_t groups = (p.nslots[l] + fanin - 1) / fanin;
    p.slot_off[l] = soff;
    p.done_off[l] = doff;
    soff += p.nslots[l];
    doff += groups;
    p.nslots[l + 1] = groups;
    ++l;
  }
  p.slot_off[l] = soff;
  p.done_off[l] = doff;
  p.levels = l;
  p.fanin = fanin;
  *total_slots = soff;
  *total_groups = doff;
}

cudaError_t launch_scan(const ScanPlan &pl, const ScanParams &p, cudaStream_t stream) {
  if (pl.stages < 1) return cudaErrorInvalidValue;
  ScanParams q = p;
  for (uint32_t m = 0; m < 4; ++m) q.colp[m] = m < p.qq ? p.table + (uint64_t)p.attr[m] * p.ld : p.table;
  q.ncta = (uint32_t)pl.grid;
  q.grid_rows = (uint64_t)pl.grid * p.tile_step;
  // id order: tiles [int_lo, int_lo + int_n) lie wholly inside [row_begin, row_end)
  q.int_lo = p.tile_begin < p.row_begin ? 1u : 0u;
  uint64_t hi = 0;
  if (p.row_end >= p.tile_begin + kTile) hi = (p.row_end - p.tile_begin - kTile) / p.tile_step + 1;
  if (hi > p.num_tiles) hi = p.num_tiles;
  q.int_n = hi > q.int_lo ? (uint32_t)(hi - q.int_lo) : 0u;
  const int grid = pl.grid + (p.pub ? 1 : 0);  // and the coordinator
  kernel_for(p.qq, p.part_list != nullptr)<<<grid, kScanThreads, pl.smem, stream>>>(q);
  return cudaGetLastError();
}

}  // namespace topk
