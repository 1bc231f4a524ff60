// Block-wide exact selection on (key, id) candidate entries, shared by the fused
// single-query scan and the batched kernels.
//
// An entry is uint2{key, id}: key = order-preserving image of an FP32 score
// (NaN -> 0), id = object id.  Selection order = the 64-bit word key<<32 | ~id
// (higher score first, then lower id), so every entry is distinct and "the best k"
// is always exactly k entries.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "device_common.cuh"

namespace topk {

// Shared-memory state of one block's select (48 bytes, 8-byte aligned).
struct SelShared {
  uint32_t digit, above, eq;  // radix-select pass result
  uint32_t valid;             // entries with key >= min_key
  uint32_t wcount;            // compaction cursor
  uint32_t kept_min;          // min key among the kept entries
  uint32_t pad[2];
  unsigned long long mm[2];   // min / max composite of a select
};

struct SmemSrc {
  const uint2 *p;
  __device__ uint2 operator()(uint32_t j) const { return p[j]; }
};

// Block-wide radix select over `count` entries of `src` with key >= min_key: finds
// (prefix, mask) such that exactly `need` valid entries satisfy
// (composite & mask) >= prefix.  Requires need <= number of valid entries.
// Digits are taken from the highest bit where the valid entries differ (min/max of
// the composites first), 8 bits at a time; histogram updates are aggregated per
// warp with __match_any_sync, because candidates crowd into few bins.  `count`
// must be the same in every thread; `hist` holds 256 bins.
template <int NT, class Src>
__device__ void block_radix_select(const Src &src, uint32_t count, uint32_t min_key, uint32_t need,
                                   uint32_t *hist, SelShared *sh, uint64_t &prefix_out, uint64_t &mask_out) {
  static_assert(NT % 32 == 0 && NT >= 32, "whole warps");
  const int t = threadIdx.x;
  const int lane = t & 31;
  if (t == 0) {
    sh->mm[0] = ~0ull;
    sh->mm[1] = 0ull;
  }
  __syncthreads();
  {
    unsigned long long lo = ~0ull, hi = 0ull;
    for (uint32_t j = t; j < count; j += NT) {
      const uint2 e = src(j);
      if (e.x < min_key) continue;
      const unsigned long long c = composite(e.x, e.y);
      lo = c < lo ? c : lo;
      hi = c > hi ? c : hi;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long a = __shfl_xor_sync(0xFFFFFFFFu, lo, o);
      const unsigned long long b = __shfl_xor_sync(0xFFFFFFFFu, hi, o);
      lo = a < lo ? a : lo;
      hi = b > hi ? b : hi;
    }
    if (lane == 0) {
      atomicMin(&sh->mm[0], lo);
      atomicMax(&sh->mm[1], hi);
    }
  }
  __syncthreads();
  const uint64_t cmin = sh->mm[0], cmax = sh->mm[1];
  const uint64_t diff = cmin ^ cmax;
  int hib = diff ? 63 - __clzll((long long)diff) : -1;  // highest differing bit
  uint64_t mask = hib >= 63 ? 0ull : (~0ull << (hib + 1));
  uint64_t prefix = cmin & mask;
  while (hib >= 0) {
    const int lob = hib >= 7 ? hib - 7 : 0;
    const uint32_t dmask = (1u << (hib - lob + 1)) - 1u;
    for (int b = t; b < 256; b += NT) hist[b] = 0;
    __syncthreads();
    for (uint32_t base = 0; base < count; base += NT) {  // uniform trip count
      const uint32_t j = base + t;
      uint32_t bin = 0xFFFFFFFFu;
      if (j < count) {
        const uint2 e = src(j);
        if (e.x >= min_key) {
          const uint64_t c = composite(e.x, e.y);
          if ((c & mask) == prefix) bin = (uint32_t)(c >> lob) & dmask;
        }
      }
      if (!__any_sync(0xFFFFFFFFu, bin != 0xFFFFFFFFu)) continue;  // warp-uniform: nothing to count
      const unsigned peers = __match_any_sync(0xFFFFFFFFu, bin);
      if (bin != 0xFFFFFFFFu && lane == __ffs(peers) - 1) atomicAdd(&hist[bin], (uint32_t)__popc(peers));
    }
    __syncthreads();
    if (t < 32) {
      // lane l owns bins [255-8l-7, 255-8l], visited from high to low
      const int top = 255 - 8 * t;
      uint32_t local[8];
      uint32_t s = 0;
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        local[b] = hist[top - b];
        s += local[b];
      }
      uint32_t incl = s;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (t >= o) incl += v;
      }
      const uint32_t excl = incl - s;
      if (excl < need && need <= incl) {
        uint32_t run = excl;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
          if (run + local[b] >= need) {
            sh->digit = (uint32_t)(top - b);
            sh->above = run;
            sh->eq = local[b];
            break;
          }
          run += local[b];
        }
      }
    }
    __syncthreads();
    const uint32_t digit = sh->digit, above = sh->above, eq = sh->eq;
    __syncthreads();  // everyone has read the result before the next pass rewrites it
    need -= above;
    prefix |= (uint64_t)digit << lob;
    mask |= (uint64_t)dmask << lob;
    if (eq == need) break;
    hib = lob - 1;
  }
  prefix_out = prefix;
  mask_out = mask;
}

// Keep the best k entries with key >= min_key of src[0..count), written to dst
// (out of place; dst must not overlap src).  Returns the number kept (the same in
// every thread); sh->kept_min gets their min key.
template <int NT>
__device__ uint32_t block_reduce(const uint2 *src, uint32_t count, uint2 *dst, uint32_t k, uint32_t min_key,
                                 uint32_t *hist, SelShared *sh) {
  const int t = threadIdx.x;
  uint32_t v = 0;
  for (uint32_t j = t; j < count; j += NT) v += (src[j].x >= min_key);
  v = warp_sum_u32(v);
  if (t == 0) {
    sh->valid = 0;
    sh->wcount = 0;
    sh->kept_min = 0xFFFFFFFFu;
  }
  __syncthreads();
  if ((t & 31) == 0) atomicAdd(&sh->valid, v);
  __syncthreads();
  const uint32_t valid = sh->valid;
  uint64_t prefix = 0, mask = 0;
  const bool select = valid > k;
  if (select) block_radix_select<NT>(SmemSrc{src}, count, min_key, k, hist, sh, prefix, mask);
  uint32_t kmin = 0xFFFFFFFFu;
  for (uint32_t base = 0; base < count; base += NT) {  // uniform trip count
    const uint32_t j = base + t;
    uint2 e = make_uint2(0u, 0u);
    bool keep = false;
    if (j < count) {
      e = src[j];
      keep = e.x >= min_key && (!select || (composite(e.x, e.y) & mask) >= prefix);
    }
    const unsigned bal = __ballot_sync(0xFFFFFFFFu, keep);
    uint32_t pos = 0;
    if ((t & 31) == 0 && bal) pos = atomicAdd(&sh->wcount, (uint32_t)__popc(bal));
    pos = __shfl_sync(0xFFFFFFFFu, pos, 0);
    if (keep) {
      dst[pos + __popc(bal & ((1u << (t & 31)) - 1u))] = e;
      kmin = min(kmin, e.x);
    }
  }
  kmin = warp_min_u32(kmin);
  if ((t & 31) == 0) atomicMin(&sh->kept_min, kmin);
  __syncthreads();
  const uint32_t kept = sh->wcount;
  __syncthreads();  // every thread has its copy before thread 0 may reset wcount
  return kept;
}

// Drop the entries below the composite `least` from buf[0..n), in place; returns how many are left
// (the same in every thread).  sh->wcount must be 0.  1024 entries at a time: read into
// registers, then written at the front, which never passes the entries still to be read.
template <int NT>
__device__ uint32_t block_compact(uint2 *buf, uint32_t n, uint64_t least, SelShared *sh) {
  constexpr int kPer = 4;
  const int t = threadIdx.x;
#pragma unroll 1
  for (uint32_t base = 0; base < n; base += NT * kPer) {
    uint2 e[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const uint32_t j = base + (uint32_t)u * NT + t;
      e[u] = j < n ? buf[j] : make_uint2(0u, 0u);
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const bool keep = base + (uint32_t)u * NT + t < n && composite(e[u].x, e[u].y) >= least;
      const unsigned bal = __ballot_sync(0xFFFFFFFFu, keep);
      uint32_t pos = 0;
      if ((t & 31) == 0 && bal) pos = atomicAdd(&sh->wcount, (uint32_t)__popc(bal));
      pos = __shfl_sync(0xFFFFFFFFu, pos, 0);
      if (keep) buf[pos + __popc(bal & ((1u << (t & 31)) - 1u))] = e[u];
    }
  }
  __syncthreads();
  const uint32_t left = sh->wcount;
  __syncthreads();  // every thread has its copy before thread 0 may reset wcount
  return left;
}

// The 32 words of a warp, descending across its lanes (bitonic).
template <class W>
__device__ __forceinline__ W warp_sort_desc(W v, int lane) {
#pragma unroll
  for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      const W o = __shfl_xor_sync(0xFFFFFFFFu, v, stride);
      v = (((lane & size) == 0) == ((lane & stride) == 0)) == (o > v) ? o : v;
    }
  return v;
}

// Bins of the linear histograms below, and what one level costs: about five block
// barriers, whatever the number of keys -- a digit-wise select pays those per 8 bits, and
// a barrier phase of a nearly idle SM takes 0.2-0.4 us.
constexpr uint32_t kLinBins = 2048;

// Of the bins [0, kLinBins), highest first: the bin in which the running count (from
// `above`) reaches k.  hist[11] = the bin, hist[12] = the count above it, hist[13] = its
// own.  With `scan` each bin is left holding the count above it instead of its own.
template <int NT>
__device__ __forceinline__ void bins_find(uint32_t *bins, uint32_t above, uint32_t k, uint32_t *hist, bool scan) {
  static_assert(kLinBins == 8 * NT, "eight bins per thread");
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  uint32_t *mine = bins + (kLinBins - 8u - 8u * (uint32_t)t);  // thread 0 owns the highest eight
  uint32_t c[8], sum = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    c[i] = mine[i];
    sum += c[i];
  }
  uint32_t incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) hist[warp] = incl;
  __syncthreads();
  uint32_t run = above + incl - sum;
  for (int w = 0; w < warp; ++w) run += hist[w];
#pragma unroll
  for (int i = 7; i >= 0; --i) {
    if (run < k && k <= run + c[i]) {
      hist[11] = (uint32_t)(mine - bins) + (uint32_t)i;
      hist[12] = run;
      hist[13] = c[i];
    }
    if (scan) mine[i] = run;
    run += c[i];
  }
  __syncthreads();
}

// A lower bound of the k-th best of the entries src[j] = (key, id), j < np, in global
// memory (key 0: not an entry), with at most k + k / 4 + 32 entries at or above it: a key
// and, where too many entries share that key, a lower bound of ~id among them (else 0).
// key 0 when fewer than k entries were read (past NT * kKthRegs + stage_cap of them the
// rest is left out, which only lowers the bound; count = those read at or above it).  Linear bins between the smallest and the largest value, and
// again inside the bin of the k-th when that is too full, over the keys and then over the
// ~ids.  Values sit in registers (kKthRegs per thread) and, past those, in `stage`.
struct KthBound {
  uint32_t key, low, count;
  __device__ uint64_t word() const { return ((uint64_t)key << 32) | low; }
};
constexpr int kKthRegs = 16;
template <int NT>
__device__ __noinline__ KthBound block_kth_bound(const uint2 *src, uint32_t np, uint32_t k, uint32_t *stage,
                                                 uint32_t stage_cap, uint32_t *bins, uint32_t *hist) {
  constexpr int kR = kKthRegs;
  const int t = threadIdx.x, lane = t & 31;
  KthBound b{0u, 0u, 0u};
  const uint32_t nr = min(np, (uint32_t)(NT * kR));
  const uint32_t ns = min(np - nr, stage_cap);
  uint32_t above = 0;  // entries above the range in hand
#pragma unroll 1
  for (int part = 0; part < 2; ++part) {  // the keys, then (ties) the ~ids of the entries with key b.key
    // values: 0 = not one
    uint32_t val[kR];
    auto value = [&](uint32_t j) {
      if (part == 0) return __ldcg(&src[j].x);
      const uint2 e = __ldcg(src + j);
      return e.x == b.key ? 0xFFFFFFFFu - e.y : 0u;
    };
#pragma unroll
    for (int u = 0; u < kR; ++u) {
      const uint32_t j = (uint32_t)u * NT + t;
      val[u] = j < nr ? value(j) : 0u;
    }
#pragma unroll 8
    for (uint32_t j = t; j < ns; j += NT) stage[j] = value(nr + j);  // read back by this thread
    // hist[8..10]: the smallest value - 1, the largest, their number
    if (t == 0) {
      hist[8] = 0xFFFFFFFFu;
      hist[9] = 0;
      hist[10] = 0;
    }
    uint32_t lo = 0xFFFFFFFFu, hi = 0, v = 0;
    auto see = [&](uint32_t x) {
      hi = max(hi, x);
      lo = min(lo, x - 1u);  // 0 wraps to the top: left out
      v += x != 0u;
    };
#pragma unroll
    for (int u = 0; u < kR; ++u) {
      if ((uint32_t)u * NT >= nr) break;  // uniform
      see(val[u]);
    }
    for (uint32_t j = t; j < ns; j += NT) see(stage[j]);
    lo = __reduce_min_sync(0xFFFFFFFFu, lo);
    hi = __reduce_max_sync(0xFFFFFFFFu, hi);
    v = __reduce_add_sync(0xFFFFFFFFu, v);
    __syncthreads();
    if (lane == 0) {
      atomicMin(&hist[8], lo);
      atomicMax(&hist[9], hi);
      atomicAdd(&hist[10], v);
    }
    __syncthreads();
    lo = hist[8] + 1u;
    hi = hist[9];
    if (above + hist[10] < k) break;  // (keys only: the ids are those of enough entries)
    uint32_t bound;
#pragma unroll 1
    for (;;) {
      const uint32_t width = hi - lo;  // bins of 2^s values each
      const int s = max(0, 21 - __clz((int)width));
      for (uint32_t i = t; i < kLinBins; i += NT) bins[i] = 0;
      __syncthreads();
      auto count = [&](uint32_t x) {
        if (x - lo <= width) atomicAdd(&bins[(x - lo) >> s], 1u);
      };
#pragma unroll
      for (int u = 0; u < kR; ++u) {
        if ((uint32_t)u * NT >= nr) break;  // uniform
        count(val[u]);
      }
      for (uint32_t j = t; j < ns; j += NT) count(stage[j]);
      __syncthreads();
      bins_find<NT>(bins, above, k, hist, false);
      bound = lo + (hist[11] << s);
      above = hist[12];
      b.count = above + hist[13];
      if (s == 0 || b.count <= k + k / 4u + 32u) break;  // uniform
      lo = bound;
      // (bound <= hi: the bin holds a value.  As a sum, the bin's end may lie past 2^32 -- the
      // ~ids of the first rows -- and a wrapped hi would let the zeros of no entry in.)
      hi = bound + min(hi - bound, (1u << s) - 1u);
      __syncthreads();  // hist has been read
    }
    if (part == 0) b.key = bound;
    else b.low = bound;
    __syncthreads();  // hist has been read
    if (b.count <= k + k / 4u + 32u) break;
  }
  __syncthreads();  // hist and bins are free again
  return b;
}

// The rank of every entry buf[0..n) among them, best first: entries fall into linear bins
// over their keys, and an entry counts the better ones of its own bin.  emit(rank, entry)
// runs once per entry.  order: n words.  False, with nothing emitted, when a bin holds so
// many entries (equal keys, mostly) that a sort is cheaper.
template <int NT, class Emit>
__device__ __forceinline__ bool block_rank_bins(const uint2 *buf, uint32_t n, uint32_t *order, uint32_t *bins,
                                                uint32_t *hist, Emit emit) {
  const int t = threadIdx.x;
  constexpr uint32_t kMostPerBin = 48;
  if (t == 0) {
    hist[8] = 0xFFFFFFFFu;
    hist[9] = 0;
    hist[10] = 0;
  }
  uint32_t lo = 0xFFFFFFFFu, hi = 0, most = 0;
  for (uint32_t j = t; j < n; j += NT) {
    lo = min(lo, buf[j].x);
    hi = max(hi, buf[j].x);
  }
  lo = __reduce_min_sync(0xFFFFFFFFu, lo);
  hi = __reduce_max_sync(0xFFFFFFFFu, hi);
  for (uint32_t i = t; i < kLinBins; i += NT) bins[i] = 0;
  __syncthreads();
  if ((t & 31) == 0) {
    atomicMin(&hist[8], lo);
    atomicMax(&hist[9], hi);
  }
  __syncthreads();
  lo = hist[8];
  hi = hist[9];
  const int s = max(0, 21 - __clz((int)(hi - lo)));
  for (uint32_t j = t; j < n; j += NT) most = max(most, atomicAdd(&bins[(buf[j].x - lo) >> s], 1u));
  most = __reduce_max_sync(0xFFFFFFFFu, most);
  if ((t & 31) == 0) atomicMax(&hist[10], most);
  __syncthreads();
  if (hist[10] >= kMostPerBin) return false;  // uniform
  bins_find<NT>(bins, 0u, 0xFFFFFFFFu, hist, true);  // each bin: the entries above it
  // the bins' members, bin by bin; afterwards a bin holds the end of its members
  for (uint32_t j = t; j < n; j += NT) order[atomicAdd(&bins[(buf[j].x - lo) >> s], 1u)] = j;
  __syncthreads();
  for (uint32_t j = t; j < n; j += NT) {
    const uint2 e = buf[j];
    const uint32_t bin = (e.x - lo) >> s;
    const uint64_t c = composite(e.x, e.y);
    // the members start where the bin above ends
    const uint32_t first = bin + 1u < kLinBins ? bins[bin + 1u] : 0u, end = bins[bin];
    uint32_t r = first;
    for (uint32_t i = first; i < end; ++i) {
      const uint2 o = buf[order[i]];
      r += composite(o.x, o.y) > c;
    }
    emit(r, e);
  }
  return true;
}

// Barrier after one stage of a bitonic network whose comparator i (thread i % NT, whole
// warps) exchanges elements lo = 2i - (i & (stride - 1)) and lo + stride.  Up to stride
// 32 the comparators of a warp touch only their own 64-element blocks, so the warp's
// own barrier orders the stage; larger strides need the block's.  The caller ends each
// size with a block barrier (the next size starts with its largest stride).
__device__ __forceinline__ void bitonic_stage_sync(uint32_t stride) {
  if (stride > 32) __syncthreads();
  else __syncwarp();
}

// Sort a[0..n) descending by composite (bitonic, padded to a power of two; the
// caller guarantees room for the padding).
template <int NT>
__device__ void block_sort_desc(uint2 *a, uint32_t n) {
  const int t = threadIdx.x;
  uint32_t P = 1;
  while (P < n) P <<= 1;
  for (uint32_t j = n + t; j < P; j += NT) a[j] = make_uint2(0u, 0xFFFFFFFFu);
  __syncthreads();
  for (uint32_t size = 2; size <= P; size <<= 1) {
    for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
      for (uint32_t i = t; i < P / 2; i += NT) {
        const uint32_t lo = 2 * i - (i & (stride - 1));
        const uint32_t hi = lo + stride;
        const bool desc = (lo & size) == 0;
        const uint2 x = a[lo], y = a[hi];
        const uint64_t cx = composite(x.x, x.y), cy = composite(y.x, y.y);
        if (desc ? (cx < cy) : (cx > cy)) {
          a[lo] = y;
          a[hi] = x;
        }
      }
      bitonic_stage_sync(stride);
    }
    __syncthreads();
  }
}

// Lowest float whose key is >= thr, for thr > 0: keys 1..key(-inf) are the
// negative-NaN patterns no score maps to, so they all mean "any number".
__device__ __forceinline__ float thr_float(uint32_t thr) {
  return thr <= 0x007FFFFFu ? __int_as_float(0xFF800000) : key2f(thr);
}

}  // namespace topk
