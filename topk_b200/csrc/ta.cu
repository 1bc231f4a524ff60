// The threshold algorithm over sorted attribute lists, on the device.
//
// The reference's TA (cpu/TA.h) sorts one list per attribute by value, descending
// (init, :40-58), then walks the queried lists in lock step: at depth i it scores every
// object it meets for the first time (random access to the table) and keeps the k best;
// the threshold is sum_m w_m * list_m[i], and it stops once the k-th score reaches it
// (:61-96).  Here the lists are built with stable device radix sorts (values
// descending, ties by the lower id) and kept as ids plus values, and a query walks them
// in blocks of growing depth (max(16384, 4k) entries per list, growing fourfold): one
// kernel takes every (list, depth) entry of the block, claims the object in a
// seen-bitmap (each object is scored once), scores it exactly in the reference order
// and appends it when it beats the current k-th; a second one selects the best k of the
// appended keys and the running top k through a histogram of the scores.  4M rows x 8,
// q = 4, k = 64, one block of depth: 194 us with a radix sort of the keys, 48 us so.
// The bound of the unseen objects after depth i is the reference's threshold with each
// weight's sign respected (w < 0 takes the attribute's minimum), in the same FP32
// operations, so it bounds their scores exactly; the walk stops when the k-th score is
// strictly above it, so no unseen object can tie the k-th with a lower id.  Results are
// those of the full scan.
//
// The reference scores an object with the weight of the list it was found in for
// every attribute (cpu/TA.h:83: the inner loop reuses the outer `weight`), which gives
// wrong scores unless all weights are equal; this implementation uses each attribute's
// own weight.
#include <cub/device/device_radix_sort.cuh>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <string>

#include "../../include/topk_b200.h"
#include "block_select.cuh"
#include "device_common.cuh"
#include "topk_internal.h"

namespace topk {

namespace {

struct TaQuery {
  uint32_t qq;
  uint8_t attr[kMaxQ];
  float w[kMaxQ];
};

__global__ void ta_keys_kernel(const float *__restrict__ col, uint64_t n, uint32_t *__restrict__ keys,
                               uint32_t *__restrict__ ids) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    keys[i] = f2key(__ldg(col + i));
    ids[i] = (uint32_t)i;
  }
}

__global__ void ta_values_kernel(const uint32_t *__restrict__ keys, uint64_t n, float *__restrict__ vals) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    vals[i] = key2f(keys[i]);
}

// The state of one query's walk, cleared before it (one block with the seen-bitmap).
constexpr uint32_t kTaBins = 2048;
constexpr uint32_t kTaSelect = 4096;  // entries the last block of ta_select_kernel sorts
struct TaHead {
  unsigned long long kth;  // key of the k-th best so far (0: fewer than k)
  uint32_t count, scored;  // keys of this block of depth, objects scored so far
  uint32_t small, done;    // ta_select_kernel's list and its finished blocks
  float lo, mid, hi;       // see TaBins
  alignas(16) uint32_t hist[kTaBins];  // keys of this block of depth by bin
};

// What a block of depth reports, in mapped pinned memory: the host reads it after the
// block's one synchronisation.
struct TaSlot {
  unsigned long long kth;
  uint32_t count, scored, kept, overflow;
  float bound;
  uint32_t pad;
  unsigned long long top[kMaxK];  // the best `kept` keys, descending
};

// Bins by score, rising: the upper half divides [mid, hi], mid the bound of the objects
// after this block of depth and hi the one of all objects; the lower half divides
// [lo, mid], lo the least score the lists allow.  The walk ends when k objects lie above
// mid, so that is where the bins must be fine.  A range that is empty or not finite is
// one bin; so is NaN, the lowest.  Any monotone map selects the same objects.
struct TaBins {
  float lo, mid, slo, shi;
  __device__ TaBins(float l, float m, float h) : lo(l), mid(m), slo(scale(l, m)), shi(scale(m, h)) {}
  __device__ static float scale(float a, float b) {
    const float r = __fdiv_rn((float)(kTaBins / 2), __fsub_rn(b, a));
    return (b > a && r > 0.0f && r <= 3.4e38f) ? r : 0.0f;
  }
  __device__ uint32_t operator()(unsigned long long key) const {
    const float x = key2f((uint32_t)(key >> 32));
    const bool up = x >= mid;
    const float t = __fmul_rn(__fsub_rn(x, up ? mid : lo), up ? shi : slo);
    const uint32_t b = t > 0.0f ? (uint32_t)fminf(t, (float)(kTaBins / 2 - 1)) : 0u;
    return b + (up ? kTaBins / 2 : 0);
  }
};

// Every entry (list m, depth i0 + j) of the block: first sight of the object claims it
// and scores it; it is appended when its key beats the current k-th key (0: fewer than
// k kept so far), after the `kept` keys carried over from the block before.  Also the
// keys' histogram and the bounds the bins stand on: a bound takes, for each weight, the
// list's entry at a depth (w < 0: at the list's end), in the query's order with one
// rounding per operation, so it bounds every object after that depth exactly.
// Bound by the gathers: one random sector per object and attribute, and the bitmap's
// atomics.
__global__ void __launch_bounds__(256)
    ta_score_kernel(const uint32_t *__restrict__ lists, const float *__restrict__ vals, uint64_t n,
                    const float *__restrict__ table, uint64_t ld, TaQuery q, uint64_t i0, uint32_t len,
                    const unsigned long long *__restrict__ top, uint32_t kept, uint32_t *__restrict__ seen,
                    unsigned long long *__restrict__ out, TaHead *__restrict__ head) {
  __shared__ uint32_t hist[kTaBins];
  __shared__ float term[3 * kMaxQ], bnd[3];
  const uint32_t t = threadIdx.x, lane = t & 31;
  for (uint32_t i = t; i < kTaBins; i += 256) hist[i] = 0;
  if (t < 3 * q.qq) {
    const uint32_t j = t % q.qq, which = t / q.qq;  // 0: lo, 1: mid, 2: hi
    const bool pos = q.w[j] >= 0.0f;
    const uint64_t at = which == 0 ? (pos ? n - 1 : 0) : (pos ? (which == 1 ? i0 + len - 1 : 0) : n - 1);
    term[t] = __fmul_rn(__ldg(vals + (uint64_t)q.attr[j] * n + at), q.w[j]);
  }
  __syncthreads();
  if (t < 3) {
    float s = 0.0f;
    for (uint32_t j = 0; j < q.qq; ++j) s = __fadd_rn(s, term[t * q.qq + j]);
    bnd[t] = s;
    if (blockIdx.x == 0) (t == 0 ? head->lo : t == 1 ? head->mid : head->hi) = s;
  }
  __syncthreads();
  const TaBins bins(bnd[0], bnd[1], bnd[2]);
  const unsigned long long bar = head->kth;
  const uint32_t total = kept + len * q.qq;
  uint32_t mine = 0;
  for (uint32_t base = blockIdx.x * 256; base < total; base += gridDim.x * 256) {
    const uint32_t e = base + t;
    unsigned long long key = 0;
    bool add = false;
    if (e < kept) {
      key = top[e];
      add = true;
    } else if (e < total) {
      const uint32_t x = e - kept, m = x / len;
      const uint32_t id = __ldg(lists + (uint64_t)q.attr[m] * n + i0 + (x - m * len));
      const uint32_t bit = 1u << (id & 31);
      if (!(atomicOr(seen + (id >> 5), bit) & bit)) {  // not met before
        ++mine;
        float s = 0.0f;
        for (uint32_t j = 0; j < q.qq; ++j)
          s = __fadd_rn(s, __fmul_rn(__ldg(table + (uint64_t)q.attr[j] * ld + id), q.w[j]));
        key = composite(f2key(s), id);
        add = key > bar;
      }
    }
    const uint32_t mask = __ballot_sync(0xFFFFFFFFu, add);
    if (!mask) continue;
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(&head->count, (uint32_t)__popc(mask));
    at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(mask & ((1u << lane) - 1));
    if (add) {
      out[at] = key;
      atomicAdd(&hist[bins(key)], 1u);
    }
  }
  mine = __reduce_add_sync(0xFFFFFFFFu, mine);
  if (lane == 0 && mine) atomicAdd(&head->scored, mine);
  __syncthreads();
  for (uint32_t i = t; i < kTaBins; i += 256)
    if (hist[i]) atomicAdd(&head->hist[i], hist[i]);
}

// The best kk of the block's keys: the histogram gives the highest bin with kk keys at or
// above it; those keys are gathered by the whole grid, and the last block sorts them,
// keeps kk and reports.  More than kTaSelect of them (ties, a range of scores much wider
// than that of the best, a large k) is reported as an overflow and left to a sort of all
// keys: 60 thousand keys sorted by a 64-bit radix sort took 90 us, this takes 13.
constexpr int kTaSelThreads = 512;
__global__ void __launch_bounds__(kTaSelThreads)
    ta_select_kernel(const unsigned long long *__restrict__ keys, uint32_t kk, unsigned long long *__restrict__ small,
                     unsigned long long *__restrict__ top, TaHead *__restrict__ head, TaSlot *__restrict__ slot) {
  static_assert(kTaBins == 4 * kTaSelThreads, "four bins a thread");
  __shared__ uint2 list[kTaSelect];
  __shared__ uint32_t wsum[kTaSelThreads / 32], s_edge, s_n, s_last;
  const uint32_t t = threadIdx.x, lane = t & 31, w = t / 32;
  const uint32_t total = head->count;
  const uint4 h4 = reinterpret_cast<const uint4 *>(head->hist)[t];
  const uint32_t c[4] = {h4.x, h4.y, h4.z, h4.w};
  const uint32_t sum = c[0] + c[1] + c[2] + c[3];
  uint32_t incl = sum;  // keys in this thread's bins and above, within the warp
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_down_sync(0xFFFFFFFFu, incl, o);
    if (lane + o < 32) incl += y;
  }
  if (lane == 0) wsum[w] = incl;
  if (t == 0) {
    s_edge = 0;  // fewer than kk keys: all of them
    s_n = total;
  }
  __syncthreads();
  for (uint32_t i = w + 1; i < kTaSelThreads / 32; ++i) incl += wsum[i];
  uint32_t above = incl - sum;
  if (above < kk && incl >= kk) {
    int i = 3;
    while ((above += c[i]) < kk) --i;
    s_edge = 4 * t + i;
    s_n = above;
  }
  __syncthreads();
  const uint32_t edge = s_edge, m = s_n;
  const bool fits = m <= kTaSelect;
  if (fits) {
    const TaBins bins(head->lo, head->mid, head->hi);
    for (uint32_t base = blockIdx.x * kTaSelThreads; base < total; base += gridDim.x * kTaSelThreads) {
      const unsigned long long key = base + t < total ? keys[base + t] : 0ull;
      const bool add = base + t < total && bins(key) >= edge;
      const uint32_t mask = __ballot_sync(0xFFFFFFFFu, add);
      if (!mask) continue;
      uint32_t at = 0;
      if (lane == 0) at = atomicAdd(&head->small, (uint32_t)__popc(mask));
      at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(mask & ((1u << lane) - 1));
      if (add) small[at] = key;
    }
  }
  __threadfence();
  __syncthreads();
  if (t == 0) s_last = atomicAdd(&head->done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const uint32_t kept = fits ? min(m, kk) : 0;
  if (fits) {
    for (uint32_t i = t; i < m; i += kTaSelThreads) {
      const unsigned long long key = __ldcg(small + i);
      list[i] = make_uint2((uint32_t)(key >> 32), 0xFFFFFFFFu - (uint32_t)key);
    }
    block_sort_desc<kTaSelThreads>(list, m);
    __syncthreads();
    for (uint32_t i = t; i < kept; i += kTaSelThreads) {
      const unsigned long long key = composite(list[i].x, list[i].y);
      top[i] = key;
      slot->top[i] = key;
    }
  }
  reinterpret_cast<uint4 *>(head->hist)[t] = make_uint4(0, 0, 0, 0);  // for the next block of depth
  if (t == 0) {
    const unsigned long long kth = kept == kk ? composite(list[kk - 1].x, list[kk - 1].y) : 0ull;
    if (fits) head->kth = kth;
    slot->kth = kth;
    slot->count = total;
    slot->scored = head->scored;
    slot->kept = kept;
    slot->overflow = !fits;
    slot->bound = head->mid;
    head->count = head->small = head->done = 0;
  }
}

int grid_of(uint64_t work, int num_sms) {
  const uint64_t b = (work + 255) / 256;
  return (int)std::max<uint64_t>(1, std::min<uint64_t>(b, (uint64_t)num_sms * 16));
}

}  // namespace

// Sorted lists of the reference's TA: per attribute the ids by value descending (ties
// by the lower id) and the values in that order.  Both [d][n].
struct TaLists {
  uint64_t n = 0;
  uint32_t d = 0;
  uint32_t *ids = nullptr;
  float *vals = nullptr;
  // query scratch
  TaHead *head = nullptr;  // followed by the seen-bitmap: one allocation, one clear
  uint32_t *seen = nullptr;
  unsigned long long *buf[2] = {nullptr, nullptr};  // a block's keys; sorted (or selected) ones
  unsigned long long *top = nullptr;                // the best k so far
  void *temp = nullptr;
  size_t temp_bytes = 0;
  TaSlot *host = nullptr, *slot = nullptr;  // mapped: host and device address
  cudaStream_t s = nullptr;
  ~TaLists() {
    if (s) cudaStreamSynchronize(s);
    cudaFree(ids);
    cudaFree(vals);
    cudaFree(head);
    cudaFree(buf[0]);
    cudaFree(buf[1]);
    cudaFree(top);
    cudaFree(temp);
    cudaFreeHost(host);
    if (s) cudaStreamDestroy(s);
  }
};

void ta_lists_free(TaLists *L) { delete L; }

// Largest block of depth: its appended keys fit the scratch.
static uint64_t ta_block_cap(uint32_t qq) { return std::max<uint64_t>(1024, (1ull << 22) / std::max(1u, qq)); }

int ta_lists_build(TaLists **out, const float *table, uint64_t ld, uint32_t d, uint64_t n, int num_sms,
                   std::string *msg) {
  if (n > 0x7FFFFFFFull) {
    *msg = "sorted lists need n < 2^31";
    return TOPK_ERR_UNSUPPORTED;
  }
  TaLists *L = new TaLists();
  L->n = n;
  L->d = d;
  uint32_t *kin = nullptr, *kout = nullptr, *iin = nullptr;
  void *stemp = nullptr;
  size_t stb = 0;
  cudaError_t e = cudaStreamCreateWithFlags(&L->s, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaMalloc(&L->ids, (size_t)d * n * sizeof(uint32_t));
  if (e == cudaSuccess) e = cudaMalloc(&L->vals, (size_t)d * n * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&kin, n * sizeof(uint32_t));
  if (e == cudaSuccess) e = cudaMalloc(&kout, n * sizeof(uint32_t));
  if (e == cudaSuccess) e = cudaMalloc(&iin, n * sizeof(uint32_t));
  if (e == cudaSuccess)
    e = cub::DeviceRadixSort::SortPairsDescending(nullptr, stb, kin, kout, iin, L->ids, (int)n, 0, 32, L->s);
  if (e == cudaSuccess) e = cudaMalloc(&stemp, std::max<size_t>(stb, 16));
  const int g = grid_of(n, num_sms);
  for (uint32_t m = 0; m < d && e == cudaSuccess; ++m) {
    ta_keys_kernel<<<g, 256, 0, L->s>>>(table + (uint64_t)m * ld, n, kin, iin);
    size_t tb = stb;
    e = cub::DeviceRadixSort::SortPairsDescending(stemp, tb, kin, kout, iin, L->ids + (uint64_t)m * n, (int)n, 0, 32,
                                                  L->s);
    if (e == cudaSuccess) ta_values_kernel<<<g, 256, 0, L->s>>>(kout, n, L->vals + (uint64_t)m * n);
  }
  // query scratch: seen bitmap, two key buffers of k + one block's appends, sort scratch
  const uint64_t cap = kMaxK + (1ull << 22) + 64;
  if (e == cudaSuccess) e = cudaMalloc(&L->head, sizeof(TaHead) + (n + 31) / 32 * sizeof(uint32_t));
  if (e == cudaSuccess) L->seen = reinterpret_cast<uint32_t *>(L->head + 1);
  if (e == cudaSuccess) e = cudaMalloc(&L->buf[0], cap * sizeof(unsigned long long));
  if (e == cudaSuccess) e = cudaMalloc(&L->buf[1], cap * sizeof(unsigned long long));
  if (e == cudaSuccess)
    e = cub::DeviceRadixSort::SortKeysDescending(nullptr, L->temp_bytes, L->buf[0], L->buf[1], (int)cap, 0, 64,
                                                  L->s);
  if (e == cudaSuccess) e = cudaMalloc(&L->temp, std::max<size_t>(L->temp_bytes, 16));
  if (e == cudaSuccess) e = cudaMalloc(&L->top, kMaxK * sizeof(unsigned long long));
  if (e == cudaSuccess) e = cudaHostAlloc(&L->host, sizeof(TaSlot), cudaHostAllocMapped);
  if (e == cudaSuccess) e = cudaHostGetDevicePointer(reinterpret_cast<void **>(&L->slot), L->host, 0);
  if (e == cudaSuccess) e = cudaStreamSynchronize(L->s);
  cudaFree(kin);
  cudaFree(kout);
  cudaFree(iin);
  cudaFree(stemp);
  if (e != cudaSuccess) {
    *msg = std::string("building the sorted lists: ") + cudaGetErrorString(e);
    delete L;
    return e == cudaErrorMemoryAllocation ? TOPK_ERR_OOM : TOPK_ERR_CUDA;
  }
  *out = L;
  return TOPK_OK;
}

int ta_lists_read(const TaLists *L, uint32_t m, uint32_t *ids, float *vals, std::string *msg) {
  cudaError_t e = cudaSuccess;
  if (ids) e = cudaMemcpy(ids, L->ids + (uint64_t)m * L->n, L->n * sizeof(uint32_t), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && vals)
    e = cudaMemcpy(vals, L->vals + (uint64_t)m * L->n, L->n * sizeof(float), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) {
    *msg = std::string("reading the lists: ") + cudaGetErrorString(e);
    return TOPK_ERR_CUDA;
  }
  return TOPK_OK;
}

int ta_query(TaLists *L, const float *table, uint64_t ld, uint64_t k, uint32_t qq, const float *weights,
             const uint8_t *attr, int num_sms, uint64_t *ids, float *scores, uint64_t *count, float *threshold,
             uint64_t *stats, std::string *msg) {
  const uint64_t n = L->n;
  const uint64_t kk = std::min<uint64_t>(k, n);
  TaQuery q{};
  q.qq = qq;
  for (uint32_t m = 0; m < qq; ++m) {
    q.attr[m] = attr[m];
    q.w[m] = weights[attr[m]];
  }
  cudaStream_t s = L->s;
  cudaError_t e = cudaMemsetAsync(L->head, 0, sizeof(TaHead) + (n + 31) / 32 * sizeof(uint32_t), s);
  uint64_t kept = 0, depth = 0, iters = 0;
  const uint64_t bmax = ta_block_cap(qq);
  uint64_t block = std::min<uint64_t>(bmax, std::max<uint64_t>(16384, 4 * kk));
  bool done = false;
  while (e == cudaSuccess && !done) {
    const uint64_t len = std::min<uint64_t>(block, n - depth);
    const uint64_t most = kept + len * qq;  // at most kMaxK + 2^22 keys
    ta_score_kernel<<<grid_of(most, num_sms), 256, 0, s>>>(L->ids, L->vals, n, table, ld, q, depth, (uint32_t)len,
                                                           L->top, (uint32_t)kept, L->seen, L->buf[0], L->head);
    const int sel = (int)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)num_sms, most / 2048));
    ta_select_kernel<<<sel, kTaSelThreads, 0, s>>>(L->buf[0], (uint32_t)kk, L->buf[1], L->top, L->head, L->slot);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) break;
    depth += len;
    ++iters;
    kept = L->host->kept;
    if (L->host->overflow) {  // sort all of them, into the place the selection would have filled
      const uint64_t total = L->host->count;
      size_t tb = L->temp_bytes;
      kept = std::min<uint64_t>(kk, total);
      e = cub::DeviceRadixSort::SortKeysDescending(L->temp, tb, L->buf[0], L->buf[1], (int)total, 0, 64, s);
      if (e == cudaSuccess)
        e = cudaMemcpyAsync(L->top, L->buf[1], kept * sizeof(unsigned long long), cudaMemcpyDeviceToDevice, s);
      if (e == cudaSuccess)
        e = cudaMemcpyAsync(L->host->top, L->buf[1], kept * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess && kept == kk)
        e = cudaMemcpyAsync(&L->head->kth, L->buf[1] + kk - 1, sizeof(unsigned long long), cudaMemcpyDeviceToDevice, s);
      if (e == cudaSuccess) e = cudaStreamSynchronize(s);
      if (e != cudaSuccess) break;
      L->host->kth = kept == kk ? L->host->top[kk - 1] : 0ull;
    }
    if (depth >= n) break;
    if (kept == kk) {
      // stop when the k-th score is strictly above every unseen object's bound
      const uint32_t kth_key = (uint32_t)(L->host->kth >> 32);
      const float b = L->host->bound;
      uint32_t bu;
      std::memcpy(&bu, &b, 4);
      const uint32_t bkey = (b != b) ? 0u : ((bu & 0x80000000u) ? ~bu : (bu | 0x80000000u));
      if (kth_key > bkey) done = true;
    }
    block = std::min<uint64_t>(bmax, block * 4);  // each block costs a host round trip
  }
  if (e != cudaSuccess) {
    *msg = std::string("TA query: ") + cudaGetErrorString(e);
    return TOPK_ERR_CUDA;
  }
  const unsigned long long *keys = L->host->top;
  // ascending by score (the reference's heap drain): the descending keys reversed
  for (uint64_t j = 0; j < kept; ++j) {
    const unsigned long long key = keys[kept - 1 - j];
    const uint32_t kf = (uint32_t)(key >> 32);
    const uint32_t u = (kf & 0x80000000u) ? (kf & 0x7FFFFFFFu) : ~kf;
    float f;
    std::memcpy(&f, &u, 4);
    ids[j] = 0xFFFFFFFFull - (key & 0xFFFFFFFFull);
    scores[j] = f;
  }
  if (count) *count = kept;
  if (threshold) *threshold = kept ? scores[0] : 0.0f;
  if (stats) {
    stats[0] = depth;
    stats[1] = L->host->scored;
    stats[2] = iters;
  }
  return TOPK_OK;
}

}  // namespace topk
