// Skyline layers of SLA (cpu/SLA.h:102-139) on the device.
//
// The reference peels layers: while more than 100 rows remain, the skyline of the
// remaining rows (no other remaining row dominates them; p dominates q when p <= q in
// every attribute and p < q in one, on the values 1 - x, cpu/SLA.h:87-100) is the next
// layer, and the last <= 100 rows form one final layer.  Here the same layers come
// from depths: a row's depth is 1 + the largest depth of the rows that dominate it (0
// for the skyline).  Every dominator of a row has an FP32 coordinate sum no larger
// (one rounding per addition is monotone) and, at an equal sum, comes first in the
// lexicographic order of its values; so with the rows sorted that way (stable radix
// sorts, least significant key first) a row's dominators all come before it.  The
// sorted rows are cut into blocks of 256.  One launch per block: every later row takes
// the largest depth + 1 of its dominators in the block, and the next block's rows, which
// are final for all earlier blocks then, are settled among themselves in the same launch
// (sky_step_kernel).  The stop rule is applied to the depths on the host: the first depth
// l with at most 100 rows at depth >= l takes all of them.
// O(n^2 d / 2) compares: meant for the table sizes the reference's SLA serves.
#include <cub/device/device_radix_sort.cuh>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <string>
#include <vector>

#include "../../include/topk_b200.h"
#include "device_common.cuh"
#include "topk_internal.h"

namespace topk {

namespace {

constexpr uint32_t kSkyBlock = 256;   // rows per block (= threads of the block kernels)
constexpr uint32_t kSkyMaxD = 32;
// Largest table the layer build accepts.  The build compares O(n^2 d / 2) pairs in
// n / 256 sequential launches: 2^22 rows are about 1.4e14 compares
// (seconds to minutes on one B200); 2^26 rows would be 256 times that.
constexpr uint64_t kSkyMaxRows = 1ull << 22;
constexpr uint64_t kSkyStopRows = 100;  // cpu/SLA.h:110

// key of column m of the sky values (m == d: the FP32 sum of all of them)
__global__ void sky_key_kernel(const float *__restrict__ table, uint64_t ld, uint32_t d, uint64_t n, uint32_t m,
                               uint32_t *__restrict__ keys, uint32_t *__restrict__ ids) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    float v;
    if (m < d) {
      v = __fsub_rn(1.0f, __ldg(table + (uint64_t)m * ld + i));
    } else {
      v = 0.0f;
      for (uint32_t j = 0; j < d; ++j) v = __fadd_rn(v, __fsub_rn(1.0f, __ldg(table + (uint64_t)j * ld + i)));
    }
    keys[i] = f2key(v);
    ids[i] = (uint32_t)i;
  }
}

// key of column m for the rows in the current order (the next stable pass)
__global__ void sky_key_perm_kernel(const float *__restrict__ table, uint64_t ld, uint32_t d, uint64_t n, uint32_t m,
                                    const uint32_t *__restrict__ order, uint32_t *__restrict__ keys) {
  for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t i = order[j];
    float v;
    if (m < d) {
      v = __fsub_rn(1.0f, __ldg(table + (uint64_t)m * ld + i));
    } else {
      v = 0.0f;
      for (uint32_t q = 0; q < d; ++q) v = __fadd_rn(v, __fsub_rn(1.0f, __ldg(table + (uint64_t)q * ld + i)));
    }
    keys[j] = f2key(v);
  }
}

// sky values of the rows in sorted order, column-major [d][n]
__global__ void sky_gather_kernel(const float *__restrict__ table, uint64_t ld, uint32_t d, uint64_t n,
                                  const uint32_t *__restrict__ order, float *__restrict__ xs) {
  for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t i = order[j];
    for (uint32_t m = 0; m < d; ++m) xs[(uint64_t)m * n + j] = __fsub_rn(1.0f, __ldg(table + (uint64_t)m * ld + i));
  }
}

// A row's d values, D >= d of them compile-time, padded with equal values (zeros).  Does
// row p (shared memory) dominate q: p <= q in every value and p < q in one?  (NaN: no.)
// Four values at a time without a branch; rows of more go on only while some lane may
// still be dominated.
template <int D>
struct SkyRow {
  static constexpr int kPad = D <= 2 ? D : (D + 3) / 4 * 4;  // floats a row in shared memory
  float x[kPad];
  __device__ __forceinline__ void load(const float *__restrict__ xs, uint64_t n, uint32_t d, uint64_t j) {
#pragma unroll
    for (int m = 0; m < kPad; ++m) x[m] = (uint32_t)m < d ? xs[(uint64_t)m * n + j] : 0.0f;
  }
  __device__ __forceinline__ void store(float *row) const {
#pragma unroll
    for (int m = 0; m < kPad; ++m) row[m] = x[m];
  }
  __device__ __forceinline__ bool dominated_by(const float *row) const {
    bool le = true, lt = false;
#pragma unroll
    for (int m = 0; m < kPad; ++m) {
      if (D > 8 && m && m % 4 == 0 && !le) return false;
      const float a = row[m];
      le = le && a <= x[m];
      lt = lt || a < x[m];
    }
    return le && lt;
  }
};

// One step: the rows from `first` on take 1 + the depth of their dominators in
// [r0, first) (at most kSkyBlock rows, settled), and block 0's rows -- the next kSkyBlock --
// are settled.  Among themselves they settle in order: a thread first finds which of the
// earlier rows of its block dominate it (a bit each), then warp by warp the lanes' depths
// become final one lane at a time (lane i's dominators are final by then), and the later
// warps take the finished warp's depths.  Nothing is repeated, whatever the data: the
// relaxation it replaced ran a pass over all pairs per link of the longest chain (30,011 x
// 4 anticorrelated rows: 16.6 ms in 236 launches, 2.6 ms in 118 now, of about 20 us each:
// the compares of one thread a row, then the 256 rows settled on one SM).
template <int D>
__global__ void __launch_bounds__(kSkyBlock)
    sky_step_kernel(const float *__restrict__ xs, uint64_t n, uint32_t d, uint64_t r0, uint64_t first,
                    uint32_t *__restrict__ cand, uint32_t *__restrict__ depth) {
  using Row = SkyRow<D>;
  __shared__ __align__(16) float sx[kSkyBlock * Row::kPad];
  __shared__ uint32_t sd[kSkyBlock];
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint32_t len = (uint32_t)(first - r0);
  Row row;
  if (t < len) {
    row.load(xs, n, d, r0 + t);
    row.store(sx + (size_t)t * Row::kPad);
    sd[t] = depth[r0 + t] + 1u;
  }
  const uint64_t j = first + (uint64_t)blockIdx.x * kSkyBlock + t;
  const bool live = j < n;
  uint32_t v = 0;
  if (live) {
    row.load(xs, n, d, j);
    v = cand[j];
  }
  __syncthreads();
  // (no branch on the depths in hand: the compares of several rows overlap)
#pragma unroll 8
  for (uint32_t i = 0; i < len; ++i) {
    const uint32_t di = sd[i];
    v = row.dominated_by(sx + (size_t)i * Row::kPad) ? max(v, di) : v;
  }
  if (blockIdx.x != 0) {
    if (live) cand[j] = v;
    return;
  }
  __syncthreads();  // the settled block has been read
  if (live) row.store(sx + (size_t)t * Row::kPad);
  __syncthreads();
  uint32_t mask[kSkyBlock / 32];  // the dominators among rows i < t
#pragma unroll
  for (uint32_t w = 0; w < kSkyBlock / 32; ++w) {
    mask[w] = 0;
    if (w > warp) continue;  // warp-uniform
#pragma unroll 8
    for (uint32_t i = 0; i < 32; ++i)
      mask[w] |= (row.dominated_by(sx + (size_t)(32u * w + i) * Row::kPad) ? 1u : 0u) << i;
    if (!live) mask[w] = 0;
    if (w == warp) mask[w] &= (1u << lane) - 1u;
  }
#pragma unroll
  for (uint32_t w = 0; w < kSkyBlock / 32; ++w) {
    if (warp == w) {
      for (uint32_t b = __reduce_or_sync(0xFFFFFFFFu, mask[w]); b; b &= b - 1u) {  // lanes that dominate one
        const int i = __ffs((int)b) - 1;
        const uint32_t di = __shfl_sync(0xFFFFFFFFu, v, i) + 1u;
        if (mask[w] >> i & 1u) v = max(v, di);
      }
      sd[t] = v + 1u;
    }
    __syncthreads();
    if (warp > w)
      for (uint32_t b = mask[w]; b; b &= b - 1u) v = max(v, sd[32u * w + (uint32_t)__ffs((int)b) - 1u]);
  }
  if (live) depth[j] = v;
}

using SkyStep = void (*)(const float *, uint64_t, uint32_t, uint64_t, uint64_t, uint32_t *, uint32_t *);
SkyStep sky_step(uint32_t d) {
  return d <= 1   ? sky_step_kernel<1>
         : d <= 2  ? sky_step_kernel<2>
         : d <= 4  ? sky_step_kernel<4>
         : d <= 8  ? sky_step_kernel<8>
         : d <= 16 ? sky_step_kernel<16>
                   : sky_step_kernel<(int)kSkyMaxD>;
}

int grid_n(uint64_t work, int num_sms) {
  const uint64_t b = (work + 255) / 256;
  return (int)std::max<uint64_t>(1, std::min<uint64_t>(b, (uint64_t)num_sms * 16));
}

}  // namespace

int skyline_layers_device(const float *table, uint64_t ld, uint32_t d, uint64_t n, int num_sms, uint32_t *layers,
                          uint64_t *num_layers, std::string *msg) {
  if (d == 0 || d > kSkyMaxD || n == 0 || n > kSkyMaxRows) {
    *msg = "skyline layers need 1 <= d <= 32 and 1 <= n <= 2^22 (the build compares O(n^2 d) pairs)";
    return TOPK_ERR_UNSUPPORTED;
  }
  cudaStream_t s = nullptr;
  uint32_t *kin = nullptr, *kout = nullptr, *oa = nullptr, *ob = nullptr, *cand = nullptr, *depth = nullptr;
  float *xs = nullptr;
  void *temp = nullptr;
  size_t tb = 0;
  cudaError_t e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cub::DeviceRadixSort::SortPairs(nullptr, tb, kin, kout, oa, ob, (int)n, 0, 32, s);
  // (an allocation each: small ones come from pages that the driver keeps mapped.  All in one,
  // 2.2 MB at 30,011 x 4, mapped its pages in every call: 0.6 ms, and now and then 5-800)
  std::vector<void *> owned;
  auto get = [&](auto **q, size_t bytes) {
    if (e != cudaSuccess) return;
    e = cudaMalloc(q, bytes);
    if (e == cudaSuccess) owned.push_back(*q);
  };
  for (uint32_t **q : {&kin, &kout, &oa, &ob, &cand, &depth}) get(q, n * sizeof(uint32_t));
  get(&xs, (size_t)d * n * sizeof(float));
  get(&temp, std::max<size_t>(tb, 16));
  const int g = grid_n(n, num_sms);
  // order: stable passes from the least significant key (the last value) to the sum
  if (e == cudaSuccess) {
    sky_key_kernel<<<g, 256, 0, s>>>(table, ld, d, n, d - 1, kin, oa);
    size_t t2 = tb;
    e = cub::DeviceRadixSort::SortPairs(temp, t2, kin, kout, oa, ob, (int)n, 0, 32, s);
    std::swap(oa, ob);
  }
  for (int m = (int)d - 2; e == cudaSuccess && m >= -1; --m) {
    const uint32_t key = m >= 0 ? (uint32_t)m : d;  // d: the sum, the most significant key
    sky_key_perm_kernel<<<g, 256, 0, s>>>(table, ld, d, n, key, oa, kin);
    size_t t2 = tb;
    e = cub::DeviceRadixSort::SortPairs(temp, t2, kin, kout, oa, ob, (int)n, 0, 32, s);
    std::swap(oa, ob);
  }
  if (e == cudaSuccess) {
    sky_gather_kernel<<<g, 256, 0, s>>>(table, ld, d, n, oa, xs);
    e = cudaMemsetAsync(cand, 0, n * sizeof(uint32_t), s);
  }
  const SkyStep step = sky_step(d);
  uint64_t r0 = 0, first = 0;  // the settled block [r0, first): none before the first step
  for (uint64_t a = 0; first < n && e == cudaSuccess; ++a) {
    step<<<(unsigned)((n - first + kSkyBlock - 1) / kSkyBlock), kSkyBlock, 0, s>>>(xs, n, d, r0, first, cand, depth);
    r0 = first;
    first = std::min<uint64_t>(n, first + kSkyBlock);
    if ((a & 255) == 255) e = cudaStreamSynchronize(s);  // keeps launch errors close to their cause
  }
  std::vector<uint32_t> dep(n), ord(n);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(dep.data(), depth, n * sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(ord.data(), oa, n * sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  for (void *q : owned) cudaFree(q);
  if (s) cudaStreamDestroy(s);
  if (e != cudaSuccess) {
    *msg = std::string("skyline layers: ") + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? TOPK_ERR_OOM : TOPK_ERR_CUDA;
  }
  // stop rule: the first depth l with at most 100 rows at depth >= l takes them all
  uint32_t dmax = 0;
  for (uint32_t v : dep) dmax = std::max(dmax, v);
  std::vector<uint64_t> beyond((size_t)dmax + 2, 0);
  for (uint32_t v : dep) beyond[v]++;
  for (int64_t l = (int64_t)dmax - 1; l >= 0; --l) beyond[(size_t)l] += beyond[(size_t)l + 1];
  uint32_t lstop = dmax + 1;
  for (uint32_t l = 0; l <= dmax; ++l)
    if (beyond[l] <= kSkyStopRows) {
      lstop = l;
      break;
    }
  uint32_t top = 0;
  for (uint64_t j = 0; j < n; ++j) {
    const uint32_t v = std::min(dep[j], lstop);
    layers[ord[j]] = v;
    top = std::max(top, v);
  }
  *num_layers = (uint64_t)top + 1;
  return TOPK_OK;
}

}  // namespace topk
