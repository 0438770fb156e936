// Device-wide exclusive prefix sum used to turn per-item counts into offsets.
#pragma once

#include "common.cuh"

namespace kups {

constexpr int kScanBlock = 1024;

template <typename T>
__global__ void scan_blocks_kernel(T *data, int64_t n, T *block_sums) {
  __shared__ T scratch[32];
  const int64_t i = (int64_t)blockIdx.x * kScanBlock + threadIdx.x;
  const T v = i < n ? data[i] : T(0);
  T total;
  const T ex = block_exclusive_scan<T>(v, scratch, &total);
  if (i < n) data[i] = ex;
  if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

// One block scans the per-block totals sequentially in chunks and writes the
// grand total (if `total` is not null).
template <typename T>
__global__ void scan_sums_kernel(T *block_sums, int64_t nb, T *total) {
  __shared__ T scratch[32];
  T carry = 0;
  for (int64_t base = 0; base < nb; base += kScanBlock) {
    const int64_t i = base + threadIdx.x;
    const T v = i < nb ? block_sums[i] : T(0);
    T chunk;
    const T ex = block_exclusive_scan<T>(v, scratch, &chunk);
    if (i < nb) block_sums[i] = ex + carry;
    carry += chunk;
    __syncthreads();
  }
  if (threadIdx.x == 0 && total != nullptr) *total = carry;
}

template <typename T>
__global__ void scan_add_kernel(T *data, int64_t n, const T *block_sums) {
  const int64_t i = (int64_t)blockIdx.x * kScanBlock + threadIdx.x;
  if (i < n) data[i] += block_sums[blockIdx.x];
}

inline int64_t scan_blocks_needed(int64_t n) { return (n + kScanBlock - 1) / kScanBlock + 1; }

// In-place exclusive scan of data[0..n); `block_sums` has scan_blocks_needed(n)
// entries; `total` (device, may be null) receives the sum of all entries.
template <typename T>
inline cudaError_t exclusive_scan(T *data, int64_t n, T *block_sums, T *total, cudaStream_t s) {
  const int64_t nb = (n + kScanBlock - 1) / kScanBlock;
  if (nb > 0) scan_blocks_kernel<T><<<(unsigned)nb, kScanBlock, 0, s>>>(data, n, block_sums);
  scan_sums_kernel<T><<<1, kScanBlock, 0, s>>>(block_sums, nb, total);
  if (nb > 0) scan_add_kernel<T><<<(unsigned)nb, kScanBlock, 0, s>>>(data, n, block_sums);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- single-pass prefix
// Chained prefix over blocks (the single-pass scan with decoupled look-back of Merrill and Garland,
// 2016) that take their numbers from a ticket, so that a block's predecessors have started before it:
// state[b] holds a 2-bit flag above a 62-bit value, 0 = nothing yet, 1 = the block's own sum, 2 = the
// sum of blocks 0..b, 3 = a predecessor's wait ran out.  The words must be zero before the launch.  A
// block first publishes its own sum, then (at once or after other work) one full warp of it asks for
// the sum of blocks 0..b-1, which every lane returns.  The wait for a predecessor is bounded: when it
// runs out the block publishes flag 3, so no later block waits on it, and ok comes back false.
constexpr int kPrefixPolls = 1 << 22;

__device__ inline unsigned long long prefix_load(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ inline void prefix_store(unsigned long long *p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Block b's own sum, before it goes on to other work; a full warp calls it.
__device__ inline void chained_publish(unsigned long long *state, int64_t b, int64_t own) {
  if ((threadIdx.x & 31) == 0) prefix_store(state + b, ((b == 0 ? 2ull : 1ull) << 62) | (unsigned long long)own);
}

__device__ inline int64_t chained_prefix(unsigned long long *state, int64_t b, int64_t own, bool &ok) {
  const int lane = threadIdx.x & 31;
  constexpr unsigned long long kValue = (1ull << 62) - 1;
  ok = true;
  if (b == 0) return 0;
  int64_t sum = 0;
  for (int64_t top = b - 1;; top -= 32) {
    const int64_t at = top - lane;
    unsigned long long v = at >= 0 ? prefix_load(state + at) : (2ull << 62);
    for (int polls = 0; __any_sync(0xffffffffu, (v >> 62) == 0); ++polls) {
      if (polls == kPrefixPolls) {
        if (lane == 0) prefix_store(state + b, 3ull << 62);
        ok = false;
        return 0;
      }
      __nanosleep(20);
      if ((v >> 62) == 0) v = prefix_load(state + at);
    }
    const unsigned last = __ballot_sync(0xffffffffu, (v >> 62) >= 2);
    const int stop = last ? __ffs(last) - 1 : 31;
    if (__shfl_sync(0xffffffffu, (unsigned)(v >> 62), stop) == 3u) {
      if (lane == 0) prefix_store(state + b, 3ull << 62);
      ok = false;
      return 0;
    }
    int64_t part = lane <= stop ? (int64_t)(v & kValue) : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    sum += part;
    if (last) break;
  }
  if (lane == 0) prefix_store(state + b, (2ull << 62) | (unsigned long long)(sum + own));
  return sum;
}

// In-place exclusive scan of data[0..n) in one launch (kScanItems entries per thread): 2 launches
// and one read of the data fewer than exclusive_scan.  state: chained_scan_blocks(n) zeroed words,
// ticket: a zeroed word.
constexpr int kScanItems = 4, kChainedThreads = 512;

inline int64_t chained_scan_blocks(int64_t n) {
  return (n + kScanItems * kChainedThreads - 1) / (kScanItems * kChainedThreads);
}

__global__ void __launch_bounds__(kChainedThreads) chained_scan_kernel(int *data, int64_t n,
                                                                       unsigned long long *state, unsigned *ticket,
                                                                       kups_status *status) {
  __shared__ int scratch[32];
  __shared__ int64_t base;
  __shared__ unsigned bid;
  if (threadIdx.x == 0) bid = atomicAdd(ticket, 1u);
  __syncthreads();
  const int64_t b = bid;
  const int64_t i0 = (b * kChainedThreads + threadIdx.x) * kScanItems;
  int v[kScanItems], own = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    v[k] = i0 + k < n ? data[i0 + k] : 0;
    own += v[k];
  }
  int total;
  int ex = block_exclusive_scan<int>(own, scratch, &total);
  if (threadIdx.x < 32) {
    bool ok;
    chained_publish(state, b, total);
    const int64_t before = chained_prefix(state, b, total, ok);
    if (threadIdx.x == 0) {
      base = before;
      if (!ok) status_error(status, KUPS_ERR_UNSUPPORTED, b);
    }
  }
  __syncthreads();
  ex += (int)base;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (i0 + k < n) data[i0 + k] = ex;
    ex += v[k];
  }
}

}  // namespace kups
