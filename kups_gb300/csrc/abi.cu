// Library identity and error strings of the kups_gb300 C ABI.
#include <algorithm>

#include "common.cuh"

extern "C" const char *kups_version(void) { return "kups_gb300 0.1.0 sm_103a"; }

extern "C" const char *kups_error_string(int32_t code) {
  switch (code) {
    case KUPS_OK: return "ok";
    case KUPS_ERR_CAPACITY: return "capacity exceeded (status.required holds the size that suffices)";
    case KUPS_ERR_NONFINITE: return "non-finite value encountered";
    case KUPS_ERR_INVALID: return "invalid argument";
    case KUPS_ERR_CUDA: return "CUDA launch or runtime error";
    case KUPS_ERR_UNSUPPORTED: return "unsupported configuration";
    default: return "unknown error";
  }
}

namespace {
__global__ void status_init_kernel(kups_status *status, int64_t *counts, int32_t n_counts) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) *status = kups_status{KUPS_OK, 0, 0, -1};
  if (i < n_counts) counts[i] = 0;
}

// Offsets of the systems' atoms: each thread counts the runs of equal indices among 16 neighbouring atoms
// (systems are usually grouped), the last block to finish turns counts into offsets.
constexpr int kOffThreads = 256, kOffPer = 16;

__global__ void __launch_bounds__(kOffThreads) system_offsets_kernel(const int32_t *system, int64_t n, int32_t n_sys,
                                                                     int32_t *off, int32_t *stats) {
  __shared__ int scan[33], most, last;
  const int64_t i0 = ((int64_t)blockIdx.x * kOffThreads + threadIdx.x) * kOffPer, i1 = min(n, i0 + kOffPer);
  for (int64_t i = i0; i < i1;) {
    const int s = system[i];
    int run = 1;
    while (i + run < i1 && system[i + run] == s) ++run;
    if (s >= 0 && s < n_sys) atomicAdd(&off[s + 1], run);
    else atomicAdd(&stats[1], run);
    i += run;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(&stats[2], 1) == (int)gridDim.x - 1;
    most = 0;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  int carry = 0;
  for (int b = 0; b < n_sys; b += kOffThreads) {
    const int s = b + threadIdx.x, c = s < n_sys ? __ldcg(&off[s + 1]) : 0;
    atomicMax(&most, c);
    int total;
    const int before = kups::block_exclusive_scan<int>(c, scan, &total);
    if (s < n_sys) off[s + 1] = carry + before + c;
    carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) stats[0] = most;
}
}  // namespace

extern "C" int32_t kups_system_offsets(const int32_t *system, int64_t n, int32_t n_systems, int32_t *offsets,
                                       int32_t stats[3], void *stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (n < 0 || n > INT32_MAX || n_systems < 0 || offsets == nullptr || stats == nullptr || (n > 0 && system == nullptr))
    return KUPS_ERR_INVALID;
  KUPS_CUDA_TRY(cudaMemsetAsync(offsets, 0, sizeof(int32_t) * ((size_t)n_systems + 1), stream));
  KUPS_CUDA_TRY(cudaMemsetAsync(stats, 0, 3 * sizeof(int32_t), stream));
  const int64_t per = (int64_t)kOffThreads * kOffPer;
  system_offsets_kernel<<<(unsigned)std::max<int64_t>(1, (n + per - 1) / per), kOffThreads, 0, stream>>>(
      system, n, n_systems, offsets, stats);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

extern "C" int32_t kups_status_init(kups_status *status, int64_t *counts, int32_t n_counts, void *stream) {
  if (status == nullptr || n_counts < 0 || (n_counts > 0 && counts == nullptr)) return KUPS_ERR_INVALID;
  status_init_kernel<<<(unsigned)(n_counts / 128 + 1), 128, 0, (cudaStream_t)stream>>>(status, counts, n_counts);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}
