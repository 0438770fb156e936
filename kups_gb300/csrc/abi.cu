// Library identity and error strings of the kups_gb300 C ABI.
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
}  // namespace

extern "C" int32_t kups_status_init(kups_status *status, int64_t *counts, int32_t n_counts, void *stream) {
  if (status == nullptr || n_counts < 0 || (n_counts > 0 && counts == nullptr)) return KUPS_ERR_INVALID;
  status_init_kernel<<<(unsigned)(n_counts / 128 + 1), 128, 0, (cudaStream_t)stream>>>(status, counts, n_counts);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}
