// Lennard-Jones energy, dE/dx and dE/dtril over a directed edge list.
//
// Replaces lennard_jones_energy (src/kups/potential/classical/lennard_jones.py:149-178)
// and the jax.vjp gradient of PotentialFromEnergy with respect to
// PositionAndUnitCell (src/kups/potential/common/energy.py:264-355,
// lennard_jones.py:481-488).  Per directed edge e = (i, j, s):
//   d = x_j - x_i + s @ L,  r2 = |d|^2,  c6 = (sigma^2 / r2)^3,
//   E_e = 4 eps (c6^2 - c6) [r2 < rc^2],  g = dE_e/dd = -24 eps c6 (2 c6 - 1) d / r2,
// and E_s = sum E_e / 2, dE/dx_j += g/2, dE/dx_i -= g/2, dE/dL_ab += s_a g_b / 2.
// The distance vector is formed in float64; the pair arithmetic runs in
// float32 (pair_fp32) or float64; every sum is float64.
#include "common.cuh"
#include "pair_runs.cuh"

namespace kups {
namespace {

// LJ terms of a run of edges sharing their first particle; the species pair's constants are kept
// while the second particle's species does not change.
template <typename R>
struct LjEval {
  const int32_t *species;
  const double *sigma, *epsilon, *cutoffs;
  int nsp;
  kups_status *status;
  int ti, key;
  R rc2, sig, eps;

  __device__ void load_system(int s) {
    const double rc = cutoffs[s];
    rc2 = (R)(rc * rc);
  }
  __device__ void load_first(int i) { ti = species[i]; }
  __device__ void eval(int64_t edge, int j, double r2d, double &en, double &dedr2) {
    const int k = ti * nsp + species[j];
    if (k != key) {
      key = k;
      sig = (R)sigma[k];
      eps = (R)epsilon[k];
    }
    const R r2 = (R)r2d;
    R e = R(0), d = R(0);
    if (r2 < rc2) {
      const R inv = R(1) / r2;
      const R s2 = sig * sig * inv;
      const R c6 = s2 * s2 * s2;
      e = R(4) * eps * (c6 * c6 - c6);
      d = R(-12) * eps * c6 * (R(2) * c6 - R(1)) * inv;
    }
    if (!isfinite(e) || !isfinite(d)) status_error(status, KUPS_ERR_NONFINITE, edge);
    en = (double)e;
    dedr2 = (double)d;
  }
};

// 264 k particles in 256 systems, 14 M directed edges, float32 pairs: 0.53 ms with PAIRED, 0.82 ms
// without (0.61 and 1.0 ms with shifted and other edges mixed); one thread per edge with six atomics and
// seven float64 warp sums took 2.47 ms.
template <typename R, bool PAIRED>
__global__ void __launch_bounds__(32 * kRunWarps) lj_edges_kernel(PairList p, LjEval<R> ev) {
  ev.key = -1;
  run_pairs<PAIRED>(p, ev, PAIRED && tables_symmetric(ev.sigma, ev.epsilon, ev.nsp));
}

template <bool PAIRED>
int32_t launch_lj_edges(const double *positions, const int32_t *system, const int32_t *species, int64_t n,
                        const double *tril, const double *cutoffs, int32_t s, const double *sigma,
                        const double *epsilon, int32_t nsp, const int32_t *edges, const int32_t *shifts,
                        int64_t n_edges, double *energy, double *grad, double *grad_tril, int32_t pair_fp32,
                        kups_status *status, cudaStream_t stream) {
  if (n < 0 || s < 0 || n_edges < 0 || nsp <= 0) return KUPS_ERR_INVALID;
  if (s > 0) {
    KUPS_CUDA_TRY(cudaMemsetAsync(energy, 0, sizeof(double) * s, stream));
    KUPS_CUDA_TRY(cudaMemsetAsync(grad_tril, 0, sizeof(double) * 6 * s, stream));
  }
  if (n > 0) KUPS_CUDA_TRY(cudaMemsetAsync(grad, 0, sizeof(double) * 3 * n, stream));
  if (n_edges == 0) return KUPS_OK;
  const int64_t per = run_edges_per_warp(n_edges);
  const PairList p{positions, system, n, tril, s, edges, shifts, n_edges, energy, grad, grad_tril, per};
  const unsigned grid = run_blocks(n_edges, per);
  if (pair_fp32) {
    const LjEval<float> ev{species, sigma, epsilon, cutoffs, nsp, status, 0, -1, 0.f, 0.f, 0.f};
    lj_edges_kernel<float, PAIRED><<<grid, 32 * kRunWarps, 0, stream>>>(p, ev);
  } else {
    const LjEval<double> ev{species, sigma, epsilon, cutoffs, nsp, status, 0, -1, 0.0, 0.0, 0.0};
    lj_edges_kernel<double, PAIRED><<<grid, 32 * kRunWarps, 0, stream>>>(p, ev);
  }
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

}  // namespace
}  // namespace kups

using namespace kups;

extern "C" int32_t kups_lj_edges(const double *positions, const int32_t *system,
                                 const int32_t *species, int64_t n, const double *tril,
                                 const double *cutoffs, int32_t s, const double *sigma,
                                 const double *epsilon, int32_t nsp, const int32_t *edges,
                                 const int32_t *shifts, int64_t n_edges, double *energy,
                                 double *grad, double *grad_tril, int32_t pair_fp32,
                                 kups_status *status, void *stream) {
  return launch_lj_edges<false>(positions, system, species, n, tril, cutoffs, s, sigma, epsilon, nsp, edges, shifts,
                                n_edges, energy, grad, grad_tril, pair_fp32, status, (cudaStream_t)stream);
}

extern "C" int32_t kups_lj_edges_paired(const double *positions, const int32_t *system,
                                        const int32_t *species, int64_t n, const double *tril,
                                        const double *cutoffs, int32_t s, const double *sigma,
                                        const double *epsilon, int32_t nsp, const int32_t *edges,
                                        const int32_t *shifts, int64_t n_edges, double *energy,
                                        double *grad, double *grad_tril, int32_t pair_fp32,
                                        kups_status *status, void *stream) {
  const auto launch = nsp <= kTableSpecies ? launch_lj_edges<true> : launch_lj_edges<false>;
  return launch(positions, system, species, n, tril, cutoffs, s, sigma, epsilon, nsp, edges, shifts,
                               n_edges, energy, grad, grad_tril, pair_fp32, status, (cudaStream_t)stream);
}

// Global analytic LJ tail correction (lennard_jones.py:276-340): per system, species counts
// N_a, density N_a N_b / V, t1 = (sigma_ab / rc)^3, t2 = t1^3,
//   E = sum_ab (8/3) pi N_a N_b / V eps_ab sigma_ab^3 (t2 / 3 - t1) mask_ab,
//   P = sum_ab (16/3) pi N_a N_b / V^2 eps_ab sigma_ab^3 (2 t2 / 3 - t1) mask_ab.
// One block per system counts its species in shared memory (atoms grouped by sys_offset).
namespace kups {
namespace {
constexpr int kTailMaxSpecies = 64;
__global__ void lj_tail_kernel(const int32_t *species, const int32_t *sys_offset, const double *tril,
                               const double *sigma, const double *eps, const int32_t *mask, int nsp,
                               const double *cutoff, double *energy, double *pressure, kups_status *status) {
  __shared__ int cnt[kTailMaxSpecies];
  __shared__ int bad;
  const int s = blockIdx.x;
  for (int t = threadIdx.x; t < nsp; t += blockDim.x) cnt[t] = 0;
  if (threadIdx.x == 0) bad = 0;
  __syncthreads();
  const int a0 = sys_offset[s], a1 = sys_offset[s + 1];
  for (int i = a0 + threadIdx.x; i < a1; i += blockDim.x) {
    const int t = species[i];
    if (t < 0 || t >= nsp) bad = 1;
    else atomicAdd(&cnt[t], 1);
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  if (bad) {
    status_error(status, KUPS_ERR_INVALID, s);
    return;
  }
  const double *t6 = tril + 6 * (int64_t)s;
  const double v = fabs(t6[0] * t6[2] * t6[5]);
  const double rc = cutoff[s];
  const double pi = 3.14159265358979323846;
  double e = 0.0, p = 0.0;
  for (int a = 0; a < nsp; ++a)
    for (int b = 0; b < nsp; ++b) {
      const int k = a * nsp + b;
      if (mask != nullptr ? mask[k] == 0 : eps[k] <= 0.0) continue;
      const double sg = sigma[k], s3 = sg * sg * sg, t1 = s3 / (rc * rc * rc), t2 = t1 * t1 * t1;
      const double rho = (double)cnt[a] * (double)cnt[b] / v;
      e += (8.0 / 3.0) * pi * rho * eps[k] * s3 * (t2 / 3.0 - t1);
      p += (16.0 / 3.0) * pi * rho / v * eps[k] * s3 * (t2 / 3.0 * 2.0 - t1);
    }
  if (energy) energy[s] = e;
  if (pressure) pressure[s] = p;
}
}  // namespace
}  // namespace kups

extern "C" int32_t kups_lj_tail_correction(const int32_t *species, const int32_t *sys_offset, int32_t n_systems,
                                           const double *tril, const double *sigma, const double *epsilon,
                                           const int32_t *tail_mask, int32_t n_species, const double *cutoff,
                                           double *energy, double *pressure, kups_status *status, void *stream) {
  if (n_systems < 0 || n_species < 1 || n_species > kups::kTailMaxSpecies) return KUPS_ERR_INVALID;
  if (n_systems == 0) return KUPS_OK;
  kups::lj_tail_kernel<<<n_systems, 256, 0, (cudaStream_t)stream>>>(species, sys_offset, tril, sigma, epsilon,
                                                                    tail_mask, n_species, cutoff, energy, pressure,
                                                                    status);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}
