// Velocity-Verlet / BAOAB building blocks on the reference's float64 particle
// table, for systems too large for the fused shared-memory kernel.
//
// kups_md_kick:  p += F dt_s * scale            (MomentumStep, src/kups/md/integrators.py:217-263)
// kups_md_drift: r += p / m dt_s * scale, then wrap into fractional
//                [-0.5, 0.5)                     (PositionStep + MinimumImageConventionFlow, :104-211)
// kups_md_kick_drift, kups_md_sum_kick: the same in one pass over the particles, the first two one after
//                the other, the last after adding up two gradients and three energies.
// kups_md_thermostat: p = c1 p + sqrt(kT (1 - c1^2)) sqrt(m) eta,
//                c1 = exp(-gamma dt)            (StochasticStep, :330-401); eta from
//                Philox4x32-10 keyed by (seed, particle), counter = step.
// Forces are F = -grad (the potential's dE/dx).
#include <algorithm>

#include "common.cuh"

namespace kups {
namespace {

__global__ void kick_kernel(double *mom, const double *grad, const int32_t *system, const double *dt,
                            double scale, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double h = dt[system[i]] * scale;
  for (int a = 0; a < 3; ++a) mom[3 * i + a] -= grad[3 * i + a] * h;
}

// r + p / m h of a particle of cell L, wrapped; the inverse does not depend on the loads before it
__device__ inline void drift_wrapped(double r[3], const double p[3], double h, const Tril64 &L, const Tril64 &inv) {
  for (int a = 0; a < 3; ++a) r[a] += p[a] * h;
  double f[3];
  row_times_tril64(r, inv, f);
  for (int a = 0; a < 3; ++a) f[a] = (f[a] + 0.5) - floor(f[a] + 0.5) - 0.5;
  row_times_tril64(f, L, r);
}

// grad == nullptr: the drift alone
__global__ void kick_drift_kernel(double *mom, const double *grad, double *pos, const double *mass,
                                  const int32_t *system, const double *dt, const double *tril, double kick,
                                  double drift, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int s = system[i];
  double r[3], p[3];
  for (int a = 0; a < 3; ++a) {
    r[a] = pos[3 * i + a];
    p[a] = mom[3 * i + a];
  }
  if (grad != nullptr) {
    const double h = dt[s] * kick;
    for (int a = 0; a < 3; ++a) {
      p[a] -= grad[3 * i + a] * h;
      mom[3 * i + a] = p[a];
    }
  }
  const Tril64 L = load_tril64(tril + 6 * (int64_t)s);
  drift_wrapped(r, p, dt[s] * drift / mass[i], L, inverse_tril64(L));
  for (int a = 0; a < 3; ++a) pos[3 * i + a] = r[a];
}

// grad = ga + gb, energy = ea + eb + ec per system, and the kick by that gradient
__global__ void sum_kick_kernel(double *mom, double *grad, const double *ga, const double *gb, const int32_t *system,
                                const double *dt, double kick, int64_t n, double *energy, const double *ea,
                                const double *eb, const double *ec, int32_t n_sys) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int64_t s = i; s < n_sys; s += (int64_t)gridDim.x * blockDim.x) energy[s] = (ea[s] + eb[s]) + ec[s];
  if (i >= n) return;
  const double h = dt[system[i]] * kick;
  for (int a = 0; a < 3; ++a) {
    const double g = ga[3 * i + a] + gb[3 * i + a];
    grad[3 * i + a] = g;
    mom[3 * i + a] -= g * h;
  }
}

__global__ void thermostat_kernel(double *mom, const double *mass, const int32_t *system,
                                  const double *dt, const double *kT, const double *friction,
                                  uint64_t seed, uint64_t step, const uint64_t *step_ptr, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (step_ptr != nullptr) step = *step_ptr;
  const int s = system[i];
  const double c1 = exp(-friction[s] * dt[s]);
  const double amp = sqrt(kT[s] * (1.0 - c1 * c1)) * sqrt(mass[i]);
  float eta[4];
  normal4(seed, (uint64_t)i, step, eta);
  for (int a = 0; a < 3; ++a) mom[3 * i + a] = c1 * mom[3 * i + a] + amp * (double)eta[a];
}

}  // namespace
// Threads per block for a per-atom float64 kernel: 256 once there are enough atoms to
// fill every SM, fewer (down to one warp) below that, so that a small system's atoms
// spread over all SMs instead of queueing on the float64 units of a few.
inline unsigned atom_block(int64_t n) {
  const int sms = device_sm_count();
  const int64_t per = (n + sms - 1) / sms;
  return (unsigned)std::min<int64_t>(256, std::max<int64_t>(32, (per + 31) / 32 * 32));
}

}  // namespace kups

using namespace kups;

extern "C" int32_t kups_md_kick(double *momenta, const double *grad, const int32_t *system,
                                const double *dt, double scale, int64_t n, void *stream) {
  if (n < 0) return KUPS_ERR_INVALID;
  if (n == 0) return KUPS_OK;
  kick_kernel<<<(unsigned)((n + atom_block(n) - 1) / atom_block(n)), atom_block(n), 0, (cudaStream_t)stream>>>(momenta, grad, system, dt,
                                                                             scale, n);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

extern "C" int32_t kups_md_drift(double *positions, const double *momenta, const double *masses,
                                 const int32_t *system, const double *dt, const double *tril,
                                 double scale, int64_t n, void *stream) {
  if (n < 0) return KUPS_ERR_INVALID;
  if (n == 0) return KUPS_OK;
  const unsigned threads = atom_block(n);
  kick_drift_kernel<<<(unsigned)((n + threads - 1) / threads), threads, 0, (cudaStream_t)stream>>>(
      const_cast<double *>(momenta), nullptr, positions, masses, system, dt, tril, 0.0, scale, n);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

extern "C" int32_t kups_md_kick_drift(double *momenta, const double *grad, double *positions, const double *masses,
                                      const int32_t *system, const double *dt, const double *tril, double kick_scale,
                                      double drift_scale, int64_t n, void *stream) {
  if (n < 0 || (n > 0 && grad == nullptr)) return KUPS_ERR_INVALID;
  if (n == 0) return KUPS_OK;
  const unsigned threads = atom_block(n);
  kick_drift_kernel<<<(unsigned)((n + threads - 1) / threads), threads, 0, (cudaStream_t)stream>>>(
      momenta, grad, positions, masses, system, dt, tril, kick_scale, drift_scale, n);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

extern "C" int32_t kups_md_sum_kick(double *momenta, double *grad, const double *grad_a, const double *grad_b,
                                    const int32_t *system, const double *dt, double scale, int64_t n, double *energy,
                                    const double *energy_a, const double *energy_b, const double *energy_c,
                                    int32_t n_systems, void *stream) {
  if (n < 0 || n_systems < 0) return KUPS_ERR_INVALID;
  if (n == 0 && n_systems == 0) return KUPS_OK;
  const unsigned threads = atom_block(n);
  sum_kick_kernel<<<(unsigned)std::max<int64_t>(1, (n + threads - 1) / threads), threads, 0, (cudaStream_t)stream>>>(
      momenta, grad, grad_a, grad_b, system, dt, scale, n, energy, energy_a, energy_b, energy_c, n_systems);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

extern "C" int32_t kups_md_thermostat(double *momenta, const double *masses, const int32_t *system,
                                      const double *dt, const double *kT, const double *friction,
                                      uint64_t seed, uint64_t step, int64_t n, void *stream) {
  if (n < 0) return KUPS_ERR_INVALID;
  if (n == 0) return KUPS_OK;
  thermostat_kernel<<<(unsigned)((n + atom_block(n) - 1) / atom_block(n)), atom_block(n), 0, (cudaStream_t)stream>>>(
      momenta, masses, system, dt, kT, friction, seed, step, nullptr, n);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

// The same with the step read from device memory when the kernel runs, so a captured CUDA
// graph that also advances the counter replays successive steps.
extern "C" int32_t kups_md_thermostat_counted(double *momenta, const double *masses, const int32_t *system,
                                              const double *dt, const double *kT, const double *friction,
                                              uint64_t seed, const uint64_t *step, int64_t n, void *stream) {
  if (n < 0 || step == nullptr) return KUPS_ERR_INVALID;
  if (n == 0) return KUPS_OK;
  thermostat_kernel<<<(unsigned)((n + atom_block(n) - 1) / atom_block(n)), atom_block(n), 0, (cudaStream_t)stream>>>(
      momenta, masses, system, dt, kT, friction, seed, 0, step, n);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}
