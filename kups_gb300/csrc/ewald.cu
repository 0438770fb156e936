// Ewald summation: reciprocal-space structure factor, energy, forces and
// cell gradient; self energy; real-space pair terms over an edge list.
//
// Replaces src/kups/potential/classical/ewald.py: EwaldLongRangeInput.kvecs
// (:265-274, k = 2 pi L^-1 n), prefactor (:363-391), _frequency_response /
// _structure_factor_full (:394-439), long_range (:349-360),
// ewald_long_range_energy (:585-601), ewald_self_interaction_energy
// (:277-302), ewald_short_range_energy (:305-325), exclusion_correction_energy
// (:328-346) with coulomb_vacuum_energy (coulomb.py:64-83), and the jax.vjp
// gradients PotentialFromEnergy takes of them (energy.py:264-355).
//
// Reciprocal space, per system s with n_k integer vectors n (zero rows are
// padding, masked like k = 0):
//   theta_ik = 2 pi n_k . f_i  (f = fractional coordinates),
//   S(k) = sum_i q_i (cos, sin)(theta_ik)            [float64 accumulation]
//   P(k) = (2 - [n_x = 0]) 2 pi / V exp(-k^2 / 4 alpha^2) / k^2
//   E = K sum_k P(k) |S(k)|^2
//   dE/dr_i = 2 K q_i sum_k P(k) k (S_s cos - S_c sin)(theta_ik)
//   dE/dL_ab = sum_i f_ia F_ib - sum_k c_k (L^-T k)_a k_b - delta_ab E / L_aa,
//   c_k = K |S|^2 P (-1 / (2 alpha^2) - 2 / k^2)    (F = -dE/dr)
// e^{i theta} is built per atom from per-axis tables e^{2 pi i m f_a},
// m in [-M, M] (the standard Ewald recurrence), so each (atom, k) costs two
// complex products.
#include <algorithm>
#include <mutex>

#include <cooperative_groups.h>

#include "common.cuh"
#include "pair_runs.cuh"

namespace kups {
namespace {

constexpr int kMaxM = 16;            // |n_a| <= 16
constexpr int kTab = 2 * kMaxM + 1;  // table entries per axis
constexpr int kRow = 3 * kTab + 1;  // an atom's tables: 8 banks on from the last atom's, no conflicts of 4 atoms x 4 k
constexpr int kAtomsPerChunk = 32;
constexpr int kKPerBlock = 128;
constexpr int kKPerThread = 2;  // of the structure factor
constexpr int kForceTile = 4 * kKPerBlock;  // k staged at a time by the force kernel
constexpr int kSetupThreads = 512;

struct Coef {
  double p, ck, pad[2];  // P(k), its cell-gradient coefficient per K |S|^2
};

struct RecipSys {
  double inv[6];  // L^-1 (tril)
  double L[6];
  double volume;
  int m[3];       // table half-widths actually used
};

__device__ inline void frac64(const double *inv, const double r[3], double f[3]) {
  f[0] = (r[0] * inv[0] + r[1] * inv[1]) + r[2] * inv[3];
  f[1] = r[1] * inv[2] + r[2] * inv[4];
  f[2] = r[2] * inv[5];
}

// k = 2 pi L^-1 n  (column vector), written for the lower-triangular inverse.
__device__ inline void kvec(const double *inv, const int n[3], double k[3]) {
  const double tp = 6.283185307179586476925286766559;
  k[0] = tp * (inv[0] * n[0]);
  k[1] = tp * (inv[1] * n[0] + inv[2] * n[1]);
  k[2] = tp * (inv[3] * n[0] + inv[4] * n[1] + inv[5] * n[2]);
}

// One block per system: cell, inverse and volume (by the last warp), the largest |n_a| over the
// system's k vectors, and zeros for what the later kernels add to: S(k), energy, cell gradient.
__global__ void __launch_bounds__(kSetupThreads) recip_setup_kernel(const double *tril, const int32_t *kn, int32_t nk,
                                                                    RecipSys *sys, double *sk, double *energy,
                                                                    double *dtril, kups_status *status) {
  __shared__ int mx[3];
  const int i = blockIdx.x;
  if (threadIdx.x < 3) mx[threadIdx.x] = 0;
  __syncthreads();
  int m[3] = {0, 0, 0};
#pragma unroll 4
  for (int k = threadIdx.x; k < nk; k += kSetupThreads)
#pragma unroll
    for (int a = 0; a < 3; ++a) m[a] = max(m[a], abs(kn[((int64_t)i * nk + k) * 3 + a]));
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const int v = __reduce_max_sync(0xffffffffu, m[c]);
    if ((threadIdx.x & 31) == 0) atomicMax(&mx[c], v);
  }
  if (sk != nullptr)
    for (int e = threadIdx.x; e < 2 * nk; e += kSetupThreads) sk[(int64_t)i * nk * 2 + e] = 0.0;
  if (threadIdx.x == 0) energy[i] = 0.0;
  if (threadIdx.x < 6 && dtril != nullptr) dtril[6 * (int64_t)i + threadIdx.x] = 0.0;
  RecipSys r;
  if (threadIdx.x == kSetupThreads - 1) {
    const Tril64 L = load_tril64(tril + 6 * (int64_t)i);
    const Tril64 inv = inverse_tril64(L);
    for (int k = 0; k < 6; ++k) {
      r.L[k] = L.t[k];
      r.inv[k] = inv.t[k];
    }
    r.volume = fabs(L.t[0] * L.t[2] * L.t[5]);
  }
  __syncthreads();
  if (threadIdx.x != kSetupThreads - 1) return;
  for (int a = 0; a < 3; ++a) {
    int v = mx[a];
    if (v > kMaxM) {
      status_error(status, KUPS_ERR_UNSUPPORTED, i);
      v = kMaxM;
    }
    r.m[a] = v;
  }
  sys[i] = r;
}

// The setup's test of |n_a| alone, for callers that need its answer before they use what the rest returns.
__global__ void __launch_bounds__(256) kvec_limit_kernel(const int32_t *kn, int64_t count, int32_t *outside) {
  int beyond = 0;
  for (int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x; e < count; e += (int64_t)gridDim.x * 256)
    beyond += kn[e] > kMaxM || kn[e] < -kMaxM;
  if (beyond != 0) atomicAdd(outside, beyond);
}

// Per-atom tables e^{2 pi i m f_a}, m in [-M_a, M_a], from sincospi of the fundamental and complex
// products (error grows ~linearly in |m| <= 16): thread t < 96 of a block fills axis t / 32 of atom
// c0 + t % 32 (three short chains side by side instead of one of 48 products per atom).
__device__ inline void fill_tables(float2 (*tab)[kRow], const double *pos, int64_t c0, int na, const RecipSys &P) {
  static_assert(kAtomsPerChunk == 32, "one warp per axis");
  const int t = threadIdx.x & 31;
  if (t >= na) return;
  for (int a = threadIdx.x >> 5; a < 3; a += (int)blockDim.x >> 5) {
    const double *r = pos + 3 * (c0 + t), *inv = P.inv;
    const double f = a == 0 ? (r[0] * inv[0] + r[1] * inv[1]) + r[2] * inv[3]
                     : a == 1 ? r[1] * inv[2] + r[2] * inv[4]
                              : r[2] * inv[5];
    float s1, c1;
    // reduce f to [-0.5, 0.5) in float64 first so the float32 argument is small
    const double fr = f - rint(f);
    sincospif((float)(2.0 * fr), &s1, &c1);
    float2 *row = tab[t] + a * kTab + kMaxM;
    row[0] = make_float2(1.f, 0.f);
    float cr = 1.f, ci = 0.f;
    const int m_max = P.m[a];
    for (int m = 1; m <= m_max; ++m) {
      const float nr = fmaf(cr, c1, -__fmul_rn(ci, s1));
      const float ni = fmaf(cr, s1, __fmul_rn(ci, c1));
      cr = nr;
      ci = ni;
      row[m] = make_float2(cr, ci);
      row[-m] = make_float2(cr, -ci);
    }
  }
}

// Row of component n in an axis' table (the setup refuses |n| > kMaxM: any row of the table then)
__device__ inline int table_row(int n) { return min(max(n, -kMaxM), kMaxM) + kMaxM; }

// Complex products of the tables' entries.  Which product of each sum is rounded is written out: the
// phases of S(k) and of the forces are the same to the bit, whatever surrounds them.
__device__ inline float2 phase_xy(float2 x, float2 y) {
  return make_float2(fmaf(x.x, y.x, -__fmul_rn(x.y, y.y)), fmaf(x.y, y.x, __fmul_rn(x.x, y.y)));
}
__device__ inline float2 phase_xyz(float2 a, float2 z) {
  return make_float2(fmaf(a.x, z.x, -__fmul_rn(a.y, z.y)), fmaf(a.x, z.y, __fmul_rn(a.y, z.x)));
}

// P(k) and the coefficient of K |S(k)|^2 in the cell gradient, 0 for k = 0.
__device__ inline Coef prefactor(const RecipSys &P, const int *nv, double a) {
  const double tp = 6.283185307179586476925286766559;
  const int n3[3] = {nv[0], nv[1], nv[2]};
  double kv[3];
  kvec(P.inv, n3, kv);
  const double k2 = kv[0] * kv[0] + kv[1] * kv[1] + kv[2] * kv[2];
  Coef c{0.0, 0.0, {0.0, 0.0}};
  if (k2 > 0.0) {
    c.p = (2.0 - (n3[0] == 0 ? 1.0 : 0.0)) * tp / P.volume * exp(-k2 / (4.0 * a * a)) / k2;
    c.ck = c.p * (-1.0 / (2.0 * a * a) - 2.0 / k2);
  }
  return c;
}

// S(k): grid (k tiles, atom chunks, systems).  Each block stages the tables of 32 atoms
// in shared memory; each thread owns two k and accumulates the chunk in float32, then adds it to S in
// float64.  Latency bounds it (of a table's fill, then of the gathers; without the additions it takes
// 15.1 us of 15.7).  The warp that has no table to fill forms
// prefactors P(k) meanwhile: their float64 exponentials and divisions were 10 us of a launch of their own.
// 2800 k, 4000 atoms: 16.6 us with one k per thread and a thread per atom's tables, now 15.7 (17.0 with one
// k per thread, 17.7 with four).
__global__ void __launch_bounds__(kKPerBlock) structure_factor_kernel(const double *pos, const double *q,
                                                                      const int32_t *sys_offset, const int32_t *kn,
                                                                      int32_t nk, const RecipSys *sysp,
                                                                      const double *alpha, Coef *coef, double *sk,
                                                                      double *grad) {
  __shared__ float2 tab[kAtomsPerChunk][kRow];
  __shared__ float qs[kAtomsPerChunk];
  const int s = blockIdx.z;
  const RecipSys &P = sysp[s];
  const int kb = blockIdx.x * kKPerBlock * kKPerThread + threadIdx.x;
  const int a0 = sys_offset[s], a1 = sys_offset[s + 1];
  const int c0 = a0 + blockIdx.y * kAtomsPerChunk;
  if (c0 >= a1) return;
  const int na = min(kAtomsPerChunk, a1 - c0);
  fill_tables(tab, pos, c0, na, P);
  if (threadIdx.x >= 96)  // the warp without a table: the prefactors of 32 k of the tile for some chunks
    for (int j = blockIdx.y; j < kKPerBlock * kKPerThread / 32; j += (a1 - a0 + kAtomsPerChunk - 1) / kAtomsPerChunk) {
      const int64_t k = (int64_t)blockIdx.x * kKPerBlock * kKPerThread + 32 * j + (threadIdx.x - 96);
      if (k < nk) coef[(int64_t)s * nk + k] = prefactor(P, kn + ((int64_t)s * nk + k) * 3, alpha[s]);
    }
  if (threadIdx.x < na) qs[threadIdx.x] = (float)q[c0 + threadIdx.x];
  // the force kernel adds its k-range partials into grad: zero this chunk's rows first
  if (blockIdx.x == 0 && grad != nullptr && threadIdx.x < 3 * na) grad[3 * (int64_t)c0 + threadIdx.x] = 0.0;
  __syncthreads();
  int row[kKPerThread][3];
  float sc[kKPerThread], ss[kKPerThread];
#pragma unroll
  for (int j = 0; j < kKPerThread; ++j) {
    const int *nv = kn + ((int64_t)s * nk + min(kb + j * kKPerBlock, nk - 1)) * 3;
#pragma unroll
    for (int a = 0; a < 3; ++a) row[j][a] = a * kTab + table_row(nv[a]);
    sc[j] = ss[j] = 0.f;
  }
  for (int t = 0; t < na; ++t)
#pragma unroll
    for (int j = 0; j < kKPerThread; ++j) {
      const float2 e = phase_xyz(phase_xy(tab[t][row[j][0]], tab[t][row[j][1]]), tab[t][row[j][2]]);
      sc[j] = fmaf(qs[t], e.x, sc[j]);
      ss[j] = fmaf(qs[t], e.y, ss[j]);
    }
#pragma unroll
  for (int j = 0; j < kKPerThread; ++j) {
    const int64_t k = kb + j * kKPerBlock;
    if (k >= nk) break;
    atomicAdd(&sk[((int64_t)s * nk + k) * 2], (double)sc[j]);
    atomicAdd(&sk[((int64_t)s * nk + k) * 2 + 1], (double)ss[j]);
  }
}

// K sum_k P(k) |S(k)|^2 of given structure factors, one warp per block: the float64 exponentials and
// divisions of 32 k each spread over many SMs.
__global__ void recip_energy_kernel(const int32_t *kn, int32_t nk, const double *alpha, const RecipSys *sysp,
                                    const double *sk, double ke, double *energy) {
  const int s = blockIdx.y;
  const int64_t k = blockIdx.x * 32 + threadIdx.x;
  double e = 0.0;
  if (k < nk) {
    const double sc = sk[((int64_t)s * nk + k) * 2], ss = sk[((int64_t)s * nk + k) * 2 + 1];
    e = ke * prefactor(sysp[s], kn + ((int64_t)s * nk + k) * 3, alpha[s]).p * (sc * sc + ss * ss);
  }
  e = warp_sum(e);
  if (threadIdx.x == 0) atomicAdd(&energy[s], e);  // zeroed by the setup
}

// dE/dr_i for every atom of every system (four threads per atom; k coefficients staged through shared
// memory), plus the sum_i f_ia F_ib part of dE/dL.  The blocks of the first atom chunk also add the
// energy of their k and its part of the cell gradient, from the S(k) they stage.
// Bound by shared memory and latency: with 32 bytes per k and a phase from three tables each time, 14
// wavefronts for 32 terms; a k is 12 bytes and the x y phase is kept while n_z runs: 6.
// 4000 atoms and 2800 k: 25.5 us and 10.5 for the launch that formed coefficients and energy, now 25.7
// with both.  (Two atoms per thread take 5, but leave 1.6 warps per
// scheduler: 28 us.)
constexpr int kForceThreads = kAtomsPerChunk * 4;

__global__ void __launch_bounds__(kForceThreads) recip_force_kernel(
    const double *pos, const double *q, const int32_t *sys_offset, const int32_t *kn, int32_t nk, const RecipSys *sysp,
    const Coef *coef, const double *sk, double ke, double *energy, double *grad, double *dtril,
    int kblocks_per_split) {
  __shared__ float2 tab[kAtomsPerChunk][kRow];
  __shared__ float2 kc[kForceTile];    // P S_c, P S_s
  __shared__ uint32_t kz[kForceTile];  // rows of the x, y and z tables from their starts, a byte each
  __shared__ float gsum[kAtomsPerChunk][3];
  __shared__ double red[40];
  const int s = blockIdx.y;
  const int a0 = sys_offset[s], a1 = sys_offset[s + 1];
  const int c0 = a0 + blockIdx.x * kAtomsPerChunk;
  if (c0 >= a1) return;
  const int na = min(kAtomsPerChunk, a1 - c0);
  const RecipSys &P = sysp[s];
  const int t = threadIdx.x, sub = t & 3, atom = t >> 2;  // every fourth k of an atom
  fill_tables(tab, pos, c0, na, P);
  // gradient in fractional components: dE/df_a = sum_k 2 K q P 2 pi n_a (Ss c - Sc s)
  float g[3] = {0.f, 0.f, 0.f};
  const float2 *row = tab[atom];
  double e = 0.0, fw[6] = {0, 0, 0, 0, 0, 0};
  // this block's share of the k vectors (blockIdx.z); partials are added into grad
  const int kbeg = blockIdx.z * kblocks_per_split * kKPerBlock;
  const int kfin = min(nk, kbeg + kblocks_per_split * kKPerBlock);
  for (int kb = kbeg; kb < kfin; kb += kForceTile) {
    __syncthreads();
    const int kend = min(kForceTile, kfin - kb);
#pragma unroll 4
    for (int j = threadIdx.x; j < kend; j += kForceThreads) {
      {
        const int64_t k = (int64_t)s * nk + kb + j;
        const int n3[3] = {kn[3 * k], kn[3 * k + 1], kn[3 * k + 2]};
        const double p = coef[k].p, sc = sk[2 * k], ss = sk[2 * k + 1];
        kc[j] = make_float2((float)(p * sc), (float)(p * ss));
        kz[j] = (uint32_t)(table_row(n3[0]) | table_row(n3[1]) << 8 | table_row(n3[2]) << 16);
        if (blockIdx.x == 0) {
          const double s2 = sc * sc + ss * ss, ek = ke * p * s2;
          e += ek;
          if (dtril != nullptr) {
            const double *iv = P.inv;
            const double ck = ke * s2 * coef[k].ck;
            double kv[3];
            kvec(iv, n3, kv);
            // u = L^-T k: (L^-T)_ab = inv_ba
            const double u0 = iv[0] * kv[0] + iv[1] * kv[1] + iv[3] * kv[2];
            const double u1 = iv[2] * kv[1] + iv[4] * kv[2];
            const double u2 = iv[5] * kv[2];
            fw[0] -= ck * u0 * kv[0] + ek * iv[0];
            fw[1] -= ck * u1 * kv[0];
            fw[2] -= ck * u1 * kv[1] + ek * iv[2];
            fw[3] -= ck * u2 * kv[0];
            fw[4] -= ck * u2 * kv[1];
            fw[5] -= ck * u2 * kv[2] + ek * iv[5];
          }
        }
      }
    }
    __syncthreads();
    uint32_t last = 0xffffffffu;
    float2 xy = make_float2(1.f, 0.f);
#pragma unroll 4
    for (int j = sub; j < kend; j += 4) {
      const uint32_t z = kz[j];
      const float2 c = kc[j];
      if ((z ^ last) & 0xffffu) xy = phase_xy(row[z & 0xffu], row[kTab + (z >> 8 & 0xffu)]);  // n_z runs fastest
      last = z;
      // the bytes as float32: 2^23 + byte by its bits, less 2^23 + kMaxM
      const float nx = __uint_as_float(0x4b000000u | (z & 0xffu)) - (8388608.f + kMaxM),
                  ny = __uint_as_float(0x4b000000u | (z >> 8 & 0xffu)) - (8388608.f + kMaxM),
                  nz = __uint_as_float(0x4b000000u | z >> 16) - (8388608.f + kMaxM);
      const float2 ph = phase_xyz(xy, row[2 * kTab + (z >> 16)]);
      const float w = fmaf(c.y, ph.x, -__fmul_rn(c.x, ph.y));  // P (S_s cos - S_c sin)
      g[0] = fmaf(w, nx, g[0]);
      g[1] = fmaf(w, ny, g[1]);
      g[2] = fmaf(w, nz, g[2]);
    }
  }
  if (blockIdx.x == 0) {
    const double et = block_sum(e, red);
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(&energy[s], et);
  }
  // reduce the 4 lanes of an atom
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    for (int o = 1; o < 4; o <<= 1) g[a] += __shfl_xor_sync(0xffffffffu, g[a], o);
    if (sub == 0) gsum[atom][a] = g[a];
  }
  __syncthreads();
  if (t < na) {  // float64, by one warp: a quarter of every warp took four times as long
    const int i = c0 + t;
    const double tp = 6.283185307179586476925286766559;
    const double scale = 2.0 * ke * q[i] * tp;
    // dE/df -> dE/dr: r = f L  =>  f = r L^-1, dE/dr_b = sum_a dE/df_a (L^-1)_{ba}
    const double df[3] = {scale * gsum[t][0], scale * gsum[t][1], scale * gsum[t][2]};
    const double *iv = P.inv;
    const double gr[3] = {df[0] * iv[0], df[0] * iv[1] + df[1] * iv[2],
                          df[0] * iv[3] + df[1] * iv[4] + df[2] * iv[5]};
    if (kblocks_per_split > 0) {  // k-range partials; the structure-factor kernel zeroed grad
      atomicAdd(&grad[3 * (int64_t)i], gr[0]);
      atomicAdd(&grad[3 * (int64_t)i + 1], gr[1]);
      atomicAdd(&grad[3 * (int64_t)i + 2], gr[2]);
    } else {  // no k vectors (no structure-factor launch): write the zero gradient
      grad[3 * (int64_t)i] = gr[0];
      grad[3 * (int64_t)i + 1] = gr[1];
      grad[3 * (int64_t)i + 2] = gr[2];
    }
    if (dtril != nullptr) {
      const double r[3] = {pos[3 * i], pos[3 * i + 1], pos[3 * i + 2]};
      double fi[3];
      frac64(P.inv, r, fi);
      // sum_i f_ia F_ib, F = -dE/dr
      fw[0] -= fi[0] * gr[0];
      fw[1] -= fi[1] * gr[0];
      fw[2] -= fi[1] * gr[1];
      fw[3] -= fi[2] * gr[0];
      fw[4] -= fi[2] * gr[1];
      fw[5] -= fi[2] * gr[2];
    }
  }
  if (dtril != nullptr && (blockIdx.x == 0 || t < 32)) {  // other blocks: the first warp has all of it
    for (int c = 0; c < 6; ++c) {
      const double v = blockIdx.x == 0 ? block_sum(fw[c], red) : warp_sum(fw[c]);
      if (blockIdx.x == 0) __syncthreads();
      if (threadIdx.x == 0) atomicAdd(&dtril[6 * (int64_t)s + c], v);
    }
  }
}

__global__ void self_energy_kernel(const double *q, const int32_t *sys_offset, const double *alpha,
                                   double ke, double *energy) {
  __shared__ double red[40];
  const int s = blockIdx.x;
  double acc = 0.0;
  for (int i = sys_offset[s] + threadIdx.x; i < sys_offset[s + 1]; i += blockDim.x) acc += q[i] * q[i];
  const double t = block_sum(acc, red);
  if (threadIdx.x == 0) energy[s] = -t * alpha[s] / sqrt(3.14159265358979323846) * ke;
}

// ---------------------------------------------------------------- real space
// Per directed edge (i, j, shift), d = x_j - x_i + s @ L, r = |d|:
//   LJ    4 eps (c6^2 - c6) [r^2 < rc_lj^2]
//   EWALD K q_i q_j erfc(alpha r) / r [r < rc_ew]
//   VACUUM (exclusion correction, subtracted) K q_i q_j / r, no cutoff
// Each term is summed / 2 per system (directed edges), gradients as in
// kups_lj_edges.  Float64 distance; pair arithmetic in float64, one reciprocal square
// root per pair in place of the divisions by r, r^2 and r^3.
struct EwaldPairEval {
  const int32_t *species;
  const double *q, *lj_sigma, *lj_eps, *rc_lj, *alpha, *rc_ew;
  int nsp, terms;
  double ke;
  int ti, key;
  double sig2, eps4, rc2_lj, al, rcew, rc2_ew, qi;

  __device__ void load_system(int s) {
    if (terms & 1) rc2_lj = rc_lj[s] * rc_lj[s];
    if (terms & 2) {
      al = alpha[s];
      rcew = rc_ew[s];
      rc2_ew = rcew * fabs(rcew);  // no pair is within a negative cutoff
    }
  }
  __device__ void load_first(int i) {
    if (terms & 1) ti = species[i];
    if (terms & 6) qi = q[i] * ke;
  }
  __device__ void eval(int64_t, int j, double r2, double &en, double &dedr2) {
    en = 0.0;
    dedr2 = 0.0;
    const double ir = rsqrt(r2), inv = ir * ir;
    if ((terms & 1) && r2 < rc2_lj) {
      const int k = ti * nsp + species[j];
      if (k != key) {
        key = k;
        sig2 = lj_sigma[k] * lj_sigma[k];
        eps4 = 4.0 * lj_eps[k];
      }
      const double s2 = sig2 * inv, c6 = s2 * s2 * s2;
      en += eps4 * (c6 * c6 - c6);
      dedr2 -= 3.0 * eps4 * c6 * (2.0 * c6 - 1.0) * inv;
    }
    if (terms & 6) {
      const double qq = qi * q[j] * ir;  // K q_i q_j / r
      // r < rc_ew as the root of r^2 decides it; the root itself only where r^2 leaves that open
      if ((terms & 2) && r2 < rc2_ew * (1.0 + 1e-14) && (r2 < rc2_ew * (1.0 - 1e-14) || sqrt(r2) < rcew)) {
        const double r = r2 * ir, er = erfc(al * r);
        en += qq * er;
        dedr2 -= 0.5 * qq * (er * inv + 2.0 * al * 0.56418958354775628695 * exp(-al * al * r2) * ir);
      }
      if (terms & 4) {
        en -= qq;
        dedr2 += 0.5 * qq * inv;
      }
    }
  }
};

// 4000 ions, 1.8 M directed edges, LJ + Ewald: 0.38 ms with PAIRED, 0.70 ms without; a thread per
// edge with thirteen atomics (seven of them on one system's sums) took 12.3 ms.
template <bool PAIRED>
__global__ void __launch_bounds__(32 * kRunWarps) pair_edges_kernel(PairList p, EwaldPairEval ev) {
  ev.key = -1;
  const bool symmetric = PAIRED && ((ev.terms & 1) == 0 || tables_symmetric(ev.lj_sigma, ev.lj_eps, ev.nsp));
  run_pairs<PAIRED>(p, ev, symmetric);
}

template <bool PAIRED>
int32_t launch_pair_edges(const double *positions, const int32_t *system, const int32_t *species,
                          const double *charges, int64_t n, const double *tril, int32_t n_systems,
                          const double *lj_sigma, const double *lj_epsilon, int32_t n_species,
                          const double *lj_cutoff, const double *alpha, const double *ewald_cutoff,
                          double coulomb_k, int32_t terms, const int32_t *edges, const int32_t *shifts,
                          int64_t n_edges, double *energy, double *grad, double *grad_tril, cudaStream_t stream) {
  if (n < 0 || n_systems < 0 || n_edges < 0 || (terms & ~7) != 0) return KUPS_ERR_INVALID;
  if ((terms & 1) && (lj_sigma == nullptr || n_species <= 0)) return KUPS_ERR_INVALID;
  if (n_systems > 0) {
    KUPS_CUDA_TRY(cudaMemsetAsync(energy, 0, sizeof(double) * n_systems, stream));
    if (grad_tril) KUPS_CUDA_TRY(cudaMemsetAsync(grad_tril, 0, sizeof(double) * 6 * n_systems, stream));
  }
  if (n > 0) KUPS_CUDA_TRY(cudaMemsetAsync(grad, 0, sizeof(double) * 3 * n, stream));
  if (n_edges == 0) return KUPS_OK;
  const int64_t per = run_edges_per_warp(n_edges);
  const PairList p{positions, system, n, tril, n_systems, edges, shifts, n_edges, energy, grad, grad_tril, per};
  EwaldPairEval ev{};
  ev.species = species;
  ev.q = charges;
  ev.lj_sigma = lj_sigma;
  ev.lj_eps = lj_epsilon;
  ev.rc_lj = lj_cutoff;
  ev.alpha = alpha;
  ev.rc_ew = ewald_cutoff;
  ev.nsp = n_species;
  ev.terms = terms;
  ev.ke = coulomb_k;
  pair_edges_kernel<PAIRED><<<run_blocks(n_edges, per), 32 * kRunWarps, 0, stream>>>(p, ev);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

// Real-space Lennard-Jones + Ewald forces of systems whose cell widths are all at
// least twice the larger cutoff, so that every pair within a cutoff is its minimum
// image and each ordered pair (i, j != i) is counted once: the edge set of
// neighbour_list at rc with the energies of lennard_jones_energy /
// ewald_short_range_energy (each pair term halved over the two directions), with no
// stored list.  A block owns 16 atoms; each half-warp holds all 16 (lane % 16 = atom)
// and the 32 half-warps split the partners j, so a half-warp reads one partner at a
// time (a broadcast from L1).  The difference is formed in float64, the minimum image
// and pair terms in float32, the 32 partial forces are summed in a fixed order through
// shared memory and the energy is float64.
constexpr int kRealBatch = 128;  // pairs whose forces a warp keeps before their atoms add them up
constexpr int kRealAtoms = 16, kRealWarps = 16, kRealStreams = 2 * kRealWarps;

__global__ void __launch_bounds__(32 * kRealWarps) real_allpairs_kernel(
    const double *pos, const double *q, const int32_t *species, const int32_t *sys_offset, const double *tril,
    const double *lj_sigma, const double *lj_eps, int nsp, const double *rc_lj, const double *alpha,
    const double *rc_ew, double ke, int terms, double *energy, double *grad, kups_status *status) {
  __shared__ float2 ljt[64];
  __shared__ float part[kRealStreams][kRealAtoms][3];
  __shared__ double red[40];
  const int s = blockIdx.y;
  const int a0 = sys_offset[s], n = sys_offset[s + 1] - a0;
  if ((int)blockIdx.x * kRealAtoms >= n) return;  // uniform over the block
  // cell, inverse and widths once per block (float64 is scarce on this part)
  __shared__ float cellf[12];
  __shared__ int refused;
  if (threadIdx.x == 0) {
    const Tril64 L64 = load_tril64(tril + 6 * (int64_t)s);
    const Tril64 I64 = inverse_tril64(L64);
    double w[3];
    perpendicular_widths64(L64, w);
    const double rm = fmax((terms & 1) ? rc_lj[s] : 0.0, (terms & 2) ? rc_ew[s] : 0.0);
    refused = fmin(w[0], fmin(w[1], w[2])) < 2.0 * rm;
    if (refused) status_error(status, KUPS_ERR_UNSUPPORTED, s);
    for (int k = 0; k < 6; ++k) {
      cellf[k] = (float)L64.t[k];
      cellf[6 + k] = (float)I64.t[k];
    }
  }
  __syncthreads();
  if (refused) return;
  const double rlj = (terms & 1) ? rc_lj[s] : 0.0, rew = (terms & 2) ? rc_ew[s] : 0.0;
  const double rmax = fmax(rlj, rew);
  float L[6], I[6];
  for (int k = 0; k < 6; ++k) {
    L[k] = cellf[k];
    I[k] = cellf[6 + k];
  }
  if ((terms & 1) && nsp * nsp <= 64)
    for (int k = threadIdx.x; k < nsp * nsp; k += blockDim.x) {
      const double sg = lj_sigma[k];
      ljt[k] = make_float2((float)(sg * sg), (float)(4.0 * lj_eps[k]));
    }
  __syncthreads();
  const float rc2_lj = (float)(rlj * rlj), rc2_ew = (float)(rew * rew), rc2 = (float)(rmax * rmax);
  const float al = (terms & 2) ? (float)alpha[s] : 0.f;
  const float two_al_rsqrtpi = 2.0f * al * 0.56418958354775628695f;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int slot = lane & (kRealAtoms - 1), stream_id = warp * 2 + (lane >> 4);
  const int il = blockIdx.x * kRealAtoms + slot;
  const bool act = il < n;
  const int gi = a0 + (act ? il : 0);
  const double xi = pos[3 * (int64_t)gi], yi = pos[3 * (int64_t)gi + 1], zi = pos[3 * (int64_t)gi + 2];
  const float qi = (float)(q[gi] * ke);
  const int ti = (terms & 1) ? species[gi] : 0;
  float fx = 0.f, fy = 0.f, fz = 0.f;  // dE/dx_i, this warp's partners
  float ef = 0.f;
  const int per = (n + kRealStreams - 1) / kRealStreams;
  const int j0 = stream_id * per, j1 = min(n, j0 + per);
  for (int j = j0; j < j1; ++j) {
    const int gj = a0 + j;
    const float d0 = (float)(pos[3 * (int64_t)gj] - xi), d1 = (float)(pos[3 * (int64_t)gj + 1] - yi),
                d2 = (float)(pos[3 * (int64_t)gj + 2] - zi);
    float f0 = (d0 * I[0] + d1 * I[1]) + d2 * I[3], f1 = d1 * I[2] + d2 * I[4], f2 = d2 * I[5];
    f0 -= rintf(f0);
    f1 -= rintf(f1);
    f2 -= rintf(f2);
    const float dx = (f0 * L[0] + f1 * L[1]) + f2 * L[3], dy = f1 * L[2] + f2 * L[4], dz = f2 * L[5];
    const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
    if (r2 >= rc2 || j == il || !act) continue;
    float dedr2 = 0.f;  // dE/d(r^2) of the pair
    const float ir = rsqrtf(r2);
    if ((terms & 1) && r2 < rc2_lj) {
      const float2 c = ljt[ti * nsp + species[gj]];
      const float inv = ir * ir, s2 = c.x * inv, c6 = s2 * s2 * s2;
      ef += c.y * (c6 * c6 - c6);
      dedr2 += -0.5f * c.y * c6 * (12.f * c6 - 6.f) * inv;
    }
    if ((terms & 2) && r2 < rc2_ew) {
      const float r = r2 * ir, qq = qi * (float)q[gj];
      const float er = erfc_cheb(al * r);
      ef += qq * er * ir;
      dedr2 += 0.5f * ir * qq * (-er * ir * ir - two_al_rsqrtpi * __expf(-al * al * r2) * ir);
    }
    // d = x_j - x_i: dE/dx_i = -2 dE/d(r^2) d for this ordered pair (both halves)
    fx = fmaf(-2.f * dedr2, dx, fx);
    fy = fmaf(-2.f * dedr2, dy, fy);
    fz = fmaf(-2.f * dedr2, dz, fz);
  }
  part[stream_id][slot][0] = fx;
  part[stream_id][slot][1] = fy;
  part[stream_id][slot][2] = fz;
  __syncthreads();
  if (threadIdx.x < kRealAtoms && act) {
    float gx = 0.f, gy = 0.f, gz = 0.f;
    for (int k = 0; k < kRealStreams; ++k) {
      gx += part[k][slot][0];
      gy += part[k][slot][1];
      gz += part[k][slot][2];
    }
    grad[3 * (int64_t)gi] = gx;
    grad[3 * (int64_t)gi + 1] = gy;
    grad[3 * (int64_t)gi + 2] = gz;
  }
  const double esum = block_sum(0.5 * (double)ef, red);
  if (threadIdx.x == 0) atomicAdd(&energy[s], esum);
}

// ---------------------------------------------------------------- packed real space
// The all-pairs kernel above forms every pair difference in float64 (three float64
// subtractions per pair test, slow on this part) and runs the LJ + erfc branch for a
// whole warp whenever any lane has a partner inside the cutoff (~11 % of pair tests
// in a dense melt, so ~98 % of warp iterations at ~11 % lane use).  The packed path:
//  * a pack kernel stores each coordinate as a float pair hi = fl(x), lo = fl(x - hi);
//    a difference (hj - hi) + (lj - li) then carries float32 relative error in d
//    itself (the rounding of hj - hi is relative to the result), with no float64;
//  * the force kernel tests 32 partners per pass into a per-lane hit mask, in float32
//    fractional coordinates and the cell's metric, two partners per instruction (17
//    instructions each, 34 for the difference of the hi / lo pairs); where a partner is
//    closer to the cutoff than the rounding of either test, the pass is tested again by
//    the pairs themselves, so the hits are exactly theirs;
//  * the hits of a warp are queued and evaluated one per lane; their forces go through
//    shared memory to the lane of their atom, which adds them up in order (shared-memory
//    atomics to the same few addresses were more than half of the instructions).
// 4000 ions, cutoff 12 in a 40 cube: 77 us, now 43, bound by issue and the latency of 26 warps per SM.
// Pair terms, the minimum image and the fixed-order reduction are those of the
// all-pairs kernel.
// Packed arrays are indexed by system * max_atoms + local index (inside the workspace
// for any sys_offset); a system above max_atoms is refused.
// What the force kernel needs of a system, formed once per call in float64 (a few hundred float64
// operations of one thread: 250 blocks forming them for themselves started 3 us late each).
struct RealSys {
  float L[6], I[6];             // cell and inverse
  float g00, g01, g02, g11, g12, g22;  // |f L|^2 of fractional f, the mixed terms doubled
  float rc2_lj, rc2_ew, rc2, alpha, ke;
  float margin;                 // |r2 - rc2| below which the fractional test does not decide
  int refused;
};

// Workspace of the packed path: hi, lo and fractional coordinates of every atom (one read past the end
// of the last by a pass of 32 partners), and the systems' constants.
struct RealWork {
  float4 *hi, *lo, *frac;
  RealSys *sys;
  size_t bytes;
};

inline RealWork real_work(char *base, int32_t n_systems, int32_t max_atoms) {
  auto align = [](size_t x) { return (x + 255) & ~size_t(255); };
  const size_t rows = align((size_t)n_systems * (size_t)max_atoms * sizeof(float4));
  RealWork w;
  w.hi = (float4 *)base;
  w.lo = (float4 *)(base + rows);
  w.frac = (float4 *)(base + 2 * rows);
  w.sys = (RealSys *)(base + 3 * rows + 32 * sizeof(float4));
  w.bytes = 3 * rows + 32 * sizeof(float4) + align(sizeof(RealSys) * (size_t)n_systems);
  return w;
}

// By threads 0 (inverse) and 32 (widths) of a block: two chains of float64 divisions side by side.
__device__ inline void set_real_system(RealSys &r, const Tril64 &L64, double rlj, double rew, double alpha, double ke) {
  const double rmax = fmax(rlj, rew), *t = L64.t;
  if (threadIdx.x == 0) {
    const Tril64 I64 = inverse_tril64(L64);
    for (int k = 0; k < 6; ++k) {
      r.L[k] = (float)t[k];
      r.I[k] = (float)I64.t[k];
    }
    r.rc2_lj = (float)(rlj * rlj);
    r.rc2_ew = (float)(rew * rew);
    r.rc2 = (float)(rmax * rmax);
    r.alpha = (float)alpha;
    r.ke = (float)ke;
  } else if (threadIdx.x == 32) {
    double w[3];
    perpendicular_widths64(L64, w);
    const double wmin = fmin(w[0], fmin(w[1], w[2]));
    const double g00 = t[0] * t[0], g11 = t[1] * t[1] + t[2] * t[2], g22 = t[3] * t[3] + t[4] * t[4] + t[5] * t[5];
    const double g01 = 2.0 * t[0] * t[1], g02 = 2.0 * t[0] * t[3], g12 = 2.0 * (t[1] * t[3] + t[2] * t[4]);
    r.refused = wmin < 2.0 * rmax;
    r.g00 = (float)g00;
    r.g01 = (float)g01;
    r.g02 = (float)g02;
    r.g11 = (float)g11;
    r.g12 = (float)g12;
    r.g22 = (float)g22;
    // Both tests work on |f_a| <= 1/2 with errors below 4e-7 in f and 2^-21 of the terms' sizes in r^2,
    // together under 5e-6 of S = sum |g| / 4; twice that decides.  Where a cell is so narrow that a
    // partner at f = 1/2 could be within the cutoff, the two may take different images of it: never then.
    const double size = 0.25 * (g00 + fabs(g01) + fabs(g02) + g11 + fabs(g12) + g22);
    r.margin = wmin < 2.0 * rmax * (1.0 + 1e-4) ? INFINITY : (float)(1e-5 * size);
  }
}

// 1 / x to about 1e-14: a float32 reciprocal and one Newton step (float64 divisions are slow here).
__device__ inline double reciprocal64(double x) {
  const double y = (double)(1.0f / (float)x);
  return y * fma(-x, y, 2.0);
}

__global__ void __launch_bounds__(256) real_pack_kernel(const double *pos, const double *q, const int32_t *species,
                                                        const int32_t *sys_offset, const double *tril,
                                                        const double *rc_lj, const double *alpha, const double *rc_ew,
                                                        double ke, int terms, int max_atoms, RealWork w,
                                                        double *energy, kups_status *status) {
  const int s = blockIdx.y;
  const int a0 = sys_offset[s], n = sys_offset[s + 1] - a0;
  const Tril64 L = load_tril64(tril + 6 * (int64_t)s);
  if (blockIdx.x == gridDim.x - 1) {  // the block after the last atom
    __shared__ RealSys made;
    set_real_system(made, L, (terms & 1) ? rc_lj[s] : 0.0, (terms & 2) ? rc_ew[s] : 0.0, (terms & 2) ? alpha[s] : 0.0,
                    ke);
    __syncthreads();
    if (threadIdx.x != 0) return;
    w.sys[s] = made;
    if (!(terms & 8)) energy[s] = 0.0;
    if (n > max_atoms) status_error(status, KUPS_ERR_INVALID, s);
    else if (n > 0 && made.refused) status_error(status, KUPS_ERR_UNSUPPORTED, s);
    return;
  }
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (n > max_atoms || k >= n) return;
  const int64_t g = a0 + k, p = (int64_t)s * max_atoms + k;
  float h[3], l[3];
  double x[3], f[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    x[a] = pos[3 * g + a];
    h[a] = (float)x[a];
    l[a] = (float)(x[a] - (double)h[a]);
  }
  // fractional coordinates to 1e-14 or so, then in [-1/2, 1/2]: f L = x solved from the last component
  f[2] = x[2] * reciprocal64(L.t[5]);
  f[1] = (x[1] - f[2] * L.t[4]) * reciprocal64(L.t[2]);
  f[0] = (x[0] - f[1] * L.t[1] - f[2] * L.t[3]) * reciprocal64(L.t[0]);
#pragma unroll
  for (int a = 0; a < 3; ++a) f[a] -= rint(f[a]);
  w.hi[p] = make_float4(h[0], h[1], h[2], (float)q[g]);
  w.lo[p] = make_float4(l[0], l[1], l[2], __int_as_float((terms & 1) ? species[g] : 0));
  w.frac[p] = make_float4((float)f[0], (float)f[1], (float)f[2], 0.f);
}

// A block's 16 warps are a cluster of four CTAs, whose forces the first adds up through distributed
// shared memory: 4000 ions are 250 blocks, one or two per SM, or 1000 CTAs, six or seven (48 us and 43).
// Ten steps in us with 1 / 2 / 4 / 8 CTAs: 216 ions 316 / 316 / 316 / 315, 1000 ions 354 / 337 / 336 / 339,
// 2000 ions 455 / 421 / 410 / 421, 4000 ions 890 / 865 / 811 / 887, 8000 ions 2178 / 2083 / 2121 / 2528, 32
// systems of 216 ions 500 / 479 / 486 / 573, 16 of 1000 ions 1343 / 1283 / 1312 / 1551: two are 2 % better
// where 16-atom blocks fill the chip by themselves, four up to 12 % where they do not.
constexpr int kRealCtas = 4, kCtaWarps = kRealWarps / kRealCtas;

__global__ void __cluster_dims__(kRealCtas, 1, 1) __launch_bounds__(32 * kCtaWarps) real_packed_kernel(
    const int32_t *sys_offset, const double *lj_sigma, const double *lj_eps, int nsp, int terms, int max_atoms,
    RealWork w, double *energy, double *grad) {
  // blockIdx.z of gridDim.z takes an equal share of every atom's partners; with more than one
  // share the blocks add their partial forces (terms & 8 is then required)
  __shared__ float2 ljt[64];
  __shared__ float part[2 * kCtaWarps][kRealAtoms][3];  // this CTA's streams
  __shared__ double red[40];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // per warp: the forces of kRealBatch hits; the hits of one pass (half << 9 | slot << 5 | t)
  float4 *force = reinterpret_cast<float4 *>(smem_raw) + kRealBatch * (threadIdx.x >> 5);
  uint16_t *wq = reinterpret_cast<uint16_t *>(smem_raw + sizeof(float4) * kRealBatch * kCtaWarps) +
                 32 * 32 * (threadIdx.x >> 5);
  const int s = blockIdx.y;
  const int a0 = sys_offset[s], n = sys_offset[s + 1] - a0;
  const int rank = (int)blockIdx.x % kRealCtas, block = (int)blockIdx.x / kRealCtas;
  if (block * kRealAtoms >= n || n > max_atoms) return;  // uniform over the cluster
  const int64_t pb = (int64_t)s * max_atoms;  // this system's rows of the packed arrays
  const float4 *hi = w.hi + pb, *lo = w.lo + pb, *frac = w.frac + pb;
  const RealSys S = w.sys[s];
  if (S.refused) return;
  const float *L = S.L, *I = S.I;
  if ((terms & 1) && nsp * nsp <= 64)
    for (int k = threadIdx.x; k < nsp * nsp; k += blockDim.x) {
      const double sg = lj_sigma[k];
      ljt[k] = make_float2((float)(sg * sg), (float)(4.0 * lj_eps[k]));
    }
  __syncthreads();
  const float two_al_rsqrtpi = 2.0f * S.alpha * 0.56418958354775628695f;
  const int lane = threadIdx.x & 31, warp = rank * kCtaWarps + (threadIdx.x >> 5);
  const int slot = lane & (kRealAtoms - 1), stream_id = warp * 2 + (lane >> 4);
  const int il = block * kRealAtoms + slot;
  const bool act = il < n;
  const int64_t gi = a0 + (act ? il : 0);
  const int own = act ? il : 0;
  const float4 frac_i = frac[own];
  // minimum-image difference of rows gj and ii from the hi / lo pairs
  auto diff = [&](const float4 &hi_i, const float4 &lo_i, const float4 &hj, const float4 &lj, float &dx, float &dy,
                  float &dz, float &r2) {
    const float d0 = (hj.x - hi_i.x) + (lj.x - lo_i.x), d1 = (hj.y - hi_i.y) + (lj.y - lo_i.y),
                d2 = (hj.z - hi_i.z) + (lj.z - lo_i.z);
    float f0 = (d0 * I[0] + d1 * I[1]) + d2 * I[3], f1 = d1 * I[2] + d2 * I[4], f2 = d2 * I[5];
    f0 -= rintf(f0);
    f1 -= rintf(f1);
    f2 -= rintf(f2);
    dx = (f0 * L[0] + f1 * L[1]) + f2 * L[3];
    dy = f1 * L[2] + f2 * L[4];
    dz = f2 * L[5];
    r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
  };
  // |f L|^2 of the fractional differences to two partners, each to its nearest image
  auto both = [](float x) { return make_float2(x, x); };
  auto nearest = [&](float2 d) {
    const float2 up = __fadd2_rn(d, both(12582912.f));  // 1.5 * 2^23: the sum is a whole number
    const float2 n2 = __fadd2_rn(up, both(-12582912.f));
    return __ffma2_rn(n2, both(-1.f), d);
  };
  auto near2 = [&](const float4 &p0, const float4 &p1) {
    const float2 f0 = nearest(make_float2(p0.x - frac_i.x, p1.x - frac_i.x));
    const float2 f1 = nearest(make_float2(p0.y - frac_i.y, p1.y - frac_i.y));
    const float2 f2 = nearest(make_float2(p0.z - frac_i.z, p1.z - frac_i.z));
    const float2 a = __ffma2_rn(both(S.g02), f2, __ffma2_rn(both(S.g01), f1, __fmul2_rn(both(S.g00), f0)));
    const float2 b = __ffma2_rn(both(S.g12), f2, __fmul2_rn(both(S.g11), f1));
    return __ffma2_rn(f0, a, __ffma2_rn(f1, b, __fmul2_rn(f2, __fmul2_rn(both(S.g22), f2))));
  };
  float ef = 0.f, fx = 0.f, fy = 0.f, fz = 0.f;  // energy of the pairs this lane evaluates; force of its atom
  const int n_streams = kRealStreams * (int)gridDim.z;
  const int per = (n + n_streams - 1) / n_streams;
  const int sbase = (int)blockIdx.z * kRealStreams;
  const int j0 = (sbase + stream_id) * per, j1 = min(n, j0 + per);
  // chunk starts of the warp's two streams
  const int j0h[2] = {(sbase + warp * 2) * per, (sbase + warp * 2 + 1) * per};
  const int passes = (per + 31) / 32;  // the same for both half-warps of a warp
  for (int pass = 0; pass < passes; ++pass) {
    const int c0 = j0 + pass * 32;
    const int cn = max(0, min(32, j1 - c0));
    const float4 *fj = frac + min(c0, n);  // reads up to 32 rows, some past the stream's end
    uint32_t hits = 0;
    float closest = INFINITY;  // to the cutoff, of any partner
#pragma unroll 4
    for (int t = 0; t < 32; t += 2) {
      const float2 d = __fadd2_rn(near2(fj[t], fj[t + 1]), both(-S.rc2));  // signs: within the cutoff
      hits = __funnelshift_l(__float_as_uint(d.x), hits, 1);
      hits = __funnelshift_l(__float_as_uint(d.y), hits, 1);
      closest = fminf(closest, fminf(fabsf(d.x), fabsf(d.y)));
    }
    hits = __brev(hits);
    if (__any_sync(0xffffffffu, closest <= S.margin)) {  // the rounding of the hi / lo test decides
      hits = 0;
#pragma unroll 4
      for (int t = 0; t < cn; ++t) {
        float dx, dy, dz, r2;
        diff(hi[own], lo[own], hi[c0 + t], lo[c0 + t], dx, dy, dz, r2);
        hits |= (uint32_t)(r2 < S.rc2) << t;
      }
    }
    if (cn < 32) hits &= (1u << cn) - 1;
    if (cn > 0 && c0 <= il && il < c0 + cn) hits &= ~(1u << (il - c0));  // not the atom itself
    if (!act) hits = 0;
    // append this lane's hits to the warp's queue (exclusive prefix of the counts)
    const int cnt = __popc(hits);
    int off = cnt;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, off, o);
      if (lane >= o) off += y;
    }
    const int total = __shfl_sync(0xffffffffu, off, 31), end = off, begin = off - cnt;
    off = begin;
    const uint16_t tag = (uint16_t)(((lane >> 4) << 9) | (slot << 5));
    while (hits) {
      const int t = __ffs(hits) - 1;
      hits &= hits - 1;
      wq[off++] = tag | (uint16_t)t;
    }
    __syncwarp();
    // the lanes evaluate queued pairs; then each adds up its own atom's, in order
    for (int eb = 0; eb < total; eb += kRealBatch) {
      const int stop = min(total, eb + kRealBatch);
#pragma unroll 2
      for (int e = eb + lane; e < stop; e += 32) {
        const int code = wq[e];
        const int h = code >> 9, sl = (code >> 5) & 15, t = code & 31;
        const int ii = block * kRealAtoms + sl, jj = j0h[h] + pass * 32 + t;
        const float4 hi_a = hi[ii], lo_a = lo[ii], hj = hi[jj], lj = lo[jj];
        float dx, dy, dz, r2;
        diff(hi_a, lo_a, hj, lj, dx, dy, dz, r2);
        float dedr2 = 0.f;
        const float ir = rsqrtf(r2);  // a few ulp; one MUFU op instead of IEEE sqrt and divisions
        if ((terms & 1) && r2 < S.rc2_lj) {
          const float2 c = ljt[__float_as_int(lo_a.w) * nsp + __float_as_int(lj.w)];
          const float inv = ir * ir, s2 = c.x * inv, c6 = s2 * s2 * s2;
          ef += c.y * (c6 * c6 - c6);
          dedr2 += -0.5f * c.y * c6 * (12.f * c6 - 6.f) * inv;
        }
        if ((terms & 2) && r2 < S.rc2_ew) {
          const float r = r2 * ir, qq = (hi_a.w * S.ke) * hj.w, al = S.alpha;
          const float er = erfc_cheb(al * r);
          ef += qq * er * ir;
          const float t = two_al_rsqrtpi * __expf(-al * al * r2);
          // which product is rounded written out: the same bits whatever surrounds it
          dedr2 = fmaf(0.5f * ir * qq, fmaf(-t, ir, __fmul_rn(-er * ir, ir)), dedr2);
        }
        const float m = -2.f * dedr2;
        force[e - eb] = make_float4(__fmul_rn(m, dx), __fmul_rn(m, dy), __fmul_rn(m, dz), 0.f);
      }
      __syncwarp();
      const int last = min(end, stop) - eb;
      for (int j = max(begin, eb) - eb; j < last; ++j) {
        const float4 v = force[j];
        fx += v.x;
        fy += v.y;
        fz += v.z;
      }
      __syncwarp();
    }
  }
  const int mine = stream_id - rank * 2 * kCtaWarps;
  part[mine][slot][0] = fx;
  part[mine][slot][1] = fy;
  part[mine][slot][2] = fz;
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  cluster.sync();
  if (rank == 0 && threadIdx.x < kRealAtoms && act) {
    float gx = 0.f, gy = 0.f, gz = 0.f;
    for (int r = 0; r < kRealCtas; ++r) {
      const float *p = cluster.map_shared_rank(&part[0][slot][0], r);
#pragma unroll
      for (int k = 0; k < 2 * kCtaWarps; ++k, p += 3 * kRealAtoms) {
        gx += p[0];
        gy += p[1];
        gz += p[2];
      }
    }
    if (gridDim.z > 1) {  // several blocks share atom gi
      atomicAdd(&grad[3 * gi], (double)gx);
      atomicAdd(&grad[3 * gi + 1], (double)gy);
      atomicAdd(&grad[3 * gi + 2], (double)gz);
    } else if (terms & 8) {  // add onto the caller's gradient (this block owns atom gi)
      grad[3 * gi] += gx;
      grad[3 * gi + 1] += gy;
      grad[3 * gi + 2] += gz;
    } else {
      grad[3 * gi] = gx;
      grad[3 * gi + 1] = gy;
      grad[3 * gi + 2] = gz;
    }
  }
  const double esum = block_sum(0.5 * (double)ef, red);
  if (threadIdx.x == 0) atomicAdd(&energy[s], esum);
  cluster.sync();  // the first CTA has read the others' forces
}

inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// The reciprocal-space launch sequence of kups_ewald_recip and
// kups_ewald_recip_static: setup, structure factor, energy and forces.
// `base` is 256-byte aligned scratch of at least recip_scratch_bytes().
inline size_t recip_scratch_bytes(int32_t n_systems, int32_t n_kvecs) {
  return align256(sizeof(RecipSys) * (size_t)n_systems) +
         align256(sizeof(Coef) * (size_t)n_systems * (size_t)n_kvecs);
}

// Kernels run on an SM at the same time only under one division of its memory into shared memory and
// cache: real and reciprocal space, side by side in a molecular-dynamics step, ask for the same (65 % of
// it shared).  A step of 4000 ions: 86.0 us with the driver's choices, 81.4 with 65, 83.4 with 80.  Ten steps
// with the driver's choice / 65 %: 216 ions 315 / 316 us, 512 ions 304 / 295, 2000 ions 436 / 410, 8000 ions
// 2290 / 2121, 32 systems of 216 ions 511 / 486.
template <typename F>
inline cudaError_t same_carveout(F *kernel) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 65);
}

int32_t recip_launch(char *base, const double *positions, const double *charges, const int32_t *sys_offset,
                     int32_t n_systems, int32_t max_atoms_per_system, const double *tril, const int32_t *kvec_n,
                     int32_t n_kvecs, const double *alpha, double coulomb_k, double *energy, double *grad,
                     double *grad_tril, double *structure_factor, kups_status *status, cudaStream_t stream) {
  RecipSys *sysp = (RecipSys *)base;
  Coef *coef = (Coef *)(base + align256(sizeof(RecipSys) * (size_t)n_systems));
  KUPS_CUDA_TRY(same_carveout(recip_setup_kernel));
  KUPS_CUDA_TRY(same_carveout(structure_factor_kernel));
  KUPS_CUDA_TRY(same_carveout(recip_force_kernel));
  recip_setup_kernel<<<n_systems, kSetupThreads, 0, stream>>>(tril, kvec_n, n_kvecs, sysp, structure_factor, energy,
                                                              grad_tril, status);
  const int chunks = (max_atoms_per_system + kAtomsPerChunk - 1) / kAtomsPerChunk;
  if (n_kvecs > 0 && chunks > 0) {
    const int tile = kKPerBlock * kKPerThread;
    dim3 g((n_kvecs + tile - 1) / tile, chunks, n_systems);
    structure_factor_kernel<<<g, kKPerBlock, 0, stream>>>(positions, charges, sys_offset, kvec_n, n_kvecs, sysp, alpha,
                                                          coef, structure_factor, grad);
  }
  if (chunks > 0 && n_kvecs > 0) {
    // enough k splits that the launch holds about 16 warps per SM
    const int kblocks = (n_kvecs + kKPerBlock - 1) / kKPerBlock;
    const int want = std::max(1, (16 * device_sm_count()) / std::max(1, 4 * chunks * n_systems));
    const int splits = std::min(kblocks, want);
    const int per = (kblocks + splits - 1) / splits;
    dim3 g(chunks, n_systems, (kblocks + per - 1) / per);
    recip_force_kernel<<<g, kForceThreads, 0, stream>>>(positions, charges, sys_offset, kvec_n,
                                                             n_kvecs, sysp, coef, structure_factor, coulomb_k, energy,
                                                             grad, grad_tril, per);
  } else if (chunks > 0) {
    dim3 g(chunks, n_systems, 1);
    recip_force_kernel<<<g, kForceThreads, 0, stream>>>(positions, charges, sys_offset, kvec_n,
                                                             n_kvecs, sysp, coef, structure_factor, coulomb_k, energy,
                                                             grad, grad_tril, 0);
  }
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

}  // namespace
}  // namespace kups

using namespace kups;

extern "C" size_t kups_ewald_recip_workspace_bytes(int32_t n_systems, int32_t n_kvecs) {
  return recip_scratch_bytes(n_systems, n_kvecs) + 512;
}

extern "C" int32_t kups_ewald_recip(const double *positions, const double *charges,
                                    const int32_t *sys_offset, int32_t n_systems,
                                    int32_t max_atoms_per_system, const double *tril,
                                    const int32_t *kvec_n, int32_t n_kvecs, const double *alpha,
                                    double coulomb_k, double *energy, double *grad,
                                    double *grad_tril, double *structure_factor,
                                    void *workspace, size_t workspace_bytes, kups_status *status,
                                    void *stream_) {
  if (n_systems < 0 || n_kvecs < 0 || max_atoms_per_system < 0) return KUPS_ERR_INVALID;
  if (workspace_bytes < kups_ewald_recip_workspace_bytes(n_systems, n_kvecs)) return KUPS_ERR_INVALID;
  if (n_systems == 0) return KUPS_OK;
  char *base = (char *)(((uintptr_t)workspace + 255) & ~uintptr_t(255));
  return recip_launch(base, positions, charges, sys_offset, n_systems, max_atoms_per_system, tril, kvec_n,
                      n_kvecs, alpha, coulomb_k, energy, grad, grad_tril, structure_factor, status,
                      (cudaStream_t)stream_);
}

extern "C" int32_t kups_ewald_kvecs_outside(const int32_t *kvec_n, int32_t n_systems, int32_t n_kvecs,
                                            int32_t *outside, void *stream) {
  if (n_systems < 0 || n_kvecs < 0 || outside == nullptr) return KUPS_ERR_INVALID;
  const int64_t count = 3 * (int64_t)n_systems * n_kvecs;
  if (count == 0) return KUPS_OK;
  const unsigned blocks = (unsigned)std::min<int64_t>((count + 255) / 256, 4 * (int64_t)device_sm_count());
  kvec_limit_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(kvec_n, count, outside);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

// Reciprocal energy from given structure factors (the energy step of the launch
// sequence above; its scratch is the same workspace).
extern "C" int32_t kups_ewald_recip_energy(const double *tril, const int32_t *kvec_n, int32_t n_kvecs,
                                           const double *alpha, int32_t n_systems, double coulomb_k,
                                           const double *structure_factor, double *energy, void *workspace,
                                           size_t workspace_bytes, kups_status *status, void *stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (n_systems < 0 || n_kvecs < 0) return KUPS_ERR_INVALID;
  if (workspace_bytes < kups_ewald_recip_workspace_bytes(n_systems, n_kvecs)) return KUPS_ERR_INVALID;
  if (n_systems == 0) return KUPS_OK;
  char *base = (char *)(((uintptr_t)workspace + 255) & ~uintptr_t(255));
  RecipSys *sysp = (RecipSys *)base;
  recip_setup_kernel<<<n_systems, kSetupThreads, 0, stream>>>(tril, kvec_n, n_kvecs, sysp, nullptr, energy, nullptr,
                                                              status);
  recip_energy_kernel<<<dim3((unsigned)std::max(1, (n_kvecs + 31) / 32), n_systems), 32, 0, stream>>>(
      kvec_n, n_kvecs, alpha, sysp, structure_factor, coulomb_k, energy);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

// ---------------------------------------------------------------------------
// kups_ewald_recip_static: the reciprocal-space computation above with its
// scratch (per-system cell data, then per-(system, k) coefficients) in one
// fixed device array instead of a caller-supplied workspace.  It serves
// callers that have no device allocator to draw a workspace from, e.g. an
// FFI handler that a host framework hands only its input and output buffers.
//
// The array is shared by every call on a device and keeps whatever the last
// call left in it; every byte a call reads is written earlier in the same
// call, so nothing in it has to start at zero.  Two calls whose launches
// overlap in time (different streams, or different host threads) race on it.
// The array lives in this file's module: every device on which any kernel of
// this file runs holds its KUPS_EWALD_RECIP_STATIC_SCRATCH_BYTES until the
// process exits (or the device is reset).
namespace kups {
namespace {
constexpr size_t kStaticScratchBytes = KUPS_EWALD_RECIP_STATIC_SCRATCH_BYTES;
constexpr int kStaticMaxDevices = 64;
std::mutex g_static_scratch_mutex;
void *g_static_scratch_ptr[kStaticMaxDevices] = {};
}  // namespace
static __device__ __align__(256) unsigned char g_recip_static_scratch[kStaticScratchBytes];
}  // namespace kups

extern "C" int32_t kups_ewald_recip_static(const double *positions, const double *charges,
                                           const int32_t *sys_offset, int32_t n_systems,
                                           int32_t max_atoms_per_system, const double *tril,
                                           const int32_t *kvec_n, int32_t n_kvecs,
                                           const double *alpha, double coulomb_k, double *energy,
                                           double *grad, double *grad_tril,
                                           double *structure_factor, kups_status *status,
                                           void *stream_) {
  if (n_systems < 0 || n_kvecs < 0 || max_atoms_per_system < 0) return KUPS_ERR_INVALID;
  // Sizes beyond the array are refused before anything is touched.
  if ((size_t)n_systems > kStaticScratchBytes / sizeof(RecipSys)) return KUPS_ERR_CAPACITY;
  if (n_kvecs > 0 && (size_t)n_systems > kStaticScratchBytes / sizeof(Coef) / (size_t)n_kvecs)
    return KUPS_ERR_CAPACITY;
  if (recip_scratch_bytes(n_systems, n_kvecs) > kStaticScratchBytes) return KUPS_ERR_CAPACITY;
  if (n_systems == 0) return KUPS_OK;
  // Once per device, with that device current: look up the array's address.
  int dev = 0;
  KUPS_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kStaticMaxDevices) return KUPS_ERR_UNSUPPORTED;
  char *base = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_static_scratch_mutex);
    if (g_static_scratch_ptr[dev] == nullptr) {
      void *p = nullptr;
      if (cudaGetSymbolAddress(&p, g_recip_static_scratch) != cudaSuccess || p == nullptr)
        return KUPS_ERR_CUDA;
      g_static_scratch_ptr[dev] = p;
    }
    base = (char *)g_static_scratch_ptr[dev];
  }
  return recip_launch(base, positions, charges, sys_offset, n_systems, max_atoms_per_system, tril, kvec_n,
                      n_kvecs, alpha, coulomb_k, energy, grad, grad_tril, structure_factor, status,
                      (cudaStream_t)stream_);
}

extern "C" int32_t kups_ewald_self(const double *charges, const int32_t *sys_offset,
                                   int32_t n_systems, const double *alpha, double coulomb_k,
                                   double *energy, void *stream) {
  if (n_systems < 0) return KUPS_ERR_INVALID;
  if (n_systems == 0) return KUPS_OK;
  self_energy_kernel<<<n_systems, 256, 0, (cudaStream_t)stream>>>(charges, sys_offset, alpha,
                                                                 coulomb_k, energy);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

extern "C" int32_t kups_pair_edges(const double *positions, const int32_t *system,
                                   const int32_t *species, const double *charges, int64_t n,
                                   const double *tril, int32_t n_systems, const double *lj_sigma,
                                   const double *lj_epsilon, int32_t n_species,
                                   const double *lj_cutoff, const double *alpha,
                                   const double *ewald_cutoff, double coulomb_k, int32_t terms,
                                   const int32_t *edges, const int32_t *shifts, int64_t n_edges,
                                   double *energy, double *grad, double *grad_tril,
                                   kups_status *status, void *stream) {
  (void)status;
  return launch_pair_edges<false>(positions, system, species, charges, n, tril, n_systems, lj_sigma, lj_epsilon,
                                  n_species, lj_cutoff, alpha, ewald_cutoff, coulomb_k, terms, edges, shifts, n_edges,
                                  energy, grad, grad_tril, (cudaStream_t)stream);
}

extern "C" int32_t kups_pair_edges_paired(const double *positions, const int32_t *system,
                                   const int32_t *species, const double *charges, int64_t n,
                                   const double *tril, int32_t n_systems, const double *lj_sigma,
                                   const double *lj_epsilon, int32_t n_species,
                                   const double *lj_cutoff, const double *alpha,
                                   const double *ewald_cutoff, double coulomb_k, int32_t terms,
                                   const int32_t *edges, const int32_t *shifts, int64_t n_edges,
                                   double *energy, double *grad, double *grad_tril,
                                   kups_status *status, void *stream) {
  (void)status;
  const bool one_of_two = (terms & 1) == 0 || n_species <= kTableSpecies;
  const auto launch = one_of_two ? launch_pair_edges<true> : launch_pair_edges<false>;
  return launch(positions, system, species, charges, n, tril, n_systems, lj_sigma, lj_epsilon,
                                  n_species, lj_cutoff, alpha, ewald_cutoff, coulomb_k, terms, edges, shifts, n_edges,
                                  energy, grad, grad_tril, (cudaStream_t)stream);
}

extern "C" int32_t kups_lj_ewald_real_forces(const double *positions, const double *charges,
                                             const int32_t *species, const int32_t *sys_offset,
                                             int32_t n_systems, int32_t max_atoms_per_system,
                                             const double *tril, const double *lj_sigma,
                                             const double *lj_epsilon, int32_t n_species,
                                             const double *lj_cutoff, const double *alpha,
                                             const double *ewald_cutoff, double coulomb_k, int32_t terms,
                                             double *energy, double *grad, kups_status *status,
                                             void *stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (n_systems < 0 || max_atoms_per_system < 0 || terms < 1 || terms > 3) return KUPS_ERR_INVALID;
  if ((terms & 1) && (n_species < 1 || n_species > 8 || lj_sigma == nullptr || lj_epsilon == nullptr))
    return KUPS_ERR_INVALID;
  if (n_systems == 0) return KUPS_OK;
  KUPS_CUDA_TRY(cudaMemsetAsync(energy, 0, sizeof(double) * (size_t)n_systems, stream));
  if (max_atoms_per_system == 0) return KUPS_OK;
  dim3 g((max_atoms_per_system + kRealAtoms - 1) / kRealAtoms, n_systems);
  real_allpairs_kernel<<<g, 32 * kRealWarps, 0, stream>>>(positions, charges, species, sys_offset, tril, lj_sigma,
                                                    lj_epsilon, n_species, lj_cutoff, alpha, ewald_cutoff,
                                                    coulomb_k, terms, energy, grad, status);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

extern "C" size_t kups_lj_ewald_real_forces_workspace_bytes(int32_t n_systems, int32_t max_atoms_per_system) {
  if (n_systems <= 0 || max_atoms_per_system <= 0) return 256;
  return real_work(nullptr, n_systems, max_atoms_per_system).bytes + 256;
}

extern "C" int32_t kups_lj_ewald_real_forces_packed(const double *positions, const double *charges,
                                                    const int32_t *species, const int32_t *sys_offset,
                                                    int32_t n_systems, int32_t max_atoms_per_system,
                                                    const double *tril, const double *lj_sigma,
                                                    const double *lj_epsilon, int32_t n_species,
                                                    const double *lj_cutoff, const double *alpha,
                                                    const double *ewald_cutoff, double coulomb_k, int32_t terms,
                                                    double *energy, double *grad, void *workspace,
                                                    size_t workspace_bytes, kups_status *status, void *stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  const int splits_req = (terms >> 8) & 15;  // partner shares per atom block; 0: chosen here
  terms &= 255;
  if (n_systems < 0 || max_atoms_per_system < 0 || (terms & ~11) != 0 || (terms & 3) == 0) return KUPS_ERR_INVALID;
  if ((terms & 1) && (n_species < 1 || n_species > 8 || lj_sigma == nullptr || lj_epsilon == nullptr))
    return KUPS_ERR_INVALID;
  if (n_systems == 0) return KUPS_OK;
  if (max_atoms_per_system == 0) {
    if (!(terms & 8)) KUPS_CUDA_TRY(cudaMemsetAsync(energy, 0, sizeof(double) * (size_t)n_systems, stream));
    return KUPS_OK;
  }
  if (workspace == nullptr ||
      workspace_bytes < kups_lj_ewald_real_forces_workspace_bytes(n_systems, max_atoms_per_system))
    return KUPS_ERR_INVALID;
  char *base = reinterpret_cast<char *>(((uintptr_t)workspace + 255) & ~uintptr_t(255));
  const RealWork w = real_work(base, n_systems, max_atoms_per_system);
  dim3 gp((max_atoms_per_system + 255) / 256 + 1, n_systems);
  KUPS_CUDA_TRY(same_carveout(real_pack_kernel));
  real_pack_kernel<<<gp, 256, 0, stream>>>(positions, charges, species, sys_offset, tril, lj_cutoff, alpha,
                                           ewald_cutoff, coulomb_k, terms, max_atoms_per_system, w, energy, status);
  // partner shares: the caller's choice (a launch-shape tuner's), else one.  Shares add their
  // partial forces, so they need terms & 8 (the caller's gradient is the base).  One share
  // measured fastest on the 4000-ion melt (250 clusters of four CTAs on 152 SMs: 0.083 ms per
  // replayed force evaluation against 0.086 / 0.097 / 0.095 for 2 / 3 / 4 shares).
  const int splits = (terms & 8) && splits_req > 0 ? splits_req : 1;
  dim3 g(kRealCtas * ((max_atoms_per_system + kRealAtoms - 1) / kRealAtoms), n_systems, splits);
  const size_t smem = kCtaWarps * (kRealBatch * sizeof(float4) + 32 * 32 * sizeof(uint16_t));
  KUPS_CUDA_TRY(cudaFuncSetAttribute(real_packed_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  KUPS_CUDA_TRY(same_carveout(real_packed_kernel));
  real_packed_kernel<<<g, 32 * kCtaWarps, smem, stream>>>(sys_offset, lj_sigma, lj_epsilon, n_species, terms,
                                                        max_atoms_per_system, w, energy, grad);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

namespace kups {
namespace {
__global__ void erfc_eval_kernel(const float *x, int64_t n, float *out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = erfc_cheb(x[i]);
}
}  // namespace
}  // namespace kups

extern "C" int32_t kups_erfc_eval(const float *x, int64_t n, float *out, void *stream) {
  if (n < 0) return KUPS_ERR_INVALID;
  if (n == 0) return KUPS_OK;
  erfc_eval_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(x, n, out);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}
