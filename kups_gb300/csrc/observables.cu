// Per-system virial observables from positions, dU/dx, dU/dtril and momenta:
// the atomic virial stress, the molecular virial stress of the RASPA convention,
// the lattice-gradient stress, the kinetic energy and the instantaneous pressure.
//
// Replaces src/kups/observables/stress.py:64-118 (_stress_via_lattice_vector_gradients,
// _stress_via_virial_theorem, _molecular_stress_via_virial_theorem),
// src/kups/md/observables.py:17-61 (particle_kinetic_energy summed per system,
// instantaneous_pressure with d = 3) and pressure.py:27-29 (_pressure_from_stress).
//
//   atomic     sigma_ab = -(sum_i r_ia g_ib + (L^T G)_ab) / V
//   molecular  sigma    = -(sym(sum_i w_i (x) g_i) + L^T G) / V,  sym(A) = (A + A^T) / 2,
//              w_i = r_i - wrap(r_i - R_g(i)), R_g = wrap(mean_j wrap(r_j - r_a) + r_a)
//              over the atoms j of group g, a the group's first atom
//   lattice    sigma    = -G / V
//   pressure   P = 2 K / (3 V) + Tr(sigma_atomic) / 3   (K = 0 without momenta)
// with g_i = dU/dr_i, G = dU/dL (lower triangular, from dU/dtril), V = |L00 L11 L22|,
// wrap() into the fractional cell [-0.5, 0.5).  Each system uses its own volume; the
// reference's molecular stress divides every system by the first system's volume
// (stress.py:114), the same number for one system or equal cells.
//
// Layout of the work.  All of it is float64, and the float64 pipe (two lanes per cycle and SM) bounds
// it: 512 k atoms at 100 operations each take 90 us there, against 7 us for their bytes.  So the
// molecular sum runs over molecules, not atoms, where it can.  With c = mean_j wrap(r_j - r_a) + r_a,
//   w_i = c + floor((r_i - c) L^-1 + 1/2) L,
// the wrap of the centre cancelling out, and of the atoms of a molecule that lies whole in one image
// and spans less than a quarter of the cell every w_i is c: sum_i w_i (x) g_i = c (x) sum_i g_i.
// Float32 copies of the displacements decide that, with a margin for their rounding; what they cannot
// decide is decided in float64.  Three kinds of work, gathered per block so that warps stay full:
//   * a group whose atoms are neighbours in memory and in one system (at most kRunMax of them):
//     one thread per group;
//   * such a group that straddles a cell face (w_i further by its atoms' images) or is wide (its
//     centre and images in float64);
//   * atoms of any other group: centres by two passes over all atoms first (sum of minimum images
//     relative to the first atom, then mean, shift back and wrap), then one thread per atom.
// Every thread keeps running sums while its warp's items stay in one system, so a warp issues one
// reduction per run of items.
// 512 k atoms in three-atom molecules: 121 + 32 + 24 + 22 us (sums, two passes for the centres, outputs)
// became 56 + 9 + 6 + 6, the sums at 70 % of the float64 pipe while a block is resident.  Blocks of 128
// threads, three per SM: 256 x 1 took 60 us, 512 x 1 63, 192 x 2 58, 128 x 4 61 (a flush costs a warp 31
// additions whatever its share of the items, too few warps leave the pipe idle).
#include <algorithm>

#include "common.cuh"

namespace kups {
namespace {

constexpr int kAcc = 19;      // per system: K, sum r_a g_b (9), sum w_a g_b (9)
constexpr int kRunMax = 16;   // atoms of a group that one thread takes
constexpr int kThreads = 256, kAccThreads = 128, kAccBlocks = 3;
constexpr int kChunkMax = 2048;  // atoms whose items a block gathers at a time
static_assert(kChunkMax / kAccThreads <= 32, "one bit per atom of a thread");

inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// wrap(r) into the fractional cell [-0.5, 0.5): f = r @ L^-1, f = mod(f + 0.5, 1) - 0.5, f @ L
// (unitcell.py:139-171), with the rounding of the float64 restatement.
__device__ inline void wrap64(const double r[3], const Tril64 &L, const Tril64 &Li, double out[3]) {
  double f[3];
  row_times_tril64(r, Li, f);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double x = __dadd_rn(f[a], 0.5);
    f[a] = __dsub_rn(__dsub_rn(x, floor(x)), 0.5);
  }
  row_times_tril64(f, L, out);
}

// The image the wrap takes: n = floor(f + 0.5), f = d @ L^-1 (the same rounding as
// wrap64), so that wrap(d) = d - n @ L.  Returns false when n = 0 (wrap(d) = d up to the
// rounding of the round trip through fractional coordinates).
__device__ inline bool wrap_image64(const double d[3], const Tril64 &Li, double n[3]) {
  double f[3];
  row_times_tril64(d, Li, f);
#pragma unroll
  for (int a = 0; a < 3; ++a) n[a] = floor(__dadd_rn(f[a], 0.5));
  return n[0] != 0.0 || n[1] != 0.0 || n[2] != 0.0;
}

__device__ inline bool valid_index(int v, int n) { return v >= 0 && v < n; }

// 1 / m to float64 accuracy without a float64 division: the float32 reciprocal
// (relative error about 1e-7) refined by one Newton step y (2 - m y), which squares
// the relative error.
__device__ inline double recip64(double m) {
  const double y = (double)(1.0f / (float)m);
  return y * fma(-m, y, 2.0);
}

// 1 / m of a small integer, rounded to nearest
__constant__ double kRecip[kRunMax + 1] = {0.0,      1.0,      1.0 / 2,  1.0 / 3,  1.0 / 4,  1.0 / 5,
                                           1.0 / 6,  1.0 / 7,  1.0 / 8,  1.0 / 9,  1.0 / 10, 1.0 / 11,
                                           1.0 / 12, 1.0 / 13, 1.0 / 14, 1.0 / 15, 1.0 / 16};

// Per group: the number of runs of neighbouring atoms that it consists of (runs longer than kRunMax
// count twice), and its first atom as INT32_MAX - index; per system the inverse cell; group sums zeroed.
// *any_other is set when a group is not a single run.
__global__ void __launch_bounds__(kThreads) group_runs_kernel(const int32_t *group, const int32_t *system, int64_t n,
                                                              int32_t n_groups, int32_t n_sys, const double *tril,
                                                              double *inv, double *gsum, int32_t *first,
                                                              int32_t *runs, int32_t *any_other,
                                                              kups_status *status) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n_sys) {
    const Tril64 Li = inverse_tril64(load_tril64(tril + 6 * i));
#pragma unroll
    for (int k = 0; k < 6; ++k) inv[6 * i + k] = Li.t[k];
  }
  if (i < n_groups) {
#pragma unroll
    for (int k = 0; k < 4; ++k) gsum[4 * i + k] = 0.0;
  }
  if (i >= n) return;
  const int g = group[i], s = system[i];
  if (!valid_index(g, n_groups) || !valid_index(s, n_sys)) {
    status_error(status, KUPS_ERR_INVALID, i);
    if (valid_index(g, n_groups)) {  // not an atom of its group: no neighbours in memory to rely on
      atomicAdd(&runs[g], 1);
      *any_other = 1;
    }
    return;
  }
  if (i == 0 || group[i - 1] != g || system[i - 1] != s) {
    atomicMax(&first[g], INT32_MAX - (int32_t)i);
    if (atomicAdd(&runs[g], 1) > 0) *any_other = 1;
  }
  if (i >= kRunMax && group[i - kRunMax] == g && (i == kRunMax || group[i - kRunMax - 1] != g)) {
    atomicAdd(&runs[g], 1);
    *any_other = 1;
  }
}

// r_i - r_a in the image nearest to a, d - img @ L
__device__ inline void nearest_offset(const double *pos, int64_t i, int64_t a, const Tril64 &L, const Tril64 &Li,
                                      double d[3]) {
  double img[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) d[c] = __dsub_rn(pos[3 * i + c], pos[3 * a + c]);
  if (wrap_image64(d, Li, img)) {
    double nL[3];
    row_times_tril64(img, L, nL);
#pragma unroll
    for (int c = 0; c < 3; ++c) d[c] = __dsub_rn(d[c], nL[c]);
  }
}

// wrap(sum / count + r_a)
__device__ inline void wrapped_centre(const double sum[3], double count, const double *ra, const Tril64 &L,
                                      const Tril64 &Li, double w[3]) {
  double c[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) c[k] = __dadd_rn(__ddiv_rn(sum[k], count), ra[k]);
  wrap64(c, L, Li, w);
}

// w = r - wrap(r - R) = R + n @ L: the centre's image nearest the atom
__device__ inline void nearest_centre(const double r[3], const double R[3], const Tril64 &L, const Tril64 &Li,
                                      double w[3]) {
  double d[3], n[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    w[c] = R[c];
    d[c] = __dsub_rn(r[c], w[c]);
  }
  if (wrap_image64(d, Li, n)) {
    double nL[3];
    row_times_tril64(n, L, nL);
#pragma unroll
    for (int c = 0; c < 3; ++c) w[c] = __dadd_rn(w[c], nL[c]);
  }
}

// gsum[g] += (wrap(r_i - r_first), 1) of the groups that are not a single run
__global__ void __launch_bounds__(kThreads) group_sum_kernel(const double *pos, const int32_t *group,
                                                             const int32_t *system, int64_t n, int32_t n_groups,
                                                             int32_t n_sys, const double *tril, const double *inv,
                                                             const int32_t *first, const int32_t *runs,
                                                             const int32_t *any_other, double *gsum) {
  if (*any_other == 0) return;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int g = group[i], s = system[i];
    if (!valid_index(g, n_groups) || !valid_index(s, n_sys) || runs[g] == 1) continue;
    double d[3];
    nearest_offset(pos, i, INT32_MAX - first[g], load_tril64(tril + 6 * (int64_t)s), load_tril64(inv + 6 * (int64_t)s),
                   d);
#pragma unroll
    for (int c = 0; c < 3; ++c) atomicAdd(&gsum[4 * (int64_t)g + c], d[c]);
    atomicAdd(&gsum[4 * (int64_t)g + 3], 1.0);
  }
}

// gsum[g] <- (wrap(sum / count + r_first), count): the group's centre in place.
__global__ void __launch_bounds__(kThreads) group_centre_kernel(const double *pos, const int32_t *system,
                                                                int32_t n_groups, const double *tril,
                                                                const double *inv, const int32_t *first,
                                                                const int32_t *runs, const int32_t *any_other,
                                                                double *gsum) {
  if (*any_other == 0) return;
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < n_groups; g += (int64_t)gridDim.x * blockDim.x) {
    if (runs[g] < 2 || first[g] == 0) continue;
    const int a = INT32_MAX - first[g];
    double w[3];
    wrapped_centre(gsum + 4 * g, gsum[4 * g + 3], pos + 3 * (int64_t)a, load_tril64(tril + 6 * (int64_t)system[a]),
                   load_tril64(inv + 6 * (int64_t)system[a]), w);
#pragma unroll
    for (int k = 0; k < 3; ++k) gsum[4 * g + k] = w[k];
  }
}

// Sums over the warp of W (a power of two) values per lane: lane l returns that of value
// l / (32 / W).  Each step halves the values a lane keeps.
template <int W>
__device__ inline double warp_columns(const double *v) {
  const int lane = threadIdx.x & 31;
  double a[W];
#pragma unroll
  for (int i = 0; i < W; ++i) a[i] = v[i];
  int o = 16;
#pragma unroll
  for (int w = W / 2; w >= 1; w /= 2, o /= 2)
#pragma unroll
    for (int i = 0; i < w; ++i) {
      const double keep = lane & o ? a[w + i] : a[i], send = lane & o ? a[i] : a[w + i];
      a[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  double t = a[0];
  for (; o >= 1; o /= 2) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

template <int NV>
__device__ inline void flush_run(double (&acc)[NV], int sys, double *out) {
  constexpr int W = NV >= 16 ? 16 : 8;
  const int lane = threadIdx.x & 31;
  const double t = warp_columns<W>(acc);
  if (sys >= 0 && lane % (32 / W) == 0 && t != 0.0) atomicAdd(&out[(int64_t)sys * kAcc + lane / (32 / W)], t);
#pragma unroll
  for (int k = W; k < NV; ++k) {
    const double v = warp_sum(acc[k]);
    if (lane == 0 && sys >= 0 && v != 0.0) atomicAdd(&out[(int64_t)sys * kAcc + k], v);
  }
#pragma unroll
  for (int k = 0; k < NV; ++k) acc[k] = 0.0;
}

// x truncated to float32 by its bits (the float64 pipe has the conversions): the smallest normal
// number below the normal range, infinite above it and for a NaN.
__device__ inline float truncated32(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), e = hi & 0x7fffffffu;
  unsigned f = ((e - 0x38000000u) << 3) | ((unsigned)__double2loint(x) >> 29);
  f = e == 0u ? 0u : e < 0x38100000u ? 0x00800000u : e >= 0x47f00000u ? 0x7f800000u : f;
  return __uint_as_float(f | (hi & 0x80000000u));
}

// Running sums of the atom's own terms: twice its kinetic energy and r_a g_b.
template <bool KE, int NV>
__device__ inline void add_atom(const double r[3], const double g[3], const double *mom, const double *mass, int64_t i,
                                double (&run)[NV]) {
  if (KE) {
    const double p0 = mom[3 * i], p1 = mom[3 * i + 1], p2 = mom[3 * i + 2];
    run[0] = fma(fma(p0, p0, fma(p1, p1, p2 * p2)), recip64(mass[i]), run[0]);
  }
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) run[1 + 3 * a + b] = fma(r[a], g[b], run[1 + 3 * a + b]);
}

template <int NV>
__device__ inline void add_centre(const double w[3], const double g[3], double (&run)[NV]) {
  if constexpr (NV == kAcc) {
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) run[10 + 3 * a + b] = fma(w[a], g[b], run[10 + 3 * a + b]);
  }
}

__device__ inline void load3(const double *p, int64_t i, double (&v)[3]) {
#pragma unroll
  for (int c = 0; c < 3; ++c) v[c] = p[3 * i + c];
}

__device__ inline void offset(const double r[3], const double ra[3], double d[3]) {
#pragma unroll
  for (int c = 0; c < 3; ++c) d[c] = __dsub_rn(r[c], ra[c]);
}

// f = d @ L^-1 in float32, and the sums e of its terms' sizes: the truncations and roundings are off by
// less than 2^-20 e together.
constexpr float kNear = 0.2499f;
__device__ inline void fractions(const double d[3], const float li[6], float f[3], float e[3]) {
  const float x = truncated32(d[0]), y = truncated32(d[1]), z = truncated32(d[2]);
  const float t1 = y * li[1], t2 = z * li[3], t4 = z * li[4];
  f[0] = x * li[0] + t1 + t2;
  f[1] = y * li[2] + t4;
  f[2] = z * li[5];
  e[0] = fabsf(x * li[0]) + fabsf(t1) + fabsf(t2);
  e[1] = fabsf(y * li[2]) + fabsf(t4);
  e[2] = fabsf(f[2]);
}

// The image img of the offset d, true unless zero; sure is cleared unless d less its image is below a
// quarter of the cell in each direction (so that the image holds relative to any mean of such offsets).
__device__ inline bool near_image(const double d[3], const float li[6], double img[3], bool &sure) {
  float f[3], e[3];
  fractions(d, li, f, e);
  bool some = false;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float n = rintf(f[c]);
    sure = sure && fabsf(f[c] - n) + 1e-6f * e[c] < kNear;
    some = some || n != 0.f;
    img[c] = (double)n;
  }
  return some;
}

__device__ inline void shift_image(const double img[3], const Tril64 &L, double d[3]) {  // d - img @ L
  d[0] = fma(-img[0], L.t[0], fma(-img[1], L.t[1], fma(-img[2], L.t[3], d[0])));
  d[1] = fma(-img[1], L.t[2], fma(-img[2], L.t[4], d[1]));
  d[2] = fma(-img[2], L.t[5], d[2]);
}

// c = sum / m + r_a: a correction step after the product with the rounded 1 / m
__device__ inline void mean_offset(const double sum[3], int m, const double ra[3], double c[3]) {
  const double inv_m = kRecip[m];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double t = sum[k] * inv_m;
    c[k] = fma(fma(-t, (double)m, sum[k]), inv_m, t) + ra[k];
  }
}

template <bool MOL, bool KE>
__global__ void __launch_bounds__(kAccThreads, kAccBlocks) virial_accumulate_kernel(
    const double *pos, const double *grad, const int32_t *system, int64_t n, int32_t n_sys,
    const int32_t *group, int32_t n_groups, const double *gcentre, const int32_t *runs, const double *tril,
    const double *inv, const double *mom, const double *mass, int chunk, double *out, kups_status *status) {
  constexpr int NV = MOL ? kAcc : 10, kWarps = kAccThreads / 32;
  __shared__ int32_t items[MOL ? kChunkMax : 1], odd[MOL ? kChunkMax : 1];  // groups from the front, atoms from the back
  __shared__ int n_other, n_odd, warp_total[kWarps];
  const unsigned full = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double run[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) run[k] = 0.0;
  int cur = -1;
  // eval() adds an item of system s (act: whether this lane has one) to the running sums.  Two systems
  // among the 32 items (a border of the usual order by system) are taken one after the other; more are
  // added to their systems lane by lane.
  auto add = [&](int s, bool act, auto &&eval) {
    unsigned todo = __ballot_sync(full, act);
    if (todo == 0) return;
    if (cur < 0) cur = __shfl_sync(full, s, __ffs(todo) - 1);
    const unsigned off = __ballot_sync(full, act && s != cur);
    const int second = __shfl_sync(full, s, off ? __ffs(off) - 1 : 0);
    const bool many = __any_sync(full, act && s != cur && s != second);
    if (many) flush_run<NV>(run, cur, out);
    while (todo) {
      if (act && (many || s == cur)) eval();
      if (many) {
#pragma unroll
        for (int k = 0; k < NV; ++k) {
          add_system(out, kAcc, k, act ? s : -1, run[k]);
          run[k] = 0.0;
        }
        cur = __shfl_sync(full, s, 31 - __clz(todo));
        todo = 0u;
      } else {
        todo = cur == second || off == 0u ? 0u : off;
        if (todo) {
          flush_run<NV>(run, cur, out);
          cur = second;
        }
      }
    }
  };
  for (int64_t c0 = (int64_t)blockIdx.x * chunk; c0 < n; c0 += (int64_t)gridDim.x * chunk) {
    const int cnt = (int)min((int64_t)chunk, n - c0);
    if (!MOL) {
      for (int j = warp * 32; j < cnt; j += kAccThreads) {
        const int64_t i = c0 + j + lane;
        const int s = j + lane < cnt ? system[i] : -1;
        const bool act = valid_index(s, n_sys);
        if (j + lane < cnt && !act) status_error(status, KUPS_ERR_INVALID, i);
        add(s, act, [&]() {
          double r[3], g[3];
          load3(pos, i, r);
          load3(grad, i, g);
          add_atom<KE, NV>(r, g, mom, mass, i, run);
        });
      }
      continue;
    }
    // the chunk's items, in order: a thread looks at kChunkMax / kAccThreads neighbouring atoms
    if (tid == 0) n_other = n_odd = 0;
    const int per = (cnt + kAccThreads - 1) / kAccThreads, j0 = min(cnt, tid * per), j1 = min(cnt, j0 + per);
    __syncthreads();
    unsigned heads = 0u;
    int gp = -1, sp = -1;
    if (j0 < j1 && c0 + j0 > 0) {
      gp = group[c0 + j0 - 1];
      sp = system[c0 + j0 - 1];
    }
    for (int j = j0; j < j1; ++j) {
      const int64_t i = c0 + j;
      const int g = group[i], s = system[i];
      const bool known = valid_index(g, n_groups), in = valid_index(s, n_sys);
      if (!known || !in) status_error(status, KUPS_ERR_INVALID, i);
      if (known && in && runs[g] == 1) {
        if (g != gp || s != sp || i == 0) heads |= 1u << (j - j0);
      } else if (in) {
        items[kChunkMax - 1 - atomicAdd(&n_other, 1)] = j;
      }
      gp = g;
      sp = s;
    }
    int at = __popc(heads), incl = at;
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(full, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) warp_total[warp] = incl;
    __syncthreads();
    int n_heads = 0;
    at = incl - at;
    for (int w = 0; w < kWarps; ++w) {
      if (w == warp) at += n_heads;
      n_heads += warp_total[w];
    }
    for (unsigned m = heads; m; m &= m - 1) items[at++] = j0 + __ffs(m) - 1;
    __syncthreads();
    for (int q = warp * 32; q < n_heads; q += kAccThreads) {  // whole groups
      const bool act = q + lane < n_heads;
      const int64_t a = act ? c0 + items[q + lane] : 0;
      const int s = act ? system[a] : -1, gi = act ? group[a] : -1;
      add(s, act, [&]() {
        float li[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) li[k] = truncated32(inv[6 * (int64_t)s + k]);
        double ra[3], gs[3], sum[3] = {0.0, 0.0, 0.0};
        load3(pos, a, ra);
        load3(grad, a, gs);
        add_atom<KE, NV>(ra, gs, mom, mass, a, run);
        bool plain = true;
        int m = 1;
        for (; m < kRunMax && a + m < n && group[a + m] == gi; ++m) {
          double r[3], g[3], d[3];
          load3(pos, a + m, r);
          load3(grad, a + m, g);
          offset(r, ra, d);
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            sum[c] += d[c];
            gs[c] += g[c];
          }
          float f[3], e[3];
          fractions(d, li, f, e);
#pragma unroll
          for (int c = 0; c < 3; ++c) plain = plain && e[c] < kNear;  // NaN: no
          add_atom<KE, NV>(r, g, mom, mass, a + m, run);
        }
        if (plain) {
          double c[3];
          mean_offset(sum, m, ra, c);
          add_centre<NV>(c, gs, run);
        } else {
          odd[atomicAdd(&n_odd, 1)] = (int32_t)(a - c0);
        }
      });
    }
    __syncthreads();
    const int odds = n_odd, others = n_other;
    for (int q = warp * 32; q < odds; q += kAccThreads) {  // groups across a face, or wide
      const bool act = q + lane < odds;
      const int64_t a = act ? c0 + odd[q + lane] : 0;
      const int s = act ? system[a] : -1, gi = act ? group[a] : -1;
      add(s, act, [&]() {
        float li[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) li[k] = truncated32(inv[6 * (int64_t)s + k]);
        const Tril64 L = load_tril64(tril + 6 * (int64_t)s);
        double ra[3], gs[3], sum[3] = {0.0, 0.0, 0.0};
        load3(pos, a, ra);
        load3(grad, a, gs);
        bool sure = true;
        unsigned moved = 0u;
        int m = 1;
        for (; m < kRunMax && a + m < n && group[a + m] == gi; ++m) {
          double r[3], g[3], d[3], img[3];
          load3(pos, a + m, r);
          load3(grad, a + m, g);
          offset(r, ra, d);
          if (near_image(d, li, img, sure)) {
            moved |= 1u << m;
            shift_image(img, L, d);
          }
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            sum[c] += d[c];
            gs[c] += g[c];
          }
        }
        if (sure) {
          double c[3];
          mean_offset(sum, m, ra, c);
          add_centre<NV>(c, gs, run);
          for (unsigned k = moved; k; k &= k - 1) {  // the centre's image nearest these is img @ L further
            const int64_t i = a + __ffs(k) - 1;
            double r[3], g[3], d[3], img[3], w[3] = {0.0, 0.0, 0.0};
            load3(pos, i, r);
            load3(grad, i, g);
            offset(r, ra, d);
            near_image(d, li, img, sure);
#pragma unroll
            for (int c2 = 0; c2 < 3; ++c2) img[c2] = -img[c2];
            shift_image(img, L, w);
            add_centre<NV>(w, g, run);
          }
        } else {
          const Tril64 Li = load_tril64(inv + 6 * (int64_t)s);
          double R[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) sum[c] = 0.0;
          for (int k = 1; k < m; ++k) {
            double d[3];
            nearest_offset(pos, a + k, a, L, Li, d);
#pragma unroll
            for (int c = 0; c < 3; ++c) sum[c] += d[c];
          }
          wrapped_centre(sum, (double)m, ra, L, Li, R);
          for (int k = 0; k < m; ++k) {
            double r[3], g[3], w[3];
            load3(pos, a + k, r);
            load3(grad, a + k, g);
            nearest_centre(r, R, L, Li, w);
            add_centre<NV>(w, g, run);
          }
        }
      });
    }
    for (int q = warp * 32; q < others; q += kAccThreads) {  // atoms of other groups
      const bool act = q + lane < others;
      const int64_t i = act ? c0 + items[kChunkMax - 1 - (q + lane)] : 0;
      const int s = act ? system[i] : -1;
      add(s, act, [&]() {
        double r[3], g[3];
        load3(pos, i, r);
        load3(grad, i, g);
        add_atom<KE, NV>(r, g, mom, mass, i, run);
        const int gi = group[i];
        if (valid_index(gi, n_groups)) {
          double R[3], w[3];
          for (int c = 0; c < 3; ++c) R[c] = gcentre[4 * (int64_t)gi + c];
          nearest_centre(r, R, load_tril64(tril + 6 * (int64_t)s), load_tril64(inv + 6 * (int64_t)s), w);
          add_centre<NV>(w, g, run);
        }
      });
    }
    __syncthreads();
  }
  flush_run<NV>(run, cur, out);
}

// Sixteen lanes per system, lane k < 9 the component (k / 3, k % 3): one division per lane and output
// (one thread per system, nine divisions in a row, took 22 us for 64 systems).
__global__ void __launch_bounds__(128) virial_finish_kernel(const double *acc, const double *tril,
                                                            const double *grad_tril, int32_t n_sys, bool have_ke,
                                                            double *stress, double *mol_stress, double *lat_stress,
                                                            double *kinetic, double *pressure) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int k = (int)(t & 15), i = k < 9 ? k / 3 : 0, j = k < 9 ? k % 3 : 0;
  const bool act = t / 16 < n_sys;
  const int64_t s = act ? t / 16 : n_sys - 1;
  const double *q = tril + 6 * s, *gt = grad_tril ? grad_tril + 6 * s : nullptr;
  auto low = [](const double *p, int r, int c) { return p != nullptr && c <= r ? p[r * (r + 1) / 2 + c] : 0.0; };
  const double V = fabs(q[0] * q[2] * q[5]);
  const double *a = acc + s * kAcc;
  double ltg = 0.0;
#pragma unroll
  for (int m = 0; m < 3; ++m) ltg += low(q, m, i) * low(gt, m, j);
  const double sa = -(a[1 + 3 * i + j] + ltg) / V;
  if (act && k < 9) {
    if (stress) stress[9 * s + k] = sa;
    if (mol_stress) mol_stress[9 * s + k] = (-0.5 * (a[10 + 3 * i + j] + a[10 + 3 * j + i]) - ltg) / V;
    if (lat_stress) lat_stress[9 * s + k] = -low(gt, i, j) / V;
  }
  const double s4 = __shfl_sync(0xffffffffu, sa, 4, 16), s8 = __shfl_sync(0xffffffffu, sa, 8, 16);
  if (act && k == 0) {
    const double tr = sa + s4 + s8, K = have_ke ? 0.5 * a[0] : 0.0;
    if (kinetic) kinetic[s] = K;
    if (pressure) pressure[s] = 2.0 * K / (3.0 * V) + tr / 3.0;
  }
}

inline unsigned blocks_for(int64_t n, int threads) { return (unsigned)std::max<int64_t>(1, (n + threads - 1) / threads); }

}  // namespace
}  // namespace kups

using namespace kups;

extern "C" size_t kups_virial_stress_workspace_bytes(int32_t n_systems, int32_t n_groups) {
  if (n_systems < 0 || n_groups < 0) return 0;
  return sizeof(double) * 6 * (size_t)n_systems + align256(sizeof(double) * kAcc * (size_t)n_systems) +
         align256(sizeof(double) * 4 * (size_t)n_groups) + sizeof(int32_t) * (2 * (size_t)n_groups + 1) + 256;
}

extern "C" int32_t kups_virial_stress(const double *positions, const double *grad, const int32_t *system,
                                      int64_t n_particles, const double *tril, const double *grad_tril,
                                      int32_t n_systems, const int32_t *group, int32_t n_groups,
                                      const double *momenta, const double *masses, double *stress,
                                      double *molecular_stress, double *lattice_stress, double *kinetic,
                                      double *pressure, void *workspace, size_t workspace_bytes,
                                      kups_status *status, void *stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  const bool mol = molecular_stress != nullptr;
  const bool ke = momenta != nullptr;
  if (n_particles < 0 || n_systems < 0 || n_groups < 0) return KUPS_ERR_INVALID;
  if (n_systems > 0 && !tril) return KUPS_ERR_INVALID;
  if (n_particles > 0 && (!positions || !grad || !system || !status)) return KUPS_ERR_INVALID;
  if (ke && !masses) return KUPS_ERR_INVALID;
  if (kinetic && !ke) return KUPS_ERR_INVALID;
  if (mol && (!group || n_particles >= (int64_t)INT32_MAX)) return KUPS_ERR_INVALID;
  if (n_systems == 0) return KUPS_OK;
  if (workspace_bytes < kups_virial_stress_workspace_bytes(n_systems, mol ? n_groups : 0)) return KUPS_ERR_INVALID;
  char *base = (char *)(((uintptr_t)workspace + 255) & ~uintptr_t(255));
  // inverse cells and group sums, then what starts as zero: system sums, first atoms, runs, flag
  const int32_t ng = mol ? n_groups : 0;
  double *gsum = (double *)base, *inv = gsum + 4 * (size_t)ng, *acc = inv + 6 * (size_t)n_systems;
  int32_t *first = (int32_t *)(acc + kAcc * (size_t)n_systems), *runs = first + ng, *any_other = runs + ng;
  KUPS_CUDA_TRY(cudaMemsetAsync(acc, 0, sizeof(double) * kAcc * (size_t)n_systems + (2 * (size_t)ng + 1) * sizeof(int32_t),
                                stream));
  const int sms = device_sm_count(), slots = kAccBlocks * sms;
  if (mol && n_particles > 0) {
    const int64_t threads = std::max<int64_t>(n_particles, std::max(ng, n_systems));
    group_runs_kernel<<<blocks_for(threads, kThreads), kThreads, 0, stream>>>(
        group, system, n_particles, ng, n_systems, tril, inv, gsum, first, runs, any_other, status);
    // both leave at once when every group is a single run
    const unsigned grid = std::min(blocks_for(n_particles, kThreads), (unsigned)(8 * sms));
    group_sum_kernel<<<grid, kThreads, 0, stream>>>(positions, group, system, n_particles, ng, n_systems, tril, inv,
                                                    first, runs, any_other, gsum);
    group_centre_kernel<<<std::min(blocks_for(ng, kThreads), (unsigned)(8 * sms)), kThreads, 0, stream>>>(
        positions, system, ng, tril, inv, first, runs, any_other, gsum);
  }
  if (n_particles > 0) {
    // equal chunks for the resident blocks, as many passes as the chunk limit asks for; no less than
    // 128 atoms, below which a block has no full warp of three-atom groups
    const int64_t passes = (n_particles + (int64_t)slots * kChunkMax - 1) / ((int64_t)slots * kChunkMax);
    const int chunk = (int)std::max<int64_t>(128, (n_particles + slots * passes - 1) / (slots * passes));
    const unsigned blocks = (unsigned)std::min<int64_t>(slots, (n_particles + chunk - 1) / chunk);
#define KUPS_VIRIAL_LAUNCH(M, K)                                                                                  \
  virial_accumulate_kernel<M, K><<<blocks, kAccThreads, 0, stream>>>(positions, grad, system, n_particles,        \
                                                                     n_systems, group, ng, gsum, runs, tril, inv, \
                                                                     momenta, masses, chunk, acc, status)
    if (mol && ke) KUPS_VIRIAL_LAUNCH(true, true);
    else if (mol) KUPS_VIRIAL_LAUNCH(true, false);
    else if (ke) KUPS_VIRIAL_LAUNCH(false, true);
    else KUPS_VIRIAL_LAUNCH(false, false);
#undef KUPS_VIRIAL_LAUNCH
  }
  virial_finish_kernel<<<blocks_for(16 * (int64_t)n_systems, 128), 128, 0, stream>>>(
      acc, tril, grad_tril, n_systems, ke, stress, molecular_stress, lattice_stress, kinetic, pressure);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}
