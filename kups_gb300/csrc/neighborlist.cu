// Reference-exact periodic neighbour list (float64 membership test).
//
// Replaces CellListNeighborList / DenseNearestNeighborList.__call__
// (src/kups/core/neighborlist.py:902-1077) for rh = None.  The edge set is the
// one basic_neighborlist (:743-786) produces; the cell grid here is this
// library's own (any grid whose cells are at least rc wide yields the same
// set, which is why the reference's Dense and CellList variants share a test
// suite).  Pipeline, all stream-ordered:
//   count atoms per system -> per-system setup (inverse cell, widths, image
//   counts, cell grid) -> bin atoms -> scan -> scatter -> order each cell by
//   particle index (deterministic) -> find and write the edges of every lh
//   particle in one pass (never past capacity) -> pad the tail.
#include <algorithm>

#include "common.cuh"
#include "scan.cuh"

namespace kups {
namespace {

struct SysNL {
  Tril64 L;
  Tril64 inv;
  double rc2;
  float Lf[6];
  float lo2, hi2;  // float32 squared distance below lo2: surely inside the cutoff, at or above hi2: outside
  int tie;         // a pair within the cutoff may lie half a cell apart, with another image far away
  int nc[3];
  int nimg[3];
  int image_mode;  // prod(nimg) > 1: explicit image offsets, all system pairs are candidates
  int n_atoms;
  int64_t cell_base;
  int refused;     // more than kMaxNLImages image offsets: no edges, KUPS_ERR_UNSUPPORTED recorded
};

// Image offsets per candidate pair beyond which a system is refused instead of searched (a
// cutoff of many cell widths: 11^3 offsets is a cutoff of about five widths; the
// reference's own image replication would materialise that many copies of every pair).
constexpr double kMaxNLImages = 1331.0;

// Neighbour cells per particle.
constexpr int kNLCells = 27;
// Pair search: warps (particles) per block.
constexpr int kPairWarps = 8;

struct NLWork {
  char *zero;           // start of the words a call zeroes first (through zero_bytes)
  size_t zero_bytes;
  SysNL *sys;           // [S], zeroed (n_atoms counts up)
  unsigned *tickets;    // [4]: block counters of the setup, cell scan and pair search
  unsigned long long *scan_state;  // [chained_scan_blocks(n_cells_cap + 1)]
  unsigned long long *pair_state;  // [pair blocks]
  int *cell_start;      // [n_cells_cap + 1], zeroed (counts, then starts)
  double *frac;         // [N, 3] unwrapped fractional coordinates
  float4 *wrapped;      // [N] f - rint(f) in float32, packed rint(f) (pack_image)
  int *cell_of;         // [N] global cell id or -1
  int *slot_of;         // [N] arrival order inside the cell
  int *cell_any;        // [N] particles by cell, in arrival order
  int *cell_items;      // [N] particles by cell, in index order
  float4 *cand;         // [N] the same order: f - rint(f), particle index
  int4 *cand_label;     // [N] the same order: inclusion, exclusion, packed rint(f)
  int64_t n_cells_cap;
  int64_t scan_blocks, pair_blocks;
};

inline size_t align_up(size_t x) { return (x + 255) & ~size_t(255); }

// Cells allotted: never more than max(1, 2 * atoms) per system, so the total
// is bounded by n_systems + 2 * n_particles.
inline int64_t cells_capacity(int64_t n, int32_t s) { return (int64_t)s + 2 * n + 1; }

size_t layout(NLWork *w, char *base, int64_t n, int32_t s) {
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char *p = base ? base + off : nullptr;
    off += align_up(bytes);
    return p;
  };
  const int64_t cc = cells_capacity(n, s);
  NLWork t;
  t.scan_blocks = chained_scan_blocks(cc + 1);
  t.pair_blocks = (n + kPairWarps - 1) / kPairWarps;
  t.zero = base;
  t.sys = (SysNL *)take(sizeof(SysNL) * (size_t)s);
  t.tickets = (unsigned *)take(sizeof(unsigned) * 4);
  t.scan_state = (unsigned long long *)take(sizeof(unsigned long long) * (size_t)t.scan_blocks);
  t.pair_state = (unsigned long long *)take(sizeof(unsigned long long) * (size_t)t.pair_blocks);
  t.cell_start = (int *)take(sizeof(int) * (size_t)(cc + 1));
  t.zero_bytes = off;
  t.frac = (double *)take(sizeof(double) * 3 * (size_t)n);
  t.wrapped = (float4 *)take(sizeof(float4) * (size_t)n);
  t.cand = (float4 *)take(sizeof(float4) * (size_t)n);
  t.cand_label = (int4 *)take(sizeof(int4) * (size_t)n);
  t.cell_of = (int *)take(sizeof(int) * (size_t)n);
  t.slot_of = (int *)take(sizeof(int) * (size_t)n);
  t.cell_any = (int *)take(sizeof(int) * (size_t)n);
  t.cell_items = (int *)take(sizeof(int) * (size_t)n);
  t.n_cells_cap = cc;
  if (w) *w = t;
  return off;
}

// Atoms per system: one atomic per warp while its particles share a system (the usual grouped table).
__global__ void count_atoms_kernel(const int32_t *system, int64_t n, int32_t s, SysNL *sys) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int32_t si = i < n ? system[i] : -1;
  const unsigned same = __match_any_sync(0xffffffffu, si);
  if (si >= 0 && si < s && (int)(threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&sys[si].n_atoms, __popc(same));
}

// Per-system parameters and the exclusive scan of cells per system.  Each block takes 32 systems
// (one per lane): warps 0..2 form the width, image count and cell count of one axis each, warp 3 the
// inverse, so the float64 divisions (a latency chain of several microseconds when one thread does
// all of them: 11 us for one system, 19 us for 256) run side by side; the block that finishes last
// scans the cell counts: 8 us for one system, 10 us for 256.
constexpr int kSetupSystems = 32;
__global__ void __launch_bounds__(4 * kSetupSystems) setup_systems_kernel(const double *tril, const double *cutoffs,
                                                                         int32_t s, SysNL *sys, unsigned *ticket,
                                                                         kups_status *status) {
  __shared__ int nimg[3][kSetupSystems], ncell[3][kSetupSystems], narrow[3][kSetupSystems];
  __shared__ int64_t scratch[32];
  __shared__ unsigned done;
  const int lane = threadIdx.x & 31, role = threadIdx.x >> 5;
  const int k = blockIdx.x * kSetupSystems + lane;
  const double rc = k < s ? cutoffs[k] : 0.0;
  const bool finite = isfinite(rc);
  if (k < s) {
    const Tril64 L = load_tril64(tril + 6 * (int64_t)k);
    if (role < 3) {
      double w3[3];
      perpendicular_widths64(L, w3);
      const double w = role == 0 ? w3[0] : role == 1 ? w3[1] : w3[2];
      int n = 1, c = 1;
      if (finite) {
        const double x = ceil(2.0 * rc / w);
        n = x > 1e6 ? 1000001 : (int)x;
        if (n < 1) n = 1;
        if (n % 2 == 0) n += 1;
        const double y = floor(w / rc);
        c = y < 1.0 ? 1 : (y > 1024.0 ? 1024 : (int)y);
      }
      nimg[role][lane] = n;
      ncell[role][lane] = c;
      narrow[role][lane] = finite && w < 2.0 * fabs(rc) * (1.0 + 1e-4);
    } else {
      const Tril64 inv = inverse_tril64(L);
      SysNL &p = sys[k];
      p.L = L;
      p.inv = inv;
    }
  }
  __syncthreads();
  if (role == 0 && k < s) {
    SysNL &p = sys[k];
    int n[3] = {nimg[0][lane], nimg[1][lane], nimg[2][lane]};
    double prod = 1.0;
    for (int a = 0; a < 3; ++a) prod *= (double)n[a];
    const bool refused = prod > kMaxNLImages;
    if (refused) {
      status_error(status, KUPS_ERR_UNSUPPORTED, k);
      n[0] = n[1] = n[2] = 1;
      prod = 1.0;
    }
    const bool image_mode = prod > 1.0;
    int64_t budget = 2 * (int64_t)p.n_atoms;
    if (budget < 1) budget = 1;
    int nc[3];
    for (int a = 0; a < 3; ++a) nc[a] = image_mode ? 1 : ncell[a][lane];
    while ((int64_t)nc[0] * nc[1] * nc[2] > budget) {
      int am = 0;
      for (int a = 1; a < 3; ++a)
        if (nc[a] > nc[am]) am = a;
      nc[am] = (nc[am] + 1) / 2;
    }
    // float32 prefilter: a fractional difference of two stored float32 coordinates is off by at most
    // 2^-24 (plus its own rounding), the products with L and their sum by a few 2^-24 of the terms;
    // 2^-19 sum|L| bounds the error of the distance with a factor of several to spare, and 2^-16 of
    // the squared cutoff the rounding of its square.  Between lo2 and hi2 the float64 test decides.
    // Two particles half a cell apart may round to the other image of the two, which in a skewed cell is
    // far away: where the cutoff reaches half a cell width, such candidates are kept whatever their distance.
    const double rc2 = rc * rc;
    double sum = 0.0;
    for (int a = 0; a < 6; ++a) {
      const double v = tril[6 * (int64_t)k + a];
      p.Lf[a] = (float)v;
      sum += fabs(v);
    }
    const double err = sum * (1.0 / 524288.0);
    const double margin = rc2 * (1.0 / 65536.0) + 2.0 * fabs(rc) * err + err * err;
    p.rc2 = rc2;
    p.hi2 = finite ? (float)(rc2 + margin) : (float)rc2;
    p.lo2 = finite ? (float)(rc2 - margin) : -1.0f;
    p.tie = (p.Lf[1] != 0.f || p.Lf[3] != 0.f || p.Lf[4] != 0.f) && (narrow[0][lane] | narrow[1][lane] | narrow[2][lane]);
    for (int a = 0; a < 3; ++a) {
      p.nimg[a] = n[a];
      p.nc[a] = nc[a];
    }
    p.image_mode = image_mode;
    p.refused = refused;
    p.cell_base = (int64_t)nc[0] * nc[1] * nc[2];  // the count until the scan below
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) done = atomicAdd(ticket, 1u);
  __syncthreads();
  if (done != gridDim.x - 1) return;
  __threadfence();
  int64_t carry = 0;
  for (int base = 0; base < s; base += blockDim.x) {
    const int q = base + threadIdx.x;
    const int64_t cells = q < s ? __ldcg(reinterpret_cast<const long long *>(&sys[q].cell_base)) : 0;
    int64_t chunk;
    const int64_t ex = block_exclusive_scan<int64_t>(cells, scratch, &chunk);
    if (q < s) sys[q].cell_base = carry + ex;
    carry += chunk;
    __syncthreads();
  }
}

__device__ inline int wrap_cell(double f, int nc) {
  double w = f - floor(f);  // [0, 1)
  int c = (int)(w * nc);
  return c >= nc ? nc - 1 : (c < 0 ? 0 : c);
}

// rint(f) of the three axes in 10 bits each (offset 512); kWideImage marks one outside [-512, 511].
constexpr int kWideImage = 1 << 30;
__device__ inline int pack_image(const double n[3]) {
  int v = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (!(n[a] >= -512.0 && n[a] <= 511.0)) return kWideImage;
    v |= ((int)n[a] + 512) << (10 * a);
  }
  return v;
}
__device__ inline int image_axis(int packed, int a) { return ((packed >> (10 * a)) & 1023) - 512; }

__global__ void bin_kernel(const double *positions, const int32_t *system, int64_t n, int32_t s, const SysNL *sys,
                           double *frac, float4 *wrapped, int *cell_of, int *slot_of, int *cell_count) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int32_t si = system[i];
  if (si < 0 || si >= s) {
    cell_of[i] = -1;
    return;
  }
  const SysNL &p = sys[si];
  const double r[3] = {positions[3 * i], positions[3 * i + 1], positions[3 * i + 2]};
  double f[3], img[3];
  row_times_tril64(r, p.inv, f);
  float w[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    frac[3 * i + a] = f[a];
    img[a] = rint(f[a]);
    w[a] = (float)(f[a] - img[a]);
  }
  wrapped[i] = make_float4(w[0], w[1], w[2], __int_as_float(pack_image(img)));
  const int cx = wrap_cell(f[0], p.nc[0]), cy = wrap_cell(f[1], p.nc[1]),
            cz = wrap_cell(f[2], p.nc[2]);
  const int c = (int)p.cell_base + (cz * p.nc[1] + cy) * p.nc[0] + cx;
  cell_of[i] = c;
  slot_of[i] = atomicAdd(&cell_count[c], 1);
}

__global__ void scatter_kernel(const int *cell_of, const int *slot_of, int64_t n, const int *cell_start,
                               int *cell_any) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int c = cell_of[i];
  if (c >= 0) cell_any[cell_start[c] + slot_of[i]] = (int)i;
}

// A particle's place in its cell is the number of smaller indices in it: each cell ends up in index
// order whatever the arrival order, with one thread per particle (an insertion sort by one thread
// per cell took 945 us for 4000 particles in 27 cells, this 14 us).  Writes the candidate records of
// the pair search in that order.
__global__ void order_cells_kernel(const int *cell_of, int64_t n, const int *cell_start, const int *cell_any,
                                   const float4 *wrapped, const int32_t *inclusion, const int32_t *exclusion,
                                   int *cell_items, float4 *cand, int4 *cand_label) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int c = cell_of[i];
  if (c < 0) return;
  const int b = cell_start[c], e = cell_start[c + 1];
  int r = b;
#pragma unroll 8
  for (int k = b; k < e; ++k) r += cell_any[k] < (int)i;
  cell_items[r] = (int)i;
  const float4 w = wrapped[i];
  cand[r] = make_float4(w.x, w.y, w.z, __int_as_float((int)i));
  cand_label[r] = make_int4(inclusion[i], exclusion[i], __float_as_int(w.w), 0);
}

// Candidate test of the reference for the pair (i, j) and offset o.
// Returns true if (i, j, shift) is an edge; writes the shift.
__device__ inline bool edge_test(const SysNL &p, const double fi[3], const double fj[3],
                                 const int o[3], bool use_image, int shift[3], bool same_excl) {
  double d0[3] = {__dadd_rn(fi[0], -fj[0]), __dadd_rn(fi[1], -fj[1]), __dadd_rn(fi[2], -fj[2])};
  double ms[3] = {rint(d0[0]), rint(d0[1]), rint(d0[2])};
  double sh[3];
  bool is_min = true;
  if (use_image) {
    for (int a = 0; a < 3; ++a) {
      sh[a] = (double)o[a];
      is_min = is_min && (ms[a] == sh[a]);
    }
  } else {
    sh[0] = ms[0];
    sh[1] = ms[1];
    sh[2] = ms[2];
  }
  double d[3] = {__dadd_rn(d0[0], -sh[0]), __dadd_rn(d0[1], -sh[1]), __dadd_rn(d0[2], -sh[2])};
  double real[3];
  row_times_tril64(d, p.L, real);
  const double d2 = norm2_64(real);
  if (!(d2 < p.rc2)) return false;
  if (same_excl && is_min) return false;
  shift[0] = (int)sh[0];
  shift[1] = (int)sh[1];
  shift[2] = (int)sh[2];
  return true;
}

// The candidates of one particle: up to 27 cells, each a contiguous run of the cell-ordered records,
// read as one flat range of `total` candidates in (cell, index) order.  Lane c holds run c (the
// non-empty ones, in order): the flat index it begins at and its first record minus that index.
struct CandRuns {
  int begin, shift, total;
};

// Record of flat candidate base + lane; `a` is the number of runs that begin before `base`, minus
// one, and is moved on to the next 32.  One reduction marks where runs begin among these 32.
__device__ inline int cand_record(const CandRuns &rg, int base, int &a) {
  const int lane = threadIdx.x & 31;
  const unsigned at = (unsigned)(rg.begin - base);
  const unsigned begins = __reduce_or_sync(0xffffffffu, at < 32u ? 1u << at : 0u);
  const int run = a + __popc(begins & (0xffffffffu >> (31 - lane)));
  a += __popc(begins);
  return __shfl_sync(0xffffffffu, rg.shift, run & 31) + base + lane;
}

// rint(x) for |x| < 2^22 by two additions (the rounding instruction runs at a quarter of their rate).
__device__ inline float rint_small(float x) { return __fadd_rn(__fadd_rn(x, 12582912.0f), -12582912.0f); }

// Minimum-image float32 difference of two wrapped coordinates: d (fractional) in [-0.5, 0.5], the
// image r, and the squared length.
__device__ inline float image_distance(const float4 &wi, const float4 &c, const float L[6], float d[3], float r[3]) {
  d[0] = wi.x - c.x;
  d[1] = wi.y - c.y;
  d[2] = wi.z - c.z;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    r[a] = rint_small(d[a]);
    d[a] -= r[a];
  }
  const float X = fmaf(d[2], L[3], fmaf(d[1], L[1], d[0] * L[0])), Y = fmaf(d[2], L[4], d[1] * L[2]), Z = d[2] * L[5];
  return fmaf(Z, Z, fmaf(Y, Y, X * X));
}

// Whether an offset lies within 2^-18 of half a cell, where float32 may take the other image.
__device__ inline bool beside_half(const float d[3]) {
  return fmaxf(fmaxf(fabsf(d[0]), fabsf(d[1])), fabsf(d[2])) > 0.5f - 1.0f / 262144.0f;
}

// What a search makes of particle i (the same in every lane of its warp).
struct PairQuery {
  int i, inc, exi, tie;
  float4 wi;
  float L[6], lo2, hi2;
};

__device__ __noinline__ bool exact_pair(const SysNL &p, const double *frac, int i, int j, const int o[3], bool image,
                                  bool same_ex, int sh[3]) {
  const double fi[3] = {frac[3 * (int64_t)i], frac[3 * (int64_t)i + 1], frac[3 * (int64_t)i + 2]};
  const double fj[3] = {frac[3 * (int64_t)j], frac[3 * (int64_t)j + 1], frac[3 * (int64_t)j + 2]};
  return edge_test(p, fi, fj, o, image, sh, same_ex);
}

// Whether record k is an edge of the particle at its minimum image, with its shift.  The float32
// distance settles nearly every candidate; within the margin of the cutoff, within 2^-18 of half a
// cell (the rounding of the image; with `tie` at any distance, see the setup) and for images beyond 10
// bits the float64 test decides, so the edge set is that of the float64 test alone.
__device__ inline bool settle_pair(const SysNL &p, const PairQuery &q, const float4 *cand, const int4 *label,
                                   const double *frac, int k, int &j, int sh[3]) {
  const float4 c = cand[k];
  float d[3], r[3];
  const float d2 = image_distance(q.wi, c, q.L, d, r);
  if (!(d2 < q.hi2) && !(q.tie && beside_half(d))) return false;
  const int4 lb = label[k];
  if (lb.x != q.inc) return false;
  j = __float_as_int(c.w);
  const int wn = __float_as_int(q.wi.w);
  const bool same_ex = lb.y == q.exi;
  if (!(d2 < q.lo2) || beside_half(d) || ((wn | lb.z) & kWideImage)) {
    const int o[3] = {0, 0, 0};
    return exact_pair(p, frac, q.i, j, o, false, same_ex, sh);
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) sh[a] = image_axis(wn, a) - image_axis(lb.z, a) + (int)r[a];
  return !same_ex;  // the shift is the minimum image, where equal exclusion labels drop the pair
}

__device__ inline bool fits_packed(const int sh[3]) {
  return (unsigned)(sh[0] + 512) < 1024u && (unsigned)(sh[1] + 512) < 1024u && (unsigned)(sh[2] + 512) < 1024u;
}
__device__ inline unsigned pack_shift(const int sh[3]) {
  return (unsigned)((sh[0] + 512) | ((sh[1] + 512) << 10) | ((sh[2] + 512) << 20));
}

// One image per axis: every candidate's distance first, keeping the records inside hi2 (a tenth of
// them), then the labels, shifts and close calls of those with every lane at work.  Returns the
// number of edges, the edges (j, packed shift) in `stage`; -1 if they do not fit its `room` rows.
__device__ int search_staged(const SysNL &p, const PairQuery &q, const CandRuns &rg, const float4 *cand,
                             const int4 *label, const double *frac, uint2 *stage, int room) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  int near = 0, a = -1;
#pragma unroll 2
  for (int base = 0; base < rg.total; base += 32) {
    const int k = cand_record(rg, base, a);
    bool in = false;
    if (base + lane < rg.total) {
      float d[3], r[3];
      in = image_distance(q.wi, cand[k], q.L, d, r) < q.hi2;
      if (q.tie) in |= beside_half(d);
    }
    const unsigned m = __ballot_sync(0xffffffffu, in);
    const int at = near + __popc(m & below);
    if (in && at < room) stage[at].x = (unsigned)k;
    near += __popc(m);
  }
  if (near > room) return -1;
  __syncwarp();
  int cnt = 0;
  bool wide = false;
  for (int base = 0; base < near; base += 32) {
    int j = 0, sh[3] = {0, 0, 0};
    const bool hit = base + lane < near && settle_pair(p, q, cand, label, frac, (int)stage[base + lane].x, j, sh);
    const unsigned m = __ballot_sync(0xffffffffu, hit);  // every lane has read its record
    if (hit) {
      wide |= !fits_packed(sh);
      stage[cnt + __popc(m & below)] = make_uint2((unsigned)j, pack_shift(sh));
    }
    cnt += __popc(m);
    __syncwarp();
  }
  return __any_sync(0xffffffffu, wide) ? -1 : cnt;
}

// The general search, edges handed to emit(hit, j, shift) 32 candidates at a time in the order of the
// reference: cells, then particle index, then image offsets.
template <typename Emit>
__device__ void search_each(const SysNL &p, const PairQuery &q, const CandRuns &rg, const float4 *cand,
                            const int4 *label, const double *frac, Emit emit) {
  const int lane = threadIdx.x & 31;
  if (!p.image_mode) {
    int a = -1;
    for (int base = 0; base < rg.total; base += 32) {
      const int k = cand_record(rg, base, a);
      int j = 0, sh[3] = {0, 0, 0};
      const bool hit = base + lane < rg.total && settle_pair(p, q, cand, label, frac, k, j, sh);
      emit(hit, j, sh);
    }
    return;
  }
  // one cell; (candidate, x, y, z offset) as a mixed-radix counter that every lane steps by 32.  An
  // excluded pair needs its minimum image, a matter of the float64 test.
  const int n0 = p.nimg[0], n1 = p.nimg[1], n2 = p.nimg[2];
  const int wn = __float_as_int(q.wi.w);
  const int step_z = 32 % n2, step_y = (32 / n2) % n1, step_x = (32 / n2 / n1) % n0, step_c = 32 / n2 / n1 / n0;
  int oz = lane % n2, oy = (lane / n2) % n1, ox = (lane / n2 / n1) % n0, c = lane / n2 / n1 / n0;
  const int first = __shfl_sync(0xffffffffu, rg.shift, 0);
  while (__any_sync(0xffffffffu, c < rg.total)) {
    bool hit = false;
    int j = 0, sh[3] = {0, 0, 0};
    if (c < rg.total) {
      const float4 w = cand[first + c];
      const int4 lb = label[first + c];
      j = __float_as_int(w.w);
      if (lb.x == q.inc) {
        const int o[3] = {ox - (n0 - 1) / 2, oy - (n1 - 1) / 2, oz - (n2 - 1) / 2};
        const bool same_ex = lb.y == q.exi;
        bool sure = !((wn | lb.z) & kWideImage);
        if (sure) {
          const float dx = (q.wi.x - w.x) + (float)(image_axis(wn, 0) - image_axis(lb.z, 0) - o[0]);
          const float dy = (q.wi.y - w.y) + (float)(image_axis(wn, 1) - image_axis(lb.z, 1) - o[1]);
          const float dz = (q.wi.z - w.z) + (float)(image_axis(wn, 2) - image_axis(lb.z, 2) - o[2]);
          const float X = fmaf(dz, q.L[3], fmaf(dy, q.L[1], dx * q.L[0])), Y = fmaf(dz, q.L[4], dy * q.L[2]),
                      Z = dz * q.L[5];
          const float d2 = fmaf(Z, Z, fmaf(Y, Y, X * X));
          if (d2 < q.hi2) {
            sure = d2 < q.lo2 && !same_ex;
            hit = sure;
#pragma unroll
            for (int a = 0; a < 3; ++a) sh[a] = o[a];
          }
        }
        if (!sure) hit = exact_pair(p, frac, q.i, j, o, true, same_ex, sh);
      }
    }
    emit(hit, j, sh);
    c += step_c;
    oz += step_z;
    oy += step_y;
    ox += step_x;
    if (oz >= n2) {
      oz -= n2;
      ++oy;
    }
    if (oy >= n1) {
      oy -= n1;
      ++ox;
    }
    if (ox >= n0) {
      ox -= n0;
      ++c;
    }
  }
}

struct PairSearch {
  const int32_t *system, *inclusion, *exclusion;
  int64_t n;
  int32_t n_incl, s;
  const SysNL *sys;
  const double *frac;
  const float4 *wrapped;
  const int *cell_of, *cell_start;
  const float4 *cand;
  const int4 *label;
};

// Whether the box of fractional offsets of centre c and half extents h may hold one whose nearest image
// has a squared length below r2: each Cartesian component is bounded over the box (z by the third offset
// alone, y by two, x by all three), an axis along which the box reaches past half a cell counts with both
// images.
__device__ inline bool offsets_within(const float c[3], const float h[3], const float L[6], float r2) {
  const float hx = h[0] * fabsf(L[0]) + h[1] * fabsf(L[1]) + h[2] * fabsf(L[3]);
  const float hy = h[1] * fabsf(L[2]) + h[2] * fabsf(L[4]), hz = h[2] * fabsf(L[5]);
  auto within = [&](float d0, float d1, float d2) {
    const float x = fmaxf(fabsf(d0 * L[0] + d1 * L[1] + d2 * L[3]) - hx, 0.f);
    const float y = fmaxf(fabsf(d1 * L[2] + d2 * L[4]) - hy, 0.f), z = fmaxf(fabsf(d2 * L[5]) - hz, 0.f);
    return x * x + y * y + z * z < r2;
  };
  if (within(c[0], c[1], c[2])) return true;
  int other = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) other |= (fabsf(c[a]) + h[a] > 0.4999f) << a;
  for (int k = 1; k < 8; ++k)
    if ((k & ~other) == 0 && within((k & 1) ? c[0] - copysignf(1.f, c[0]) : c[0],
                                    (k & 2) ? c[1] - copysignf(1.f, c[1]) : c[1],
                                    (k & 4) ? c[2] - copysignf(1.f, c[2]) : c[2]))
      return true;
  return false;
}

// The query of particle i and its candidate runs, by a whole warp; null if it has no edges.  Cells that
// the cutoff does not reach from where the particle lies in its own are left out (a third to a half of
// the candidates where an axis has four cells or more; hi2's margin and 1e-4 cover the float32 offsets).  `tmp`:
// 32 rows of shared memory of the warp's own.
__device__ const SysNL *pair_query(const PairSearch &a, int64_t i, PairQuery &q, CandRuns &rg, uint2 *tmp) {
  const int lane = threadIdx.x & 31;
  if (i >= a.n) return nullptr;
  const int32_t si = a.system[i], inc = a.inclusion[i];
  if (si < 0 || si >= a.s || inc < 0 || inc >= a.n_incl) return nullptr;
  const SysNL &p = a.sys[si];
  if (p.refused) return nullptr;
  q.i = (int)i;
  q.inc = inc;
  q.exi = a.exclusion[i];
  q.wi = a.wrapped[i];
  q.lo2 = p.lo2;
  q.hi2 = p.hi2;
  q.tie = p.tie;
#pragma unroll
  for (int k = 0; k < 6; ++k) q.L[k] = p.Lf[k];
  int first = 0, len = 0;
  if (lane < kNLCells) {
    const int nx = p.nc[0], ny = p.nc[1], nz = p.nc[2];
    const int ci = a.cell_of[i] - (int)p.cell_base;
    const int cx = ci % nx, cy = (ci / nx) % ny, cz = ci / (nx * ny);
    // the distinct neighbour cells of an axis (1, 2 or 3 of them), in this order
    auto axis = [](int c, int nc, int t, int &out) {
      out = c + t - 1;
      if (nc <= 2) out = t;
      else if (out < 0) out += nc;
      else if (out >= nc) out -= nc;
      return t < min(nc, 3);
    };
    int x, y, z;
    if (axis(cx, nx, lane % 3, x) & axis(cy, ny, (lane / 3) % 3, y) & axis(cz, nz, lane / 9, z)) {
      const int c = (int)p.cell_base + (z * ny + y) * nx + x;
      float centre[3], half[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const int m = k == 0 ? nx : k == 1 ? ny : nz, at = k == 0 ? cx : k == 1 ? cy : cz;
        const int t = (k == 0 ? lane % 3 : k == 1 ? (lane / 3) % 3 : lane / 9) - 1;
        const float w = k == 0 ? q.wi.x : k == 1 ? q.wi.y : q.wi.z;
        float u = (w - floorf(w)) * (float)m - (float)at;  // place in the own cell, of m cells around
        u -= (float)m * rintf(u / (float)m);
        centre[k] = m > 2 ? (u - (float)t - 0.5f) / (float)m : 0.f;
        half[k] = m > 2 ? 0.5f / (float)m : 1.f;
      }
      if (offsets_within(centre, half, q.L, 1.0001f * q.hi2)) {
        first = a.cell_start[c];
        len = a.cell_start[c + 1] - first;
      }
    }
  }
  int sum = len;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, sum, o);
    if (lane >= o) sum += v;
  }
  rg.total = __shfl_sync(0xffffffffu, sum, 31);
  // the non-empty runs to the leading lanes, in order
  const unsigned full = __ballot_sync(0xffffffffu, len > 0);
  if (len > 0) tmp[__popc(full & ((1u << lane) - 1u))] = make_uint2((unsigned)(sum - len), (unsigned)first);
  __syncwarp();
  const uint2 run = lane < __popc(full) ? tmp[lane] : make_uint2(0x7fffffffu, 0u);
  rg.begin = (int)run.x;
  rg.shift = (int)(run.y - run.x);
  __syncwarp();
  return &p;
}

// The edge list in one pass: a warp per particle (index order) finds its edges into shared memory,
// the block's count joins the chained prefix over blocks, and the rows are written at their final
// place with coalesced stores.  With `defer`, blocks take the next eight particles before they resolve
// the prefix of the last eight, so no warp waits for a slower predecessor (with a wait after every
// search a third of the warps' time went into it); a list of few groups takes one buffer instead, so
// that more blocks fit an SM (4000 ions with 450 edges each: 85 against 124 us).  A particle whose edges
// do not fit its `room` rows, or with shifts beyond 10 bits, is searched again to write them.  Bounded
// by issue: about 40 instructions per 32 candidates, and 80 per 32 edges.  264 k particles in 256
// systems (about 500 candidates each, 350 in cells within reach): 0.70 ms (0.73 ms with all 27 cells,
// 0.89 ms with the wait, 1.29 ms also with labels and shifts taken up candidate by candidate); the
// float64 test per candidate (30 operations at 2 per clock per SM, one thread per particle, a counting
// and a writing pass) took 19.3 ms.
__global__ void __launch_bounds__(32 * kPairWarps, 4) pairs_kernel(PairSearch a, int room, bool defer, int64_t n_groups,
                                                                   unsigned *ticket, unsigned long long *state,
                                                                   int64_t *n_edges, int32_t *edges, int32_t *shifts,
                                                                   int64_t cap, kups_status *status) {
  extern __shared__ uint2 stage_all[];  // [1 + defer][kPairWarps][room]
  __shared__ int counts[2][kPairWarps];
  __shared__ int64_t base;
  __shared__ unsigned next;
  __shared__ bool chained;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  int64_t last = -1;  // the group found but not yet written
  int last_cnt = 0;
  bool last_again = false;
  for (int buf = 0;; buf ^= defer) {
    if (threadIdx.x == 0) next = atomicAdd(ticket, 1u);
    __syncthreads();
    const int64_t group = next < n_groups ? (int64_t)next : -1;
    if (group < 0 && last < 0) return;
    uint2 *stage = stage_all + (size_t)(buf * kPairWarps + warp) * room;
    PairQuery q;
    CandRuns rg;
    int cnt = 0;
    bool again = false;
    if (group >= 0) {
      const SysNL *p = pair_query(a, group * kPairWarps + warp, q, rg, stage);
      if (p != nullptr) {  // the same for the whole warp
        cnt = p->image_mode ? -1 : search_staged(*p, q, rg, a.cand, a.label, a.frac, stage, room);
        if (cnt < 0) {
          cnt = 0;
          search_each(*p, q, rg, a.cand, a.label, a.frac, [&](bool hit, int j, const int *sh) {
            const unsigned m = __ballot_sync(0xffffffffu, hit);
            const int at = cnt + __popc(m & below);
            if (hit) {
              again |= !fits_packed(sh) || at >= room;
              if (at < room) stage[at] = make_uint2((unsigned)j, pack_shift(sh));
            }
            cnt += __popc(m);
          });
          again = __any_sync(0xffffffffu, again);
        }
      }
    }
    if (lane == 0) counts[buf][warp] = cnt;
    __syncthreads();
    const int done_buf = defer ? buf ^ 1 : buf;
    if (!defer) {
      last = group;
      last_cnt = cnt;
      last_again = again;
    }
    if (warp == 0) {  // this group's count for the blocks behind, then the place of the last group
      int own = 0, before_own = 0;
#pragma unroll
      for (int k = 0; k < kPairWarps; ++k) {
        own += counts[buf][k];
        before_own += counts[done_buf][k];
      }
      if (group >= 0) chained_publish(state, group, own);
      if (last >= 0) {
        bool ok;
        const int64_t before = chained_prefix(state, last, before_own, ok);
        if (lane == 0) {
          base = before;
          chained = ok;
          if (!ok) status_error(status, KUPS_ERR_UNSUPPORTED, last);
          if (last == n_groups - 1) {
            const int64_t all = ok ? before + before_own : 0;
            *n_edges = all;
            if (all > cap) status_capacity(status, KUPS_CAP_EDGES, all, -1);
          }
        }
      }
    }
    __syncthreads();
    if (last >= 0 && chained && last_cnt > 0) {
      const int64_t i = last * kPairWarps + warp;
      uint2 *done = stage_all + (size_t)(done_buf * kPairWarps + warp) * room;
      int64_t out = base;
      for (int k = 0; k < warp; ++k) out += counts[done_buf][k];
      if (last_again) {
        PairQuery ql;
        CandRuns rl;
        const SysNL *p = pair_query(a, i, ql, rl, done);
        search_each(*p, ql, rl, a.cand, a.label, a.frac, [&](bool hit, int j, const int *sh) {
          const unsigned m = __ballot_sync(0xffffffffu, hit);
          const int64_t o = out + __popc(m & below);
          if (hit && o < cap) {
            edges[2 * o] = (int32_t)i;
            edges[2 * o + 1] = j;
            for (int k = 0; k < 3; ++k) shifts[3 * o + k] = sh[k];
          }
          out += __popc(m);
        });
      } else {
        const int rows = (int)max((int64_t)0, min((int64_t)last_cnt, cap - out));
        for (int t = lane; t < 2 * rows; t += 32) edges[2 * out + t] = (t & 1) ? (int)done[t >> 1].x : (int)i;
        for (int t = lane; t < 3 * rows; t += 32) {
          const int e = t / 3;
          shifts[3 * out + t] = image_axis((int)done[e].y, t - 3 * e);
        }
      }
    }
    last = defer ? group : -1;
    last_cnt = cnt;
    last_again = again;
  }
}

// Rows a warp stages: twice the edge rows per particle that the caller allots (a guess at the longest
// list), 64 to 512; more only costs resident blocks, fewer a second search.
inline int pair_room(int64_t cap, int64_t n) {
  const int64_t want = 2 * (cap / std::max<int64_t>(n, 1));
  return (int)std::min<int64_t>(512, std::max<int64_t>(64, (want + 31) / 32 * 32));
}

__global__ void check_capacity_kernel(const int64_t *n_edges, int64_t cap, kups_status *st) {
  if (*n_edges > cap) status_capacity(st, KUPS_CAP_EDGES, *n_edges, -1);
}

// Rows [n_edges, cap) hold index n and a zero shift; a fixed grid walks from the first of them, so a
// nearly full list costs nothing.
__global__ void pad_kernel(const int64_t *n_edges, int64_t cap, int64_t n, int32_t *edges,
                           int32_t *shifts) {
  const int64_t first = *n_edges, step = (int64_t)gridDim.x * blockDim.x;
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int64_t t = 2 * first + t0; t < 2 * cap; t += step) edges[t] = (int32_t)n;
  for (int64_t t = 3 * first + t0; t < 3 * cap; t += step) shifts[t] = 0;
}

inline unsigned pad_blocks(int64_t cap) {
  return (unsigned)std::min<int64_t>((cap + 255) / 256, 8 * (int64_t)device_sm_count());
}

// Cells, candidate records and per-system parameters of a particle table (both searches start here).
cudaError_t bin_particles(const NLWork &w, const double *positions, const int32_t *system, const int32_t *inclusion,
                          const int32_t *exclusion, int64_t n, const double *tril, const double *cutoffs, int32_t s,
                          kups_status *status, cudaStream_t stream) {
  const unsigned gb = (unsigned)((n + 255) / 256);
  cudaError_t e = cudaMemsetAsync(w.zero, 0, w.zero_bytes, stream);
  if (e != cudaSuccess) return e;
  count_atoms_kernel<<<gb, 256, 0, stream>>>(system, n, s, w.sys);
  setup_systems_kernel<<<(unsigned)((s + kSetupSystems - 1) / kSetupSystems), 4 * kSetupSystems, 0, stream>>>(
      tril, cutoffs, s, w.sys, w.tickets, status);
  bin_kernel<<<gb, 256, 0, stream>>>(positions, system, n, s, w.sys, w.frac, w.wrapped, w.cell_of, w.slot_of,
                                     w.cell_start);
  chained_scan_kernel<<<(unsigned)w.scan_blocks, kChainedThreads, 0, stream>>>(w.cell_start, w.n_cells_cap + 1,
                                                                               w.scan_state, w.tickets + 1, status);
  scatter_kernel<<<gb, 256, 0, stream>>>(w.cell_of, w.slot_of, n, w.cell_start, w.cell_any);
  order_cells_kernel<<<gb, 256, 0, stream>>>(w.cell_of, n, w.cell_start, w.cell_any, w.wrapped, inclusion, exclusion,
                                             w.cell_items, w.cand, w.cand_label);
  return cudaGetLastError();
}

}  // namespace
}  // namespace kups

using namespace kups;

extern "C" size_t kups_neighborlist_workspace_bytes(int64_t n_particles, int32_t n_systems) {
  return layout(nullptr, nullptr, n_particles, n_systems) + 256;
}

extern "C" int32_t kups_neighborlist_build(const double *positions, const int32_t *system,
                                           const int32_t *inclusion, const int32_t *exclusion,
                                           int64_t n, int32_t n_incl, const double *tril,
                                           const double *cutoffs, int32_t s, int32_t *edges,
                                           int32_t *shifts, int64_t cap, int64_t *n_edges,
                                           void *workspace, size_t ws_bytes,
                                           kups_status *status, void *stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (n < 0 || s < 0 || cap < 0 || n >= (int64_t)INT32_MAX) return KUPS_ERR_INVALID;
  if (ws_bytes < kups_neighborlist_workspace_bytes(n, s)) return KUPS_ERR_INVALID;
  char *base = (char *)(((uintptr_t)workspace + 255) & ~uintptr_t(255));
  NLWork w;
  layout(&w, base, n, s);
  if (s == 0 || n == 0) {
    KUPS_CUDA_TRY(cudaMemsetAsync(n_edges, 0, sizeof(int64_t), stream));
    if (cap > 0) pad_kernel<<<pad_blocks(cap), 256, 0, stream>>>(n_edges, cap, n, edges, shifts);
    return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
  }
  KUPS_CUDA_TRY(bin_particles(w, positions, system, inclusion, exclusion, n, tril, cutoffs, s, status, stream));
  const PairSearch a{system,    inclusion,    exclusion, n,      n_incl,      s,      w.sys,
                     w.frac, w.wrapped, w.cell_of, w.cell_start, w.cand, w.cand_label};
  const int room = pair_room(cap, n);
  // at most two groups for each block that can be resident: one wave, nothing to defer behind
  const bool defer = w.pair_blocks > 8 * (int64_t)device_sm_count();
  const size_t smem = sizeof(uint2) * (defer ? 2 : 1) * kPairWarps * (size_t)room;
  KUPS_CUDA_TRY(cudaFuncSetAttribute(pairs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(sizeof(uint2) * 2 * kPairWarps * 512)));
  const unsigned blocks = (unsigned)std::min<int64_t>(w.pair_blocks, 4 * (int64_t)device_sm_count());
  pairs_kernel<<<blocks, 32 * kPairWarps, smem, stream>>>(a, room, defer, w.pair_blocks, w.tickets + 2, w.pair_state,
                                                          n_edges, edges, shifts, cap, status);
  if (cap > 0) pad_kernel<<<pad_blocks(cap), 256, 0, stream>>>(n_edges, cap, n, edges, shifts);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

// ---------------------------------------------------------------------------
// rh subset: edges (i in lh, j in rh) within the cutoff of the pair's system,
// the rh particles given separately (NearestNeighborList.__call__ with rh,
// src/kups/core/neighborlist.py:226-255; basic_neighborlist :743-786).  The lh
// particles are binned into the cell grid of the full mode; each rh particle
// scans the lh cells around its own cell.  Candidate rules as the reference's
// _build_segmentation_mask (:505-539), _filter_candidates (:692-740) and
// _compact_edges (:651-689):
//   * same system, same valid inclusion label (lh and rh labels);
//   * the image rule and strict d^2 < rc^2 of the full mode, difference lh - rh;
//   * exclusion labels equal (lh vs rh) drop the minimum image only;
//   * with rh_index_remap (rh particle j stands for lh particle remap[j]):
//     a pair whose lh particle is itself one of the remapped ones is kept only
//     for i >= remap[j], and every edge (i, remap[j], s) is written together
//     with its reverse (remap[j], i, -s);
//   * without remap, edges are (i, j) with j indexing rh.
// Padding rows hold max(n_lh, n_rh).
namespace kups {
namespace {

struct RhWork {
  NLWork lh;
  uint8_t *in_remap;  // [n_lh]: lh particle i is some remap[j]
  int64_t *rh_off;    // [n_rh + 1]
  int64_t *rh_scan;   // scan block sums
};

size_t rh_layout(RhWork *w, char *base, int64_t n_lh, int64_t n_rh, int32_t s) {
  size_t off = layout(w ? &w->lh : nullptr, base, n_lh, s);
  auto take = [&](size_t bytes) {
    char *p = base ? base + off : nullptr;
    off += align_up(bytes);
    return p;
  };
  uint8_t *flags = (uint8_t *)take((size_t)std::max<int64_t>(n_lh, 1));
  int64_t *roff = (int64_t *)take(sizeof(int64_t) * (size_t)(n_rh + 1));
  int64_t *rscan = (int64_t *)take(sizeof(int64_t) * (size_t)scan_blocks_needed(n_rh + 1));
  if (w) {
    w->in_remap = flags;
    w->rh_off = roff;
    w->rh_scan = rscan;
  }
  return off;
}

__global__ void mark_remap_kernel(const int32_t *remap, int64_t n_rh, int64_t n_lh, uint8_t *flags) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n_rh) return;
  const int32_t r = remap[j];
  if (r >= 0 && r < n_lh) flags[r] = 1;
}

template <bool WRITE>
__global__ void pairs_rh_kernel(const int32_t *lh_incl, const int32_t *lh_excl, int64_t n_lh,
                                const double *rh_pos, const int32_t *rh_system, const int32_t *rh_incl,
                                const int32_t *rh_excl, int64_t n_rh, const int32_t *remap,
                                const uint8_t *in_remap, int32_t n_incl, int32_t s, const SysNL *sys,
                                const double *frac, const int *cell_start, const int *cell_items,
                                int64_t *rh_off, int64_t oob, int32_t *edges, int32_t *shifts, int64_t cap) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n_rh) return;
  const int32_t sj = rh_system[j];
  const int32_t inc = rh_incl[j];
  int64_t count = 0;
  int64_t out = WRITE ? rh_off[j] : 0;
  if (sj >= 0 && sj < s && inc >= 0 && inc < n_incl && !sys[sj].refused) {
    const SysNL p = sys[sj];
    const double r[3] = {rh_pos[3 * j], rh_pos[3 * j + 1], rh_pos[3 * j + 2]};
    double fj[3];
    row_times_tril64(r, p.inv, fj);
    const int cx = wrap_cell(fj[0], p.nc[0]), cy = wrap_cell(fj[1], p.nc[1]), cz = wrap_cell(fj[2], p.nc[2]);
    const int32_t exj = rh_excl[j];
    const int64_t ro = remap != nullptr ? (int64_t)remap[j] : j;
    int lx[3], ly[3], lz[3], nx, ny, nz;
    auto axis = [](int c, int nc, int *l, int &m) {
      if (nc == 1) {
        l[0] = 0;
        m = 1;
      } else if (nc == 2) {
        l[0] = 0;
        l[1] = 1;
        m = 2;
      } else {
        l[0] = (c + nc - 1) % nc;
        l[1] = c;
        l[2] = (c + 1) % nc;
        m = 3;
      }
    };
    axis(cx, p.nc[0], lx, nx);
    axis(cy, p.nc[1], ly, ny);
    axis(cz, p.nc[2], lz, nz);
    const int hx = (p.nimg[0] - 1) / 2, hy = (p.nimg[1] - 1) / 2, hz = (p.nimg[2] - 1) / 2;
    auto emit = [&](int i, const int sh[3]) {
      if (WRITE) {
        if (out < cap) {
          edges[2 * out] = i;
          edges[2 * out + 1] = (int32_t)ro;
          shifts[3 * out] = sh[0];
          shifts[3 * out + 1] = sh[1];
          shifts[3 * out + 2] = sh[2];
        }
        ++out;
        if (remap != nullptr) {
          if (out < cap) {
            edges[2 * out] = (int32_t)ro;
            edges[2 * out + 1] = i;
            shifts[3 * out] = -sh[0];
            shifts[3 * out + 1] = -sh[1];
            shifts[3 * out + 2] = -sh[2];
          }
          ++out;
        }
      }
      count += remap != nullptr ? 2 : 1;
    };
    for (int az = 0; az < nz; ++az)
      for (int ay = 0; ay < ny; ++ay)
        for (int ax = 0; ax < nx; ++ax) {
          const int c = (int)p.cell_base + (lz[az] * p.nc[1] + ly[ay]) * p.nc[0] + lx[ax];
          const int b = cell_start[c], e = cell_start[c + 1];
          for (int k = b; k < e; ++k) {
            const int i = cell_items[k];
            if (lh_incl[i] != inc) continue;
            if (remap != nullptr && in_remap[i] && !((int64_t)i >= ro)) continue;
            const double fi[3] = {frac[3 * i], frac[3 * i + 1], frac[3 * i + 2]};
            const bool same_ex = lh_excl[i] == exj;
            int sh[3];
            if (!p.image_mode) {
              const int o[3] = {0, 0, 0};
              if (edge_test(p, fi, fj, o, false, sh, same_ex)) emit(i, sh);
            } else {
              for (int ox = -hx; ox <= hx; ++ox)
                for (int oy = -hy; oy <= hy; ++oy)
                  for (int oz = -hz; oz <= hz; ++oz) {
                    const int o[3] = {ox, oy, oz};
                    if (edge_test(p, fi, fj, o, true, sh, same_ex)) emit(i, sh);
                  }
            }
          }
        }
  }
  (void)oob;
  if (!WRITE) rh_off[j] = count;
}

// neighborlist_changes' split of the combined call (src/kups/core/neighborlist.py:1425-1515):
// removed = both ends < n (old positions), added = an end >= n (a new position) and no end
// that is the old copy of a changed particle; appended indices n + m become p_idx[m].
__global__ void split_flags_kernel(const int32_t *edges, const int64_t *n_edges, int64_t n, int64_t k,
                                   const uint8_t *is_changed, int64_t *add_flag, int64_t *rem_flag, int64_t total) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= total) return;
  int64_t a = 0, r = 0;
  if (e < *n_edges && e < total - 1) {  // entry total - 1 only closes the scan
    const int64_t c0 = edges[2 * e], c1 = edges[2 * e + 1];
    r = (c0 < n) && (c1 < n);
    const bool stale = ((c0 < n) && is_changed[c0]) || ((c1 < n) && is_changed[c1]);
    a = (c0 < n + k) && (c1 < n + k) && ((c0 >= n) || (c1 >= n)) && !stale;
  }
  add_flag[e] = a;
  rem_flag[e] = r;
}

__global__ void split_write_kernel(const int32_t *edges, const int32_t *shifts, const int64_t *n_edges, int64_t n,
                                   const int32_t *p_idx, const int64_t *add_off, const int64_t *rem_off,
                                   int64_t total, int32_t *add_e, int32_t *add_s, int64_t add_cap, int32_t *rem_e,
                                   int32_t *rem_s, int64_t rem_cap) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= total || e >= *n_edges) return;
  const bool a = add_off[e + 1] > add_off[e], r = rem_off[e + 1] > rem_off[e];
  if (!a && !r) return;
  int64_t c[2] = {edges[2 * e], edges[2 * e + 1]};
  for (int t = 0; t < 2; ++t)
    if (c[t] >= n) c[t] = p_idx[c[t] - n];
  int32_t *oe = a ? add_e : rem_e;
  int32_t *os = a ? add_s : rem_s;
  const int64_t slot = a ? add_off[e] : rem_off[e];
  if (slot >= (a ? add_cap : rem_cap)) return;
  oe[2 * slot] = (int32_t)c[0];
  oe[2 * slot + 1] = (int32_t)c[1];
  for (int t = 0; t < 3; ++t) os[3 * slot + t] = shifts[3 * e + t];
}

__global__ void pad_from_kernel(const int64_t *count, int64_t cap, int64_t fill, int32_t *edges, int32_t *shifts) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= cap || e < *count) return;
  edges[2 * e] = (int32_t)fill;
  edges[2 * e + 1] = (int32_t)fill;
  shifts[3 * e] = shifts[3 * e + 1] = shifts[3 * e + 2] = 0;
}

__global__ void split_check_kernel(const int64_t *n_add, int64_t add_cap, const int64_t *n_rem, int64_t rem_cap,
                                   kups_status *st) {
  if (*n_add > add_cap) status_capacity(st, KUPS_CAP_EDGES, *n_add, -1);
  if (*n_rem > rem_cap) status_capacity(st, KUPS_CAP_EDGES, *n_rem, -1);
}

__global__ void mark_changed_kernel(const int32_t *p_idx, int64_t k, int64_t n, uint8_t *is_changed) {
  const int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (m < k && p_idx[m] >= 0 && p_idx[m] < n) is_changed[p_idx[m]] = 1;
}

}  // namespace
}  // namespace kups

extern "C" size_t kups_neighborlist_rh_workspace_bytes(int64_t n_lh, int64_t n_rh, int32_t n_systems) {
  return rh_layout(nullptr, nullptr, n_lh, n_rh, n_systems) + 256;
}

extern "C" int32_t kups_neighborlist_build_rh(
    const double *lh_positions, const int32_t *lh_system, const int32_t *lh_inclusion, const int32_t *lh_exclusion,
    int64_t n_lh, const double *rh_positions, const int32_t *rh_system, const int32_t *rh_inclusion,
    const int32_t *rh_exclusion, int64_t n_rh, const int32_t *rh_index_remap, int32_t n_incl, const double *tril,
    const double *cutoffs, int32_t s, int32_t *edges, int32_t *shifts, int64_t cap, int64_t *n_edges,
    void *workspace, size_t ws_bytes, kups_status *status, void *stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (n_lh < 0 || n_rh < 0 || s < 0 || cap < 0 || n_lh >= (int64_t)INT32_MAX || n_rh >= (int64_t)INT32_MAX)
    return KUPS_ERR_INVALID;
  if (ws_bytes < kups_neighborlist_rh_workspace_bytes(n_lh, n_rh, s)) return KUPS_ERR_INVALID;
  const int64_t oob = std::max(n_lh, n_rh);
  char *base = (char *)(((uintptr_t)workspace + 255) & ~uintptr_t(255));
  RhWork w;
  rh_layout(&w, base, n_lh, n_rh, s);
  KUPS_CUDA_TRY(cudaMemsetAsync(n_edges, 0, sizeof(int64_t), stream));
  if (s == 0 || n_lh == 0 || n_rh == 0) {
    if (cap > 0) pad_kernel<<<pad_blocks(cap), 256, 0, stream>>>(n_edges, cap, oob, edges, shifts);
    return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
  }
  const int64_t n = n_lh;
  NLWork &l = w.lh;
  KUPS_CUDA_TRY(cudaMemsetAsync(w.in_remap, 0, (size_t)std::max<int64_t>(n, 1), stream));
  KUPS_CUDA_TRY(bin_particles(l, lh_positions, lh_system, lh_inclusion, lh_exclusion, n, tril, cutoffs, s, status,
                              stream));
  if (rh_index_remap != nullptr)
    mark_remap_kernel<<<(unsigned)((n_rh + 255) / 256), 256, 0, stream>>>(rh_index_remap, n_rh, n, w.in_remap);
  const unsigned gr = (unsigned)((n_rh + 127) / 128);
  pairs_rh_kernel<false><<<gr, 128, 0, stream>>>(lh_inclusion, lh_exclusion, n, rh_positions, rh_system,
                                                 rh_inclusion, rh_exclusion, n_rh, rh_index_remap, w.in_remap,
                                                 n_incl, s, l.sys, l.frac, l.cell_start, l.cell_items, w.rh_off, oob,
                                                 edges, shifts, cap);
  KUPS_CUDA_TRY(exclusive_scan<int64_t>(w.rh_off, n_rh, w.rh_scan, n_edges, stream));
  pairs_rh_kernel<true><<<gr, 128, 0, stream>>>(lh_inclusion, lh_exclusion, n, rh_positions, rh_system,
                                                rh_inclusion, rh_exclusion, n_rh, rh_index_remap, w.in_remap, n_incl,
                                                s, l.sys, l.frac, l.cell_start, l.cell_items, w.rh_off, oob, edges,
                                                shifts, cap);
  check_capacity_kernel<<<1, 1, 0, stream>>>(n_edges, cap, status);
  if (cap > 0) pad_kernel<<<pad_blocks(cap), 256, 0, stream>>>(n_edges, cap, oob, edges, shifts);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

extern "C" size_t kups_neighborlist_split_workspace_bytes(int64_t n_edges_total, int64_t n) {
  const int64_t m = n_edges_total + 1;
  return 2 * align_up(sizeof(int64_t) * (size_t)m) + 2 * align_up(sizeof(int64_t) * (size_t)scan_blocks_needed(m)) +
         align_up((size_t)std::max<int64_t>(n, 1)) + 256;
}

extern "C" int32_t kups_neighborlist_split_changes(const int32_t *edges, const int32_t *shifts,
                                                   const int64_t *n_edges, int64_t edge_rows, int64_t n,
                                                   const int32_t *p_idx, int64_t k, int32_t *added_edges,
                                                   int32_t *added_shifts, int64_t added_cap, int64_t *n_added,
                                                   int32_t *removed_edges, int32_t *removed_shifts,
                                                   int64_t removed_cap, int64_t *n_removed, void *workspace,
                                                   size_t ws_bytes, kups_status *status, void *stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (edge_rows < 0 || n < 0 || k < 0 || added_cap < 0 || removed_cap < 0) return KUPS_ERR_INVALID;
  if (ws_bytes < kups_neighborlist_split_workspace_bytes(edge_rows, n)) return KUPS_ERR_INVALID;
  const int64_t m = edge_rows + 1;
  char *base = (char *)(((uintptr_t)workspace + 255) & ~uintptr_t(255));
  int64_t *add_off = (int64_t *)base;
  int64_t *rem_off = (int64_t *)(base + align_up(sizeof(int64_t) * (size_t)m));
  int64_t *scan_a = (int64_t *)(base + 2 * align_up(sizeof(int64_t) * (size_t)m));
  int64_t *scan_r = (int64_t *)((char *)scan_a + align_up(sizeof(int64_t) * (size_t)scan_blocks_needed(m)));
  uint8_t *changed = (uint8_t *)((char *)scan_r + align_up(sizeof(int64_t) * (size_t)scan_blocks_needed(m)));
  KUPS_CUDA_TRY(cudaMemsetAsync(changed, 0, (size_t)std::max<int64_t>(n, 1), stream));
  if (k > 0) mark_changed_kernel<<<(unsigned)((k + 255) / 256), 256, 0, stream>>>(p_idx, k, n, changed);
  const unsigned g = (unsigned)((m + 255) / 256);
  split_flags_kernel<<<g, 256, 0, stream>>>(edges, n_edges, n, k, changed, add_off, rem_off, m);
  KUPS_CUDA_TRY(exclusive_scan<int64_t>(add_off, m, scan_a, n_added, stream));
  KUPS_CUDA_TRY(exclusive_scan<int64_t>(rem_off, m, scan_r, n_removed, stream));
  split_write_kernel<<<g, 256, 0, stream>>>(edges, shifts, n_edges, n, p_idx, add_off, rem_off, edge_rows,
                                            added_edges, added_shifts, added_cap, removed_edges, removed_shifts,
                                            removed_cap);
  split_check_kernel<<<1, 1, 0, stream>>>(n_added, added_cap, n_removed, removed_cap, status);
  if (added_cap > 0)
    pad_from_kernel<<<(unsigned)((added_cap + 255) / 256), 256, 0, stream>>>(n_added, added_cap, n, added_edges,
                                                                            added_shifts);
  if (removed_cap > 0)
    pad_from_kernel<<<(unsigned)((removed_cap + 255) / 256), 256, 0, stream>>>(n_removed, removed_cap, n,
                                                                              removed_edges, removed_shifts);
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}
