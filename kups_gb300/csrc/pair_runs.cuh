// Pair energies, dE/dx and dE/dtril over a directed edge list, shared by the Lennard-Jones and the
// LJ + Ewald edge kernels.
//
// What bounds them is the float64 pipe (2 operations per clock per SM) and the float64 atomics, so
// the layout spends neither where it can be helped:
//  * a warp reads its edges 32 at a time (coalesced), drops padding rows, and collects the edges to
//    evaluate in shared memory; each lane then takes a few consecutive ones, which in a list grouped
//    by the first particle mostly share it: its forces add up in registers and go out with one atomic
//    per component per run (a shuffle tree over the warp costs five float64 additions per edge and
//    component, an atomic per edge as much traffic again as the second particle's);
//  * with PAIRED the list is known to hold every edge together with its reverse (what the neighbour
//    list writes): only one of the two is evaluated, with twice its weight, unless the species tables
//    are not symmetric and the two differ.  Every block looks through the tables first, which leaves
//    the loop over pairs as it is (a test of the species pair in there made pair_edges 10 % slower);
//  * edges with and without an image shift are collected apart, so that the shift's three float64
//    additions and the six of dE/dtril are spent on shifted edges only, with every lane at work
//    (mixed, 40 float64 instructions were issued per 32 pairs of which 17 lanes' worth did work);
//    a shift of 0 or +-1 times a cell vector is a selection and a sign, and cells without
//    off-diagonal entries add one term per axis.
// Per-system sums leave as one atomic per warp while it stays in one system.
#pragma once

#include "common.cuh"

namespace kups {

struct PairList {
  const double *pos;
  const int32_t *system;
  int64_t n;
  const double *tril;
  int32_t s;
  const int32_t *edges, *shifts;
  int64_t n_edges;
  double *energy, *grad, *grad_tril;
  int64_t edges_per_warp;  // a multiple of 128
};

constexpr int kRunWarps = 4;    // warps per block
constexpr int kRunQueue = 256;  // edges a warp holds: fewer than 128 left over + 128 read

// s * v for a small integer s, exactly as the product rounds (s v is exact for s in {-1, 0, 1}).
__device__ inline double shift_times(int s, double v) {
  if (s == 0) return 0.0;
  if (s == 1) return v;
  if (s == -1) return -v;
  return __dmul_rn((double)s, v);
}

// (double)s, without a conversion (which takes the float64 pipe's time) for s in {-1, 0, 1}.
__device__ inline double shift_double(int s) {
  if (s >= -1 && s <= 1) return __hiloint2double(s == 0 ? 0 : 0x3ff00000 | (s & (int)0x80000000), 0);
  return (double)s;
}

// s @ L for small integers s (the sums in the order of row_times_tril64).
__device__ inline void shift_vector(const int s[3], const Tril64 &L, double y[3]) {
  y[0] = shift_times(s[0], L.t[0]);
  y[1] = shift_times(s[1], L.t[2]);
  y[2] = shift_times(s[2], L.t[5]);
  // (a test of the bits: float64 comparisons take the float64 pipe)
  const long long skew = __double_as_longlong(L.t[1]) | __double_as_longlong(L.t[3]) | __double_as_longlong(L.t[4]);
  if ((skew << 1) != 0) {
    y[0] = __dadd_rn(__dadd_rn(y[0], shift_times(s[1], L.t[1])), shift_times(s[2], L.t[3]));
    y[1] = __dadd_rn(y[1], shift_times(s[2], L.t[4]));
  }
}

__device__ inline bool finite64(double v) { return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000; }

template <bool B>
struct Const {
  static constexpr bool value = B;
};

// Species up to which a block looks through the tables; with more, every edge is evaluated.  14 M edges,
// float32 pairs: 528 us with one species, 548 with 32, against 824 edge by edge (at 32 the look takes 4 us
// of a kernel's start).
constexpr int kTableSpecies = 32;

// Whether two tables [n, n] are symmetric, by a whole block.
__device__ inline bool tables_symmetric(const double *a, const double *b, int n) {
  bool same = true;
  for (int k = threadIdx.x; k < n * n; k += blockDim.x) {
    const int i = k / n, j = k - i * n;
    if (i < j) same = same && a[k] == a[j * n + i] && b[k] == b[j * n + i];
  }
  return __syncthreads_and(same);
}

// Eval: load_system(s), load_first(i), and eval(e, j, r2, en, dedr2): energy and dE/d(r^2) of edge e.
// symmetric (PAIRED): whether an edge and its reverse carry the same terms.
template <bool PAIRED, typename Eval>
__device__ void run_pairs(const PairList &p, Eval &ev, bool symmetric) {
  // edges to evaluate: [0] without a shift, [1] shifted; qe: the edge's number from the warp's first
  // (a report names it)
  __shared__ int q_i[kRunWarps][2][kRunQueue], q_j[kRunWarps][2][kRunQueue], q_e[kRunWarps][2][kRunQueue];
  __shared__ int q_s[kRunWarps][3][kRunQueue];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int *q0 = q_s[warp][0], *q1 = q_s[warp][1], *q2 = q_s[warp][2];
  const int64_t w = (int64_t)blockIdx.x * kRunWarps + warp;
  const int64_t e0 = w * p.edges_per_warp, e1 = min(p.n_edges, e0 + p.edges_per_warp);
  if (e0 >= e1) return;  // the same for the whole warp; no block barrier below
  int sys = -1, fi = -1;
  double en_sum = 0.0, dl[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, gi[3] = {0.0, 0.0, 0.0}, xi[3] = {0.0, 0.0, 0.0};
  Tril64 L;
  bool any_dl = false;
  const bool single = PAIRED && symmetric;  // one edge of each pair
  const double share = single ? 1.0 : 0.5;  // of an edge's energy
  auto flush_first = [&]() {
    if (fi >= 0)
      for (int a = 0; a < 3; ++a) atomicAdd(&p.grad[3 * (int64_t)fi + a], gi[a]);
    gi[0] = gi[1] = gi[2] = 0.0;
  };
  auto flush_system = [&]() {  // this lane's sums of the system it leaves
    if (sys >= 0) {
      atomicAdd(&p.energy[sys], share * en_sum);
      if (any_dl && p.grad_tril)
        for (int a = 0; a < 6; ++a) atomicAdd(&p.grad_tril[6 * (int64_t)sys + a], dl[a]);
    }
    en_sum = 0.0;
    for (int a = 0; a < 6; ++a) dl[a] = 0.0;
    any_dl = false;
  };
  // evaluates the first `count` edges of a queue, `per` consecutive ones per lane
  auto evaluate = [&](auto shifted, int count, int per) {
    constexpr bool kShifted = decltype(shifted)::value;
    const int *qi = q_i[warp][kShifted], *qj = q_j[warp][kShifted], *qe = q_e[warp][kShifted];
    const int k1 = min(count, (lane + 1) * per);
    for (int k = lane * per; k < k1; ++k) {
      const int i = qi[k], j = qj[k];
      int s0 = 0, s1 = 0, s2 = 0;
      if (kShifted) {
        s0 = q0[k];
        s1 = q1[k];
        s2 = q2[k];
      }
      if (i != fi) {
        flush_first();
        fi = i;
        const int si = p.system[i];
        if (si != sys) {
          flush_system();
          sys = si;
          L = load_tril64(p.tril + 6 * (int64_t)si);
          ev.load_system(si);
        }
        for (int a = 0; a < 3; ++a) xi[a] = p.pos[3 * (int64_t)i + a];
        ev.load_first(i);
      }
      const double *xj = p.pos + 3 * (int64_t)j;
      double d[3] = {xj[0] - xi[0], xj[1] - xi[1], xj[2] - xi[2]};
      if (kShifted) {
        const int sh[3] = {s0, s1, s2};
        double y[3];
        shift_vector(sh, L, y);
        for (int a = 0; a < 3; ++a) d[a] += y[a];
      }
      const double r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
      double en, dedr2;
      ev.eval(e0 + qe[k], j, r2, en, dedr2);
      // a directed edge carries half of its pair: g / 2 = dE/d(r^2) d
      const double f = PAIRED ? 2.0 * share * dedr2 : dedr2;
      const double h[3] = {f * d[0], f * d[1], f * d[2]};
      en_sum += en;
      for (int a = 0; a < 3; ++a) {
        atomicAdd(&p.grad[3 * (int64_t)j + a], h[a]);
        gi[a] -= h[a];
      }
      if (kShifted || !(finite64(h[0]) && finite64(h[1]) && finite64(h[2]))) {
        any_dl = true;
        const double t0 = shift_double(s0), t1 = shift_double(s1), t2 = shift_double(s2);
        dl[0] += t0 * h[0];
        dl[1] += t1 * h[0];
        dl[2] += t1 * h[1];
        dl[3] += t2 * h[0];
        dl[4] += t2 * h[1];
        dl[5] += t2 * h[2];
      }
    }
  };
  int queued[2] = {0, 0};
  // the first 128 of a queue, then the rest moves to the front (at most 127 entries)
  auto drain = [&](auto shifted) {
    constexpr bool kShifted = decltype(shifted)::value;
    evaluate(shifted, 128, 4);
    __syncwarp();
    const int rest = queued[kShifted] - 128;
    int *qi = q_i[warp][kShifted], *qj = q_j[warp][kShifted], *qe = q_e[warp][kShifted];
    for (int k = lane; k < rest; k += 32) {
      qi[k] = qi[128 + k];
      qj[k] = qj[128 + k];
      qe[k] = qe[128 + k];
      if (kShifted) {
        q0[k] = q0[128 + k];
        q1[k] = q1[128 + k];
        q2[k] = q2[128 + k];
      }
    }
    queued[kShifted] = rest;
    __syncwarp();
  };
  const Const<false> plain;
  const Const<true> shifted;
  for (int64_t base = e0; base < e1; base += 128) {
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int64_t e = base + 32 * t + lane;
      int i = -1, j = -1;
      if (e < e1) {
        i = p.edges[2 * e];
        j = p.edges[2 * e + 1];
      }
      bool take = i >= 0 && i < p.n && j >= 0 && j < p.n;
      int s0 = 0, s1 = 0, s2 = 0;
      if (take && single) take = j >= i;
      if (take) {
        s0 = p.shifts[3 * e];
        s1 = p.shifts[3 * e + 1];
        s2 = p.shifts[3 * e + 2];
        const int si = p.system[i];
        take = si >= 0 && si < p.s;
        // a particle and its own images: the shift that is lexicographically positive
        if (single && i == j) take = take && (s0 > 0 || (s0 == 0 && (s1 > 0 || (s1 == 0 && s2 > 0))));
      }
      const int kind = (s0 | s1 | s2) != 0;
      const unsigned m1 = __ballot_sync(0xffffffffu, take && kind == 1);
      const unsigned m0 = __ballot_sync(0xffffffffu, take && kind == 0);
      if (take) {
        const int at = (kind ? queued[1] : queued[0]) + __popc((kind ? m1 : m0) & ((1u << lane) - 1u));
        q_i[warp][kind][at] = i;
        q_j[warp][kind][at] = j;
        q_e[warp][kind][at] = (int)(e - e0);
        if (kind) {
          q0[at] = s0;
          q1[at] = s1;
          q2[at] = s2;
        }
      }
      queued[0] += __popc(m0);
      queued[1] += __popc(m1);
    }
    __syncwarp();
    if (queued[0] >= 128) drain(plain);
    if (queued[1] >= 128) drain(shifted);
  }
  evaluate(plain, queued[0], (queued[0] + 31) / 32);
  evaluate(shifted, queued[1], (queued[1] + 31) / 32);
  flush_first();
  // one system in the whole warp (lanes without an edge have none): summed over the warp first
  const int top = __reduce_max_sync(0xffffffffu, sys);
  if (__all_sync(0xffffffffu, sys == top || sys < 0)) {
    if (top >= 0) {
      en_sum = warp_sum(en_sum);
      if (lane == 0) atomicAdd(&p.energy[top], share * en_sum);
      if (__any_sync(0xffffffffu, any_dl) && p.grad_tril)
        for (int a = 0; a < 6; ++a) {
          const double v = warp_sum(dl[a]);
          if (lane == 0) atomicAdd(&p.grad_tril[6 * (int64_t)top + a], v);
        }
    }
  } else {
    flush_system();
  }
}

// Edges per warp: 1024 once that still gives every SM 16 warps, down to 128 for short lists.
inline int64_t run_edges_per_warp(int64_t n_edges) {
  const int64_t warps = 16 * (int64_t)device_sm_count();
  const int64_t per = (n_edges / warps) / 128 * 128;
  return per < 128 ? 128 : (per > 1024 ? 1024 : per);
}
inline unsigned run_blocks(int64_t n_edges, int64_t per) {
  return (unsigned)((n_edges + per * kRunWarps - 1) / (per * kRunWarps));
}

}  // namespace kups
