// Bonded edge-set potentials: energy, dE/dx and dE/dtril over an edge list of
// order D (bonds 2, angles 3, dihedrals and inversions 4).
//
// Replaces the energies of src/kups/potential/classical/ harmonic.py:83-163
// (harmonic bond, harmonic angle), morse.py:142-171, cosine_angle.py:152-221,
// dihedral.py:214-273 and inversion.py:136-209 evaluated on the HyperGraph of an
// EdgeSetGraphConstructor (src/kups/potential/common/graph.py:289-361), with the
// gradient PotentialFromEnergy takes by jax.vjp with respect to
// PositionAndUnitCell (src/kups/potential/common/energy.py:264-355).
//
// One thread per edge (i_0, ..., i_{D-1}) with integer image shifts s_m:
//   v_m = x_{i_m} - x_{i_0} + s_m @ L  (Edges.difference_vectors,
//   src/kups/core/neighborlist.py:164-204), E_e(v_1 .. v_{D-1}) with the
//   parameter row of the edge's species tuple, g_m = dE_e/dv_m analytic, then
//   dE/dx_{i_m} += g_m, dE/dx_{i_0} -= sum_m g_m, dE/dL_ab += sum_m s_ma g_mb,
//   E_s += E_e for the system of i_0.  Difference vectors in float64; the
//   edge's arithmetic in float64, or in float32 with fp32 (this part issues
//   about 2 float64 FMA per cycle per SM, so the float64 angles, square roots
//   and trigonometry bound the float64 mode); per-system sums are warp sums (in
//   float in the float32 mode) added by one float64 atomic per warp, per-atom
//   gradients float64 atomics (atom 0's summed over the edge first), and the
//   image term s @ L is formed only for non-zero shifts.  The float32
//   mode takes angles as atan2 of cross and dot products and the cosine-angle and
//   inversion energies in factored forms, equal to the reference's in exact
//   arithmetic but without its cancellations, which float32 would amplify.
// Angle derivatives: d cos t / dv1 = v2 / (r1 r2) - cos t v1 / r1^2 (and 1 <-> 2).
// Dihedral: phi = atan2(|b2| b1 . (b2 x b3), (b1 x b2) . (b2 x b3)) with
// b1 = x_j - x_i, b2 = x_k - x_j, b3 = x_l - x_k, m = b1 x b2, n = b2 x b3; its
// position derivatives are the closed forms of Blondel and Karplus (J. Comput.
// Chem. 17, 1132, 1996): dphi/dx_i = -|b2| m / |m|^2, dphi/dx_l = |b2| n / |n|^2,
// dphi/dx_j = -(1 + p) dphi/dx_i + q dphi/dx_l, dphi/dx_k = p dphi/dx_i - (1 + q) dphi/dx_l,
// p = b1.b2 / |b2|^2, q = b3.b2 / |b2|^2.  Inversion: derivatives of
// sin w = (v1 . n / (|n| + eps)) / (|v1| + eps), n = v2 x v3, with the
// reference's 1e-10 regularisers kept.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "pair_runs.cuh"

namespace kups {
namespace {

constexpr double kEps = 1e-10;

template <typename R>
__device__ inline void cross3(const R a[3], const R b[3], R c[3]) {
  c[0] = a[1] * b[2] - a[2] * b[1];
  c[1] = a[2] * b[0] - a[0] * b[2];
  c[2] = a[0] * b[1] - a[1] * b[0];
}
template <typename R>
__device__ inline R dot3(const R a[3], const R b[3]) {
  return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}

template <int KIND>
struct Kind;
template <>
struct Kind<0> { static constexpr int order = 2, params = 2; };  // harmonic bond: x0, k
template <>
struct Kind<1> { static constexpr int order = 2, params = 3; };  // Morse: r0, D, alpha
template <>
struct Kind<2> { static constexpr int order = 3, params = 2; };  // harmonic angle: theta0 (deg), k
template <>
struct Kind<3> { static constexpr int order = 3, params = 3; };  // cosine angle: theta0 (rad), k, linear_tol
template <>
struct Kind<4> { static constexpr int order = 4, params = 3; };  // dihedral: V, n, phi0
template <>
struct Kind<5> { static constexpr int order = 4, params = 2; };  // inversion: omega0, k

// What an edge's parameter row contributes, formed once per row (block) instead of once per edge:
// the trigonometry of equilibrium angles and the force constants' factors.
//   0: x0, k   1: r0, D, alpha   2: theta0, k
//   3: linear (0 / 1), k, then (float64) k c0, k c1, k c2 of k (c0 + c1 c + c2 (2 c^2 - 1)),
//      (float32) cos theta0, 2 k c2, 4 k c2 of 2 k c2 (c - cos theta0)^2
//   4: V / 2, n, cos(n phi0), V / 2 cos(n phi0) n, n as a small integer (0: none)
//   5: (float64) ks c0, ks c1, ks c2; (float32) planar (0 / 1), k, omega0, 8 ks c2
constexpr int kRowConsts = 5;

template <int KIND, typename R>
__device__ inline void row_constants(const double *raw, R c[kRowConsts]) {
  R p[Kind<KIND>::params];
  for (int k = 0; k < Kind<KIND>::params; ++k) p[k] = (R)raw[k];
  for (int k = 0; k < kRowConsts; ++k) c[k] = k < Kind<KIND>::params ? p[k] : R(0.0);
  if (KIND == 3) {
    const R th0 = p[0], k = p[1];
    c[0] = fabs(th0 - R(M_PI)) < p[2] ? R(1.0) : R(0.0);
    const R s2 = sin(th0) * sin(th0), ct0 = cos(th0);
    const R c2 = R(1.0) / (R(4.0) * fmax(s2, R(1e-10)));
    if (sizeof(R) == 4) {
      c[2] = ct0;
      c[3] = R(2.0) * k * c2;
      c[4] = R(4.0) * k * c2;
    } else {
      c[2] = k * (c2 * (R(2.0) * ct0 * ct0 + R(1.0)));
      c[3] = k * (-R(4.0) * c2 * ct0);
      c[4] = k * c2;
    }
  } else if (KIND == 4) {
    const R V = p[0], per = p[1], cp = cos(per * p[2]);
    c[0] = R(0.5) * V;
    c[2] = cp;
    c[3] = R(0.5) * V * cp * per;
    c[4] = per == R(1.0) || per == R(2.0) || per == R(3.0) || per == R(4.0) || per == R(6.0) ? per : R(0.0);
  } else if (KIND == 5) {
    const R om0 = p[0], k = p[1];
    const bool planar = fabs(om0) < R(1e-6);
    const R s2 = sin(om0) * sin(om0);
    if (sizeof(R) == 4) {
      const R h0 = sin(R(0.5) * om0);
      const R c2 = R(1.0) / (R(4.0) * (s2 > R(1e-10) ? s2 : R(1.0)));
      const R ks = k / fmax(R(8.0) * c2 * h0 * h0 * h0 * h0, R(1e-10));
      c[0] = planar ? R(1.0) : R(0.0);
      c[1] = k;
      c[2] = om0;
      c[3] = R(8.0) * ks * c2;
    } else {
      const R cw0 = cos(om0);
      const R c2 = planar ? R(0.0) : R(1.0) / (R(4.0) * (s2 > R(1e-10) ? s2 : R(1.0)));
      const R c1 = planar ? -R(1.0) : -R(4.0) * c2 * cw0;
      const R c0 = planar ? R(1.0) : c2 * (R(2.0) * cw0 * cw0 + R(1.0));
      const R ks = planar ? k : k / fmax(c0 + c1 + c2, R(1e-10));
      c[0] = ks * c0;
      c[1] = ks * c1;
      c[2] = ks * c2;
    }
  }
}

// sqrt(x) and 1 / sqrt(x) of x > 0 from one reciprocal root (the root corrected to its last bit), a
// third of the float64 instructions of a root and a division.
__device__ inline double root64(double x, double &inv) {
  inv = rsqrt(x);
  const double r = x * inv;
  return fma(0.5 * inv, fma(-r, r, x), r);
}

// Tests of float64 values by their bits: a float64 comparison, minimum or conversion takes the
// float64 pipe like an addition.  A NaN of either sign is not zero.
__device__ inline bool nonzero64(double x) { return (__double_as_longlong(x) << 1) != 0; }
__device__ inline int exponent64(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }  // biased by 1023
__device__ inline double clamp_unit(double c) {  // c to [-1, 1] (a NaN to an end)
  const int hi = __double2hiint(c);
  return (hi & 0x7fffffff) >= 0x3ff00000 ? __hiloint2double(0x3ff00000 | (hi & (int)0x80000000), 0) : c;
}

// x / (sqrt(x) + eps) and 1 / (sqrt(x) + eps) from inv = 1 / sqrt(x), eps = 1e-10: eps / sqrt(x) = u
// is below 1e-7 from x = 2^-19 on, where 1 / (1 + u) = 1 - u + u^2 to 1e-21; a division below that.
__device__ inline double inverse_regularised(double root, double inv) {
  if (exponent64(root) < 1023 - 10) return 1.0 / (root + kEps);
  const double u = kEps * inv;
  return fma(inv, fma(u, u, -u), inv);
}

// Energy of one edge and g[m] = dE/dv_{m+1}; p the row's constants.
template <int KIND, typename R>
__device__ R edge_energy_grad(const R (*v)[3], const R *p, R (*g)[3]) {
  if (KIND == 0 || KIND == 1) {
    const R rr = dot3(v[0], v[0]);
    R r, inv = R(0.0);
    if (sizeof(R) == 8) r = rr > R(0.0) ? (R)root64((double)rr, (double &)inv) : R(0.0);
    else r = sqrt(rr);
    R e, dedr;
    if (KIND == 0) {
      e = (r - p[0]) * (r - p[0]) * p[1];
      dedr = R(2.0) * p[1] * (r - p[0]);
    } else {
      const R x = exp(-p[2] * (r - p[0]));
      e = p[1] * (R(1.0) - x) * (R(1.0) - x);
      dedr = R(2.0) * p[1] * (R(1.0) - x) * p[2] * x;
    }
    const R f = sizeof(R) == 8 ? dedr * inv : (r > R(0.0) ? dedr / r : R(0.0));
    for (int a = 0; a < 3; ++a) g[0][a] = f * v[0][a];
    return e;
  } else if ((KIND == 2 || KIND == 3) && sizeof(R) == 4) {
    // float32: theta = atan2(|v1 x v2|, v1 . v2) and the derivatives through
    // v1 x (v1 x v2), which keep float32 digits near 0 and pi where acos and
    // 1 / sqrt(1 - cos^2) lose them
    R cr[3], t1[3], t2[3];
    cross3(v[0], v[1], cr);
    cross3(v[0], cr, t1);
    cross3(v[1], cr, t2);
    const R sn = sqrt(dot3(cr, cr)), cs = dot3(v[0], v[1]);
    const R r1s = dot3(v[0], v[0]), r2s = dot3(v[1], v[1]);
    R e, f1, f2;  // g[0] = f1 * v1 x (v1 x v2), g[1] = f2 * v2 x (v1 x v2)
    if (KIND == 2) {
      const R th = atan2(sn, cs) * (R(180.0) / R(M_PI));
      e = (th - p[0]) * (th - p[0]) * p[1];
      const R f = sn > R(0.0) ? R(2.0) * p[1] * (th - p[0]) * (R(180.0) / R(M_PI)) / sn : R(0.0);
      f1 = f / r1s;
      f2 = -f / r2s;
    } else {
      // k (c0 + c1 c + c2 (2c^2 - 1)) = 2 k c2 (c - cos theta0)^2
      const R r12 = sqrt(r1s * r2s), c = cs / r12;
      const R cc = fmin(fmax(c, -R(1.0)), R(1.0));
      R dedc;
      if (p[0] != R(0.0)) {
        e = p[1] * (R(1.0) + cc);
        dedc = p[1];
      } else {
        const R d = cc - p[2];
        e = p[3] * d * d;
        dedc = p[4] * d;
      }
      if (fabs(c) > R(1.0)) dedc = R(0.0);
      f1 = -dedc / (r1s * r12);
      f2 = dedc / (r2s * r12);
    }
    for (int a = 0; a < 3; ++a) {
      g[0][a] = f1 * t1[a];
      g[1][a] = f2 * t2[a];
    }
    return e;
  } else if (KIND == 2 || KIND == 3) {
    // one reciprocal root per length and one of 1 - cos^2, which serves the gradient and, as
    // theta = pi / 2 - atan(cot theta), the angle (arccos takes two branches, both by most warps)
    const R i1 = rsqrt(dot3(v[0], v[0])), i2 = rsqrt(dot3(v[1], v[1])), i12 = i1 * i2;
    const R c = dot3(v[0], v[1]) * i12;
    R e, dedc;
    if (KIND == 2) {
      // the reference takes arccos of the unclipped cosine; clamping keeps
      // round-off above 1 from turning a straight angle into NaN
      const double cc = clamp_unit((double)c);
      double w = fma(-cc, cc, 1.0);
      if (exponent64(w) < 1023 - 100) w = 1e-30;
      const double is = rsqrt(w);
      const double th = (M_PI / 2 - atan(cc * is)) * (180.0 / M_PI), d = th - (double)p[0];
      e = (R)(d * d * (double)p[1]);
      dedc = (R)((-2.0 * 180.0 / M_PI) * (double)p[1] * d * is);
    } else {
      const double cc = clamp_unit((double)c);
      if (__double2hiint((double)p[0]) != 0) {
        e = (R)((double)p[1] * (1.0 + cc));
        dedc = p[1];
      } else {
        e = (R)((double)p[2] + (double)p[3] * cc + (double)p[4] * (2.0 * cc * cc - 1.0));
        dedc = (R)((double)p[3] + 4.0 * (double)p[4] * cc);
      }
      if (fabs(c) > R(1.0)) dedc = R(0.0);  // clipped: no gradient
    }
    const R f12 = dedc * i12, fc = -dedc * c, f1 = fc * i1 * i1, f2 = fc * i2 * i2;
    for (int a = 0; a < 3; ++a) {
      g[0][a] = f12 * v[1][a] + f1 * v[0][a];
      g[1][a] = f12 * v[0][a] + f2 * v[1][a];
    }
    return e;
  } else if (KIND == 4 && sizeof(R) == 8) {
    // tan phi = |b2|^2 (b1 . n) / (|b2| + eps) : m . n, since m x n = b2 (b1 . n) and the regularised
    // lengths of m and n are common positive factors
    R b2[3], b3[3], m[3], n[3];
    const R *b1 = v[0];
    for (int a = 0; a < 3; ++a) {
      b2[a] = v[1][a] - v[0][a];
      b3[a] = v[2][a] - v[1][a];
    }
    cross3(b1, b2, m);
    cross3(b2, b3, n);
    const R mm = dot3(m, m), nn = dot3(n, n), l2 = dot3(b2, b2);
    const bool bent = nonzero64((double)mm) && nonzero64((double)nn) && nonzero64((double)l2);
    double ilb = 0.0;
    const R lb = bent ? (R)root64((double)l2, ilb) : R(0.0);
    R y = R(0.0), x = R(0.0);
    if (bent) {
      y = l2 * dot3(b1, n) * (R)inverse_regularised((double)lb, ilb);
      x = dot3(m, n);
    }
    R cn, sn;  // cos and sin of n phi
    const R h2 = x * x + y * y;
    const int small_n = __double2hiint((double)p[4]), eh = exponent64((double)h2);
    if (small_n != 0 && eh > 100 && eh < 1946) {
      // integer n: the n-th power of (cos phi, sin phi), no inverse tangent and no sine
      const R ih = rsqrt(h2), c = x * ih, s = y * ih;
      const int per = small_n == 0x3ff00000   ? 1
                      : small_n == 0x40000000 ? 2
                      : small_n == 0x40080000 ? 3
                      : small_n == 0x40100000 ? 4
                                              : 6;
      cn = c;
      sn = s;
      if (per == 2 || per == 4 || per == 6) {
        cn = c * c - s * s;
        sn = R(2.0) * c * s;
      }
      const R c1 = cn, s1 = sn;
      if (per == 4) {
        cn = c1 * c1 - s1 * s1;
        sn = R(2.0) * c1 * s1;
      } else if (per == 3 || per == 6) {
        const R c2 = c1 * c1 - s1 * s1, s2 = R(2.0) * c1 * s1;
        cn = c2 * c1 - s2 * s1;
        sn = s2 * c1 + c2 * s1;
      }
    } else {
      sincos((double)(p[1] * atan2(y, x)), (double *)&sn, (double *)&cn);
    }
    const R e = p[0] * (R(1.0) - p[2] * cn);
    if (bent) {
      const R dedphi = p[3] * sn, il2 = (R)(ilb * ilb);
      const R pp = dot3(b1, b2) * il2, qq = dot3(b3, b2) * il2;
      const R f = dedphi * lb, fi = -f * (R)__drcp_rn((double)mm), fl = f * (R)__drcp_rn((double)nn);
      for (int a = 0; a < 3; ++a) {
        const R di = fi * m[a], dl = fl * n[a];
        g[0][a] = -(R(1.0) + pp) * di + qq * dl;
        g[1][a] = pp * di - (R(1.0) + qq) * dl;
        g[2][a] = dl;
      }
    } else {
      for (int k = 0; k < 3; ++k)
        for (int a = 0; a < 3; ++a) g[k][a] = R(0.0);
    }
    return e;
  } else if (KIND == 4) {
    R b1[3], b2[3], b3[3];
    for (int a = 0; a < 3; ++a) {
      b1[a] = v[0][a];
      b2[a] = v[1][a] - v[0][a];
      b3[a] = v[2][a] - v[1][a];
    }
    R m[3], n[3];
    cross3(b1, b2, m);
    cross3(b2, b3, n);
    const R mm = dot3(m, m), nn = dot3(n, n), lb = sqrt(dot3(b2, b2));
    const R lm = sqrt(mm), ln = sqrt(nn);
    R n1[3], n2[3], bn[3], x[3];
    for (int a = 0; a < 3; ++a) {
      n1[a] = m[a] / (lm + R(kEps));
      n2[a] = n[a] / (ln + R(kEps));
      bn[a] = b2[a] / (lb + R(kEps));
    }
    cross3(n1, n2, x);
    const R phi = atan2(dot3(x, bn), dot3(n1, n2));
    const R per = p[1];
    const R e = p[0] * (R(1.0) - p[2] * cos(per * phi));
    const R dedphi = p[3] * sin(per * phi);
    if (mm > R(0.0) && nn > R(0.0) && lb > R(0.0)) {
      const R pp = dot3(b1, b2) / (lb * lb), qq = dot3(b3, b2) / (lb * lb);
      for (int a = 0; a < 3; ++a) {
        const R di = -lb / mm * m[a], dl = lb / nn * n[a];
        g[0][a] = dedphi * (-(R(1.0) + pp) * di + qq * dl);
        g[1][a] = dedphi * (pp * di - (R(1.0) + qq) * dl);
        g[2][a] = dedphi * dl;
      }
    } else {
      for (int k = 0; k < 3; ++k)
        for (int a = 0; a < 3; ++a) g[k][a] = R(0.0);
    }
    return e;
  } else if (sizeof(R) == 4) {
    // float32 inversion: w = atan2(v1 . n, |v1 x n|), n = v2 x v3, and the
    // energy in the cancellation-free form
    //   ks (c0 + c1 cos w + c2 cos 2w) = 8 ks c2 X^2, X = sin((w + w0)/2) sin((w - w0)/2),
    //   c0 + c1 + c2 = 8 c2 sin^4(w0 / 2)
    // dw/dv1 = (|u1| n - (v1 . n) n x u1 / |u1|) / (|n| |v1|)^2,
    // dw/dn = (|u1| v1 + (v1 . n) v1 x u1 / |u1|) / (|n| |v1|)^2, u1 = v1 x n
    R n[3], u[3], nu[3], vu[3];
    cross3(v[1], v[2], n);
    cross3(v[0], n, u);
    cross3(n, u, nu);
    cross3(v[0], u, vu);
    const R nn = dot3(n, n), la2 = dot3(v[0], v[0]), an = dot3(v[0], n), lu = sqrt(dot3(u, u));
    const R w = atan2(an, lu);
    const R om0 = p[2], k = p[1];
    const R den = nn * la2;
    const R sw = den > R(0.0) ? an * rsqrt(den) : R(0.0);
    R e, dedw;
    if (p[0] != R(0.0)) {
      const R h = sin(R(0.5) * w);
      e = R(2.0) * k * h * h;  // k (1 - cos w)
      dedw = k * sw;
    } else {
      const R X = sin(R(0.5) * (w + om0)) * sin(R(0.5) * (w - om0));
      e = p[3] * X * X;
      dedw = p[3] * X * sw;
    }
    const R f = den > R(0.0) ? dedw / den : R(0.0);
    const R q = lu > R(0.0) ? an / lu : R(0.0);
    R G[3], t[3];
    for (int a = 0; a < 3; ++a) {
      g[0][a] = f * (lu * n[a] - q * nu[a]);
      G[a] = f * (lu * v[0][a] + q * vu[a]);
    }
    cross3(v[2], G, t);
    for (int a = 0; a < 3; ++a) g[1][a] = t[a];
    cross3(G, v[1], t);
    for (int a = 0; a < 3; ++a) g[2][a] = t[a];
    return e;
  } else {
    // w = asin s lies in [-pi/2, pi/2]: cos w = sqrt(1 - s^2), cos 2w = 1 - 2 s^2, sin 2w = 2 s cos w
    R n[3];
    cross3(v[1], v[2], n);
    const R nn = dot3(n, n), aa = dot3(v[0], v[0]), an = dot3(v[0], n);
    double iln = 1.0, ila = 1.0;
    const R ln = nonzero64((double)nn) ? (R)root64((double)nn, iln) : R(0.0);
    const R la = nonzero64((double)aa) ? (R)root64((double)aa, ila) : R(0.0);
    const R inv_la = (R)inverse_regularised((double)la, ila), inv_ln = (R)inverse_regularised((double)ln, iln);
    const double s_raw = (double)(an * inv_ln * inv_la), s = clamp_unit(s_raw);
    const double w2 = fma(-s, s, 1.0), icw = rsqrt(exponent64(w2) < 1023 - 100 ? 1e-30 : w2), cw = w2 * icw;
    const R e = (R)((double)p[0] + (double)p[1] * cw + (double)p[2] * (w2 - s * s));
    const R deds = fabs(s_raw) <= 1.0 ? (R)(-s * ((double)p[1] + 4.0 * (double)p[2] * cw) * icw) : R(0.0);
    // ds/dv1 and ds/dn; dn/dv2 (x) and dn/dv3 (x) through the cross product
    const R f = deds * inv_la * inv_ln, f0 = -f * an * inv_la * (R)ila, f1 = -f * an * inv_ln * (R)iln;
    R wv[3], t[3];
    for (int a = 0; a < 3; ++a) {
      g[0][a] = f * n[a] + f0 * v[0][a];
      wv[a] = f * v[0][a] + f1 * n[a];
    }
    cross3(v[2], wv, t);
    for (int a = 0; a < 3; ++a) g[1][a] = t[a];
    cross3(wv, v[1], t);
    for (int a = 0; a < 3; ++a) g[2][a] = t[a];
    return e;
  }
}

// Running per-system sums of one lane (float64 mode) or one warp (float32 mode: lane 0 holds the
// float64 total of the warps' float sums of 32 edges), added to the caller's arrays when the system
// changes and at the end.
struct SystemSums {
  int sys;
  double en, dl[6];

  __device__ void flush(double *energy, double *grad_tril) {
    if (sys >= 0) {
      atomicAdd(&energy[sys], en);
      if (grad_tril != nullptr)
        for (int k = 0; k < 6; ++k)
          if (dl[k] != 0.0) atomicAdd(&grad_tril[6 * (int64_t)sys + k], dl[k]);
    }
    clear(-1);
  }
  __device__ void clear(int s) {
    sys = s;
    en = 0.0;
    for (int k = 0; k < 6; ++k) dl[k] = 0.0;
  }
};

__device__ inline bool is_finite(double v) { return finite64(v); }
__device__ inline bool is_finite(float v) { return (__float_as_int(v) & 0x7f800000) != 0x7f800000; }

template <typename R>
__device__ inline R shift_real(int s);
template <>
__device__ inline double shift_real<double>(int s) { return shift_double(s); }
template <>
__device__ inline float shift_real<float>(int s) { return (float)s; }

constexpr int kBondedThreads = 128, kRowTable = 256;  // parameter rows kept in shared memory

struct BondedArgs {
  const double *pos;
  const int32_t *system, *species;
  int64_t n;
  const double *tril;
  int32_t n_sys;
  const int32_t *edges, *shifts;
  int64_t n_edges;
  const double *params;
  int32_t nsp;
  int n_rows, per;
  double *energy, *grad, *grad_tril;
  kups_status *status;
};

// Atoms, parameter row and system of edge e; false (status recorded) for an index, species or system
// out of range.
template <int D>
__device__ inline bool bonded_atoms(const BondedArgs &a, int64_t e, int idx[D], int64_t &row, int &sys) {
  bool ok = true;
  for (int d = 0; d < D; ++d) {
    idx[d] = a.edges[(int64_t)D * e + d];
    ok &= idx[d] >= 0 && idx[d] < a.n;
  }
  row = 0;
  if (ok)
    for (int d = 0; d < D; ++d) {
      const int k = a.species[idx[d]];
      ok &= k >= 0 && k < a.nsp;
      row = row * a.nsp + k;
    }
  sys = ok ? a.system[idx[0]] : -1;
  if (sys < 0 || sys >= a.n_sys) {
    status_error(a.status, KUPS_ERR_INVALID, e);
    sys = -1;
    return false;
  }
  return true;
}

template <int D>
__device__ inline bool bonded_shifts(const BondedArgs &a, int64_t e, int sh[D - 1][3]) {
  int any = 0;
  for (int m = 0; m < D - 1; ++m)
    for (int k = 0; k < 3; ++k) {
      sh[m][k] = a.shifts[((int64_t)(D - 1) * e + m) * 3 + k];
      any |= sh[m][k];
    }
  return any != 0;
}

// Energy of edge e with its gradient added to the atoms; `shifted`: some sh is not zero, and dl
// receives sum_m s_ma g_mb (also for a non-finite gradient, which reaches dE/dtril through a zero
// shift).  Returns whether dl was set.
template <int KIND, typename R>
__device__ inline bool bonded_edge(const BondedArgs &a, const R (*table)[kRowConsts], int64_t e, const int *idx,
                                   int64_t row, int sys, const int (*sh)[3], bool shifted, R &en, R dl[6]) {
  constexpr int D = Kind<KIND>::order, P = Kind<KIND>::params;
  // difference vectors in float64 (positions are float64), then the edge's arithmetic in R
  R v[D - 1][3], g[D - 1][3], own[kRowConsts];
  const double *x0 = a.pos + 3 * (int64_t)idx[0];
  const double o[3] = {x0[0], x0[1], x0[2]};
  Tril64 L;
  if (shifted) L = load_tril64(a.tril + 6 * (int64_t)sys);
  for (int m = 0; m < D - 1; ++m) {
    const double *xm = a.pos + 3 * (int64_t)idx[m + 1];
    double d[3] = {xm[0] - o[0], xm[1] - o[1], xm[2] - o[2]};
    if (shifted && (sh[m][0] | sh[m][1] | sh[m][2])) {
      double sL[3];
      shift_vector(sh[m], L, sL);
      for (int k = 0; k < 3; ++k) d[k] += sL[k];
    }
    for (int k = 0; k < 3; ++k) v[m][k] = (R)d[k];
  }
  const R *c = table[a.n_rows > 0 ? row : 0];
  if (a.n_rows == 0) {  // more rows than the table holds
    row_constants<KIND, R>(a.params + row * P, own);
    c = own;
  }
  en = edge_energy_grad<KIND, R>(v, c, g);
  bool finite = is_finite(en);
  for (int m = 0; m < D - 1; ++m)
    for (int k = 0; k < 3; ++k) finite &= is_finite(g[m][k]);
  if (!finite) status_error(a.status, KUPS_ERR_NONFINITE, e);
  R g0[3] = {R(0.0), R(0.0), R(0.0)};  // atom 0 takes -sum_m g_m in one atomic per axis
  for (int m = 0; m < D - 1; ++m)
    for (int k = 0; k < 3; ++k) {
      atomicAdd(&a.grad[3 * (int64_t)idx[m + 1] + k], (double)g[m][k]);
      g0[k] -= g[m][k];
    }
  for (int k = 0; k < 3; ++k) atomicAdd(&a.grad[3 * (int64_t)idx[0] + k], (double)g0[k]);
  if (!shifted && finite) return false;
  for (int m = 0; m < D - 1; ++m) {
    const R t[3] = {shift_real<R>(sh[m][0]), shift_real<R>(sh[m][1]), shift_real<R>(sh[m][2])};
    dl[0] += t[0] * g[m][0];
    dl[1] += t[1] * g[m][0];
    dl[2] += t[1] * g[m][1];
    dl[3] += t[2] * g[m][0];
    dl[4] += t[2] * g[m][1];
    dl[5] += t[2] * g[m][2];
  }
  return true;
}

// A warp takes `per` groups of 32 consecutive edges.  Float64 mode is bound by the float64 pipe (2
// operations per clock per SM): edges with an image shift are put aside and evaluated 32 at a time,
// so that the shift vectors and dE/dtril (27 operations per difference vector) cost nothing for the
// others, and the per-system sums leave as one warp sum at the end (one for every 32 edges was 35 of a
// bond's 111 float64 instructions).  Float32 mode sums each 32 edges in float, as its callers' results
// have always been rounded, and adds those totals in float64.
// 5.2e5 edges of each kind, float64: 66 us (bonds), 187 (angles), 228 (dihedrals), 208 (inversions);
// with a division or root for every quotient, trigonometry of the row's constants per edge and the
// angle taken through acos / atan2 / asin and back: 99, 281, 443 and 438 us.
template <int KIND, typename R>
__global__ void __launch_bounds__(kBondedThreads) bonded_kernel(BondedArgs a) {
  constexpr int D = Kind<KIND>::order, P = Kind<KIND>::params, kWarps = kBondedThreads / 32;
  __shared__ R table[kRowTable][kRowConsts];
  __shared__ int aside[kWarps][64];  // shifted edges of a warp, from its first
  for (int r = threadIdx.x; r < a.n_rows; r += kBondedThreads) row_constants<KIND, R>(a.params + (int64_t)r * P, table[r]);
  __syncthreads();
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * kBondedThreads + threadIdx.x) >> 5;
  const int64_t first = warp * a.per * 32;
  SystemSums sum;
  sum.clear(-1);
  if constexpr (sizeof(R) == 8) {
    int *queue = aside[threadIdx.x >> 5];
    int queued = 0;
    auto add = [&](int sys, R en, bool has_dl, const R *dl) {
      if (sys != sum.sys) {
        sum.flush(a.energy, a.grad_tril);
        sum.sys = sys;
      }
      sum.en += (double)en;
      if (has_dl)
        for (int k = 0; k < 6; ++k) sum.dl[k] += (double)dl[k];
    };
    auto shifted_edges = [&](int count) {  // the first `count` put aside, a lane each
      if (lane < count) {
        const int64_t e = first + queue[lane];
        int idx[D], sh[D - 1][3], sys;
        int64_t row;
        bonded_atoms<D>(a, e, idx, row, sys);
        bonded_shifts<D>(a, e, sh);
        R en, dl[6] = {R(0.0), R(0.0), R(0.0), R(0.0), R(0.0), R(0.0)};
        bonded_edge<KIND, R>(a, table, e, idx, row, sys, sh, true, en, dl);
        add(sys, en, true, dl);
      }
    };
    for (int t = 0; t < a.per; ++t) {
      const int64_t e = first + 32 * t + lane;
      int idx[D], sh[D - 1][3], sys = -1;
      int64_t row;
      const bool ok = e < a.n_edges && bonded_atoms<D>(a, e, idx, row, sys);
      const bool shifted = ok && bonded_shifts<D>(a, e, sh);
      const unsigned m = __ballot_sync(full, shifted);
      if (shifted) queue[queued + __popc(m & ((1u << lane) - 1u))] = 32 * t + lane;
      queued += __popc(m);
      if (ok && !shifted) {
        R en, dl[6] = {R(0.0), R(0.0), R(0.0), R(0.0), R(0.0), R(0.0)};
        const bool has_dl = bonded_edge<KIND, R>(a, table, e, idx, row, sys, sh, false, en, dl);
        add(sys, en, has_dl, dl);
      }
      __syncwarp();
      if (queued >= 32) {
        shifted_edges(32);
        queued -= 32;
        const int keep = lane < queued ? queue[32 + lane] : 0;
        __syncwarp();
        if (lane < queued) queue[lane] = keep;
        __syncwarp();
      }
    }
    shifted_edges(queued);
    __syncwarp();
    const int s0 = __reduce_max_sync(full, sum.sys);
    if (__all_sync(full, sum.sys == s0 || sum.sys < 0)) {
      sum.en = warp_sum(sum.en);
      bool some = false;
      for (int k = 0; k < 6; ++k) some |= sum.dl[k] != 0.0;
      if (__any_sync(full, some))
        for (int k = 0; k < 6; ++k) sum.dl[k] = warp_sum(sum.dl[k]);
      sum.sys = lane == 0 ? s0 : -1;
    }
    sum.flush(a.energy, a.grad_tril);
  } else {
    for (int t = 0; t < a.per; ++t) {
      const int64_t e = first + 32 * t + lane;
      if (e - lane >= a.n_edges) break;  // the same for the whole warp
      int idx[D], sh[D - 1][3], sys = -1;
      int64_t row;
      bool has_dl = false;
      R en = R(0.0), dl[6] = {R(0.0), R(0.0), R(0.0), R(0.0), R(0.0), R(0.0)};
      if (e < a.n_edges && bonded_atoms<D>(a, e, idx, row, sys)) {
        const bool shifted = bonded_shifts<D>(a, e, sh);
        has_dl = bonded_edge<KIND, R>(a, table, e, idx, row, sys, sh, shifted, en, dl);
      }
      // 32 edges of one system: summed in float over the warp, else edge by edge
      const int s0 = __shfl_sync(full, sys, 0);
      const bool any_dl = __any_sync(full, has_dl);
      if (__all_sync(full, sys == s0)) {
        if (s0 != sum.sys) {
          if (lane == 0) sum.flush(a.energy, a.grad_tril);
          sum.clear(s0);
        }
        sum.en += (double)warp_sum(en);
        if (any_dl)
          for (int k = 0; k < 6; ++k) sum.dl[k] += (double)warp_sum(dl[k]);
      } else if (sys >= 0) {
        atomicAdd(&a.energy[sys], (double)en);
        if (a.grad_tril != nullptr && has_dl)
          for (int k = 0; k < 6; ++k) atomicAdd(&a.grad_tril[6 * (int64_t)sys + k], (double)dl[k]);
      }
    }
    if (lane == 0) sum.flush(a.energy, a.grad_tril);
  }
}

// slot[i] = k for the k-th changed particle, -1 for every other particle (slot preset to -1).
__global__ void changed_slot_kernel(const int32_t *changed, int64_t n_changed, int64_t n, int32_t *slot,
                                    kups_status *status) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n_changed) return;
  const int32_t i = changed[k];
  if (i < 0 || i >= n) {
    status_error(status, KUPS_ERR_INVALID, k);
    return;
  }
  slot[i] = (int32_t)k;
}

// delta[s] += E_e(new) - E_e(old) over the edges with at least one changed atom: the
// old graph (weight -1) and new graph (weight +1) of LocalGraphSumComposer
// (src/kups/potential/common/graph.py:412-450) restricted, as EdgeSetGraphConstructor's
// probe path restricts them (:336-361), to the affected edges.  A changed atom d takes
// new_pos[slot[d]]; its wrap image n_d (new position = unwrapped - n_d @ L) moves the
// edge's shifts to s_m + n_{m+1} - n_0, which keeps each difference vector on the same
// image (the edge data the reference's probe updates).
// E_e(new) - E_e(old) of edge e whose atoms idx[] have slots sl[] (-1: not moved);
// returns the edge's system, or -1 (status recorded) for an invalid species or system.
template <int KIND, typename R>
__device__ int edge_delta(int64_t e, const int *idx, const int *sl, const double *pos, const int32_t *system,
                          const int32_t *species, const double *tril, int32_t n_sys, const int32_t *shifts,
                          const double *params, int32_t nsp, const double *new_pos, const int32_t *new_image,
                          double &de, kups_status *status) {
  constexpr int D = Kind<KIND>::order, P = Kind<KIND>::params;
  bool ok = true;
  int64_t row = 0;
  for (int d = 0; d < D; ++d) {
    const int t = species[idx[d]];
    ok &= t >= 0 && t < nsp;
    row = row * nsp + t;
  }
  const int s0 = system[idx[0]];
  if (!ok || s0 < 0 || s0 >= n_sys) {
    status_error(status, KUPS_ERR_INVALID, e);
    return -1;
  }
  const Tril64 L = load_tril64(tril + 6 * (int64_t)s0);
  double x_old[D][3], x_new[D][3], img[D][3];
  for (int d = 0; d < D; ++d)
    for (int a = 0; a < 3; ++a) {
      x_old[d][a] = pos[3 * (int64_t)idx[d] + a];
      x_new[d][a] = sl[d] >= 0 ? new_pos[3 * (int64_t)sl[d] + a] : x_old[d][a];
      img[d][a] = (sl[d] >= 0 && new_image) ? (double)new_image[3 * (int64_t)sl[d] + a] : 0.0;
    }
  R v_old[D - 1][3], v_new[D - 1][3], g[D - 1][3], pr[kRowConsts];
  for (int m = 0; m < D - 1; ++m) {
    double sh[3], sh_new[3], sL[3], sL_new[3];
    for (int a = 0; a < 3; ++a) {
      sh[a] = shifts[((int64_t)(D - 1) * e + m) * 3 + a];
      sh_new[a] = sh[a] + img[m + 1][a] - img[0][a];
    }
    row_times_tril64(sh, L, sL);
    row_times_tril64(sh_new, L, sL_new);
    for (int a = 0; a < 3; ++a) {
      v_old[m][a] = (R)(x_old[m + 1][a] - x_old[0][a] + sL[a]);
      v_new[m][a] = (R)(x_new[m + 1][a] - x_new[0][a] + sL_new[a]);
    }
  }
  row_constants<KIND, R>(params + row * P, pr);
  const double e_new = (double)edge_energy_grad<KIND, R>(v_new, pr, g);
  const double e_old = (double)edge_energy_grad<KIND, R>(v_old, pr, g);
  de = e_new - e_old;
  if (!isfinite(de)) status_error(status, KUPS_ERR_NONFINITE, e);
  return s0;
}

// delta[s] += E_e(new) - E_e(old) over the edges with at least one changed atom: the
// old graph (weight -1) and new graph (weight +1) of LocalGraphSumComposer
// (src/kups/potential/common/graph.py:412-450) restricted, as EdgeSetGraphConstructor's
// probe path restricts them (:336-361), to the affected edges.  A changed atom d takes
// new_pos[slot[d]]; its wrap image n_d (new position = unwrapped - n_d @ L) moves the
// edge's shifts to s_m + n_{m+1} - n_0, which keeps each difference vector on the same
// image (the edge data the reference's probe updates).  This form scans every edge.
template <int KIND, typename R>
__global__ void bonded_delta_kernel(const double *pos, const int32_t *system, const int32_t *species, int64_t n,
                                    const double *tril, int32_t n_sys, const int32_t *edges, const int32_t *shifts,
                                    int64_t n_edges, const double *params, int32_t nsp, const int32_t *slot,
                                    const double *new_pos, const int32_t *new_image, double *delta,
                                    kups_status *status) {
  constexpr int D = Kind<KIND>::order;
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int sys = -1;
  double de = 0.0;
  if (e < n_edges) {
    int idx[D], sl[D];
    bool ok = true, touched = false;
    for (int d = 0; d < D; ++d) {
      idx[d] = edges[(int64_t)D * e + d];
      ok &= idx[d] >= 0 && idx[d] < n;
    }
    if (ok)
      for (int d = 0; d < D; ++d) {
        sl[d] = slot[idx[d]];
        touched |= sl[d] >= 0;
      }
    if (!ok)
      status_error(status, KUPS_ERR_INVALID, e);
    else if (touched)
      sys = edge_delta<KIND, R>(e, idx, sl, pos, system, species, tril, n_sys, shifts, params, nsp, new_pos,
                                new_image, de, status);
  }
  add_system(delta, 1, 0, sys, de);
}

// The same sum through the atom -> edge incidence lists: changed atom k's edges are
// split over kDeltaSplit consecutive threads (edge j to thread j mod kDeltaSplit), so
// that a batch of a few thousand moved atoms spreads over every SM; an edge with
// several changed atoms belongs to the one earliest in `changed`.
constexpr int kDeltaSplit = 4;
template <int KIND, typename R>
__global__ void bonded_delta_incident_kernel(const double *pos, const int32_t *system, const int32_t *species,
                                             int64_t n, const double *tril, int32_t n_sys, const int32_t *edges,
                                             const int32_t *shifts, int64_t n_edges, const double *params,
                                             int32_t nsp, const int32_t *changed, int64_t n_changed,
                                             const int64_t *inc_offsets, const int32_t *inc_edges,
                                             const int32_t *slot, const double *new_pos, const int32_t *new_image,
                                             double *delta, kups_status *status) {
  constexpr int D = Kind<KIND>::order;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t k = t / kDeltaSplit;
  if (k >= n_changed) return;
  const int32_t i = changed[k];
  if (i < 0 || i >= n) return;  // recorded by changed_slot_kernel
  for (int64_t q = inc_offsets[i] + t % kDeltaSplit; q < inc_offsets[i + 1]; q += kDeltaSplit) {
    const int64_t e = inc_edges[q];
    if (e < 0 || e >= n_edges) {
      status_error(status, KUPS_ERR_INVALID, e);
      continue;
    }
    int idx[D], sl[D];
    bool ok = true, mine = true;
    for (int d = 0; d < D; ++d) {
      idx[d] = edges[(int64_t)D * e + d];
      ok &= idx[d] >= 0 && idx[d] < n;
    }
    if (!ok) {
      status_error(status, KUPS_ERR_INVALID, e);
      continue;
    }
    for (int d = 0; d < D; ++d) {
      sl[d] = slot[idx[d]];
      mine &= sl[d] < 0 || sl[d] >= k;
    }
    if (!mine) continue;
    double de = 0.0;
    const int s = edge_delta<KIND, R>(e, idx, sl, pos, system, species, tril, n_sys, shifts, params, nsp, new_pos,
                                      new_image, de, status);
    if (s >= 0) atomicAdd(&delta[s], de);
  }
}

template <int KIND, typename R>
cudaError_t launch_bonded(const double *pos, const int32_t *system, const int32_t *species, int64_t n,
                          const double *tril, int32_t s, const int32_t *edges, const int32_t *shifts,
                          int64_t n_edges, const double *params, int32_t nsp, double *energy, double *grad,
                          double *grad_tril, kups_status *status, cudaStream_t stream) {
  int64_t rows = 1;
  for (int d = 0; d < Kind<KIND>::order && rows <= kRowTable; ++d) rows *= nsp;
  // up to eight edges per thread while every SM still gets four blocks
  const int64_t wave = 4 * (int64_t)device_sm_count() * kBondedThreads;
  const int per = (int)std::min<int64_t>(8, std::max<int64_t>(1, n_edges / wave));
  const int64_t block = (int64_t)kBondedThreads * per;
  const BondedArgs args{pos,    system, species, n,   tril,   s,    edges,     shifts, n_edges,
                        params, nsp,    rows <= kRowTable ? (int)rows : 0, per, energy, grad, grad_tril, status};
  bonded_kernel<KIND, R><<<(unsigned)((n_edges + block - 1) / block), kBondedThreads, 0, stream>>>(args);
  return cudaGetLastError();
}

}  // namespace
}  // namespace kups

using namespace kups;

extern "C" int32_t kups_bonded_order(int32_t kind) {
  switch (kind) {
    case 0: return Kind<0>::order;
    case 1: return Kind<1>::order;
    case 2: return Kind<2>::order;
    case 3: return Kind<3>::order;
    case 4: return Kind<4>::order;
    case 5: return Kind<5>::order;
    default: return -1;
  }
}

extern "C" int32_t kups_bonded_param_count(int32_t kind) {
  switch (kind) {
    case 0: return Kind<0>::params;
    case 1: return Kind<1>::params;
    case 2: return Kind<2>::params;
    case 3: return Kind<3>::params;
    case 4: return Kind<4>::params;
    case 5: return Kind<5>::params;
    default: return -1;
  }
}

extern "C" int32_t kups_bonded_edges(int32_t kind, const double *positions, const int32_t *system,
                                     const int32_t *species, int64_t n_particles, const double *tril,
                                     int32_t n_systems, const int32_t *edges, const int32_t *shifts, int64_t n_edges,
                                     const double *params, int32_t n_species, double *energy, double *grad,
                                     double *grad_tril, int32_t fp32, kups_status *status, void *stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (kind < 0 || kind > 5 || n_particles < 0 || n_systems < 0 || n_edges < 0 || n_species <= 0 ||
      n_species > 1024)
    return KUPS_ERR_INVALID;
  if (n_edges == 0) return KUPS_OK;
  if (positions == nullptr || system == nullptr || species == nullptr || tril == nullptr || edges == nullptr ||
      shifts == nullptr || params == nullptr || energy == nullptr || grad == nullptr || status == nullptr)
    return KUPS_ERR_INVALID;
  cudaError_t err;
  switch (kind * 2 + (fp32 ? 1 : 0)) {
#define KUPS_BONDED_CASE(K, R)                                                                                   \
  case 2 * K + (sizeof(R) == 4 ? 1 : 0):                                                                         \
    err = launch_bonded<K, R>(positions, system, species, n_particles, tril, n_systems, edges, shifts, n_edges,  \
                              params, n_species, energy, grad, grad_tril, status, stream);                       \
    break;
    KUPS_BONDED_CASE(0, double)
    KUPS_BONDED_CASE(0, float)
    KUPS_BONDED_CASE(1, double)
    KUPS_BONDED_CASE(1, float)
    KUPS_BONDED_CASE(2, double)
    KUPS_BONDED_CASE(2, float)
    KUPS_BONDED_CASE(3, double)
    KUPS_BONDED_CASE(3, float)
    KUPS_BONDED_CASE(4, double)
    KUPS_BONDED_CASE(4, float)
    KUPS_BONDED_CASE(5, double)
    KUPS_BONDED_CASE(5, float)
#undef KUPS_BONDED_CASE
    default:
      return KUPS_ERR_INVALID;
  }
  return err == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}

extern "C" size_t kups_bonded_delta_workspace_bytes(int64_t n_particles) {
  return n_particles < 0 ? 0 : sizeof(int32_t) * (size_t)n_particles + 256;
}

extern "C" int32_t kups_bonded_delta(int32_t kind, const double *positions, const int32_t *system,
                                     const int32_t *species, int64_t n_particles, const double *tril,
                                     int32_t n_systems, const int32_t *edges, const int32_t *shifts, int64_t n_edges,
                                     const double *params, int32_t n_species, const int64_t *incidence_offsets,
                                     const int32_t *incidence_edges, const int32_t *changed,
                                     const double *new_positions, const int32_t *new_image, int64_t n_changed,
                                     double *delta, int32_t fp32, void *workspace, size_t workspace_bytes,
                                     kups_status *status, void *stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  // slots hold positions in `changed` as int32
  if (kind < 0 || kind > 5 || n_particles < 0 || n_systems < 0 || n_edges < 0 || n_changed < 0 ||
      n_changed >= (int64_t)INT32_MAX || n_species <= 0 || n_species > 1024)
    return KUPS_ERR_INVALID;
  if (n_edges == 0 || n_changed == 0) return KUPS_OK;
  if (positions == nullptr || system == nullptr || species == nullptr || tril == nullptr || edges == nullptr ||
      shifts == nullptr || params == nullptr || changed == nullptr || new_positions == nullptr ||
      delta == nullptr || status == nullptr || workspace == nullptr)
    return KUPS_ERR_INVALID;
  if (n_particles >= (int64_t)INT32_MAX || workspace_bytes < kups_bonded_delta_workspace_bytes(n_particles))
    return KUPS_ERR_INVALID;
  int32_t *slot = (int32_t *)(((uintptr_t)workspace + 255) & ~uintptr_t(255));
  KUPS_CUDA_TRY(cudaMemsetAsync(slot, 0xff, sizeof(int32_t) * (size_t)n_particles, stream));  // -1
  changed_slot_kernel<<<(unsigned)((n_changed + 127) / 128), 128, 0, stream>>>(changed, n_changed, n_particles, slot,
                                                                              status);
  if ((incidence_offsets == nullptr) != (incidence_edges == nullptr)) return KUPS_ERR_INVALID;
  const bool incident = incidence_offsets != nullptr;
  const unsigned grid = (unsigned)((n_edges + 127) / 128);
  const unsigned grid_k = (unsigned)((n_changed * kDeltaSplit + 63) / 64);
  switch (kind * 2 + (fp32 ? 1 : 0)) {
#define KUPS_DELTA_CASE(K, R)                                                                                     \
  case 2 * K + (sizeof(R) == 4 ? 1 : 0):                                                                          \
    if (incident)                                                                                                 \
      bonded_delta_incident_kernel<K, R><<<grid_k, 64, 0, stream>>>(                                              \
          positions, system, species, n_particles, tril, n_systems, edges, shifts, n_edges, params, n_species,    \
          changed, n_changed, incidence_offsets, incidence_edges, slot, new_positions, new_image, delta, status); \
    else                                                                                                          \
      bonded_delta_kernel<K, R><<<grid, 128, 0, stream>>>(positions, system, species, n_particles, tril,          \
                                                          n_systems, edges, shifts, n_edges, params, n_species,   \
                                                          slot, new_positions, new_image, delta, status);         \
    break;
    KUPS_DELTA_CASE(0, double)
    KUPS_DELTA_CASE(0, float)
    KUPS_DELTA_CASE(1, double)
    KUPS_DELTA_CASE(1, float)
    KUPS_DELTA_CASE(2, double)
    KUPS_DELTA_CASE(2, float)
    KUPS_DELTA_CASE(3, double)
    KUPS_DELTA_CASE(3, float)
    KUPS_DELTA_CASE(4, double)
    KUPS_DELTA_CASE(4, float)
    KUPS_DELTA_CASE(5, double)
    KUPS_DELTA_CASE(5, float)
#undef KUPS_DELTA_CASE
    default:
      return KUPS_ERR_INVALID;
  }
  return cudaGetLastError() == cudaSuccess ? KUPS_OK : KUPS_ERR_CUDA;
}
