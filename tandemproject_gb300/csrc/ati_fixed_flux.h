// ati_fixed_flux.h — the FP64 fast path's fluxes at one point in 64-bit fixed point (see ati_fixed.h for why).
//
// Every operand is an integer just below 2^60 times its own power of two, whatever the others' sizes: along a stretched
// grid the metrics of two directions differ by a thousand, and a small velocity component has its own accuracy.  Sums of
// products run in integers (three 32 x 32 + 64 bit multiply-adds a product, the lowest partial product left out), each
// product aligned to the sum's largest.  A sum's error is some 2^-57 of its largest term, where FP64 rounds each operation
// at 2^-53.  Measured against extended precision in units of the terms that make a component up, over metric ratios of 1
// to 10^6, velocity components 1 to 10^-30 of the largest, derivatives of all sizes: 0.49 to 0.80 of the FP64 arithmetic's
// error, inviscid momentum 0.84 to 1.001 (correctly rounded there but for 2^-57).
//
// As the FP64 kernels do (src/Main3D.f90:631-766): contravariant velocities S_n = M_n . (u + u_inf), then along n
//   rho S,  (rho u_m) S + M . (p delta - tau)_m,  (rhoE + p) S + M . w,   w = u . (-tau) - r2 grad T - p u_inf
#pragma once
#include "ati_fixed_num.h"

namespace ati {

namespace fxf {

// a sum of products of fixed-point values, in units of 2^64 of the product's; value(K): in units of 2^(64-K)
struct Dot {
  i64 hi, mid;
  ATI_HD Dot() : hi(0), mid(0) {}
  ATI_HD void add(Split a, Split b) {
    mid = mad_wide(a.hi, b.lo, mid);
    mid = mad_wide(a.lo, b.hi, mid);
    hi = mad_wide(a.hi, b.hi, hi);
  }
  ATI_HD i64 value(int K = 0) const { return (i64)((u64)hi << K) + (mid >> (32 - K)); }
};

// an operand: x 2^e
struct Num {
  i64 x;
  int e;
};

// Inputs with an exponent above E_MAX (infinities and NaNs among them) leave the point to the FP64 arithmetic: products of
// five inputs stay in FP64's range.  Results below FP64's normal range are zero.
constexpr int E_MAX = 1023 + 200;
// a double as it is: 2^59 <= |x| < 2^60, but for subnormals and zero (x = 0)
ATI_HD Num num(double f) {
  const int h = hi_word(f), g = (h >> 20) & 0x7ff;
  const u64 m = ((u64)(((unsigned)h & 0xfffffu) | (g ? 0x100000u : 0u)) << 32 | lo_word(f)) << 7;
  const i64 s = (i64)(h >> 31);
  return {((i64)m ^ s) - s, imax(g, 1) - 1023 - 59};
}
ATI_HD double to_double(Num a) {
  const double d = (double)a.x;
  const int h = hi_word(d), m = (h & 0x7fffffff) + imax(a.e, -2000) * (1 << 20);
  return m < (1 << 20) || a.x == 0 ? 0.0 : from_words(m | (h & (int)0x80000000), lo_word(d));
}
// |x| < 2^60 moved up to 2^59 and above (a value below 2^32 by 28 bits)
ATI_HD Num norm(Num a) {
  const int h = (int)(a.x >> 32), s = imax(clz((unsigned)(h ^ (h >> 31))) - 4, 0);
  return {(i64)((u64)a.x << s), a.e - s};
}
// a sum of N <= 5 products of operands below 2^60, each aligned to the largest: below 2^60
template <int N>
ATI_HD Num dot(const Num (&a)[N], const Num (&b)[N]) {
  constexpr int K = N == 1 ? 4 : (N == 2 ? 3 : (N <= 4 ? 2 : 1));
  int E = a[0].e + b[0].e;
#pragma unroll
  for (int k = 1; k < N; k++) E = imax(E, a[k].e + b[k].e);
  Dot d;
  d.mid = (i64)1 << (31 - K);  // (to the nearest)
#pragma unroll
  for (int k = 0; k < N; k++) {
    const Split u = split(N == 1 ? a[k].x : shr(a[k].x, E - a[k].e - b[k].e)), v = split(b[k].x);
    d.add(u, v);
    if (N == 2) d.mid += mad_wide(u.lo, v.lo, (i64)1 << 31) >> 32;
  }
  return {d.value(K), E + 64 - K};
}
ATI_HD Num mul(Num a, Num b) { return dot<1>({a}, {b}); }

}  // namespace fxf

// one point's inputs: metrics m[direction][component], derivatives dv[field u v w T][direction], velocity, pressure,
// state, r1 = mu J (the viscosity times the Jacobian), r2 = r1 / ((gamma - 1) Pr), frame velocity
struct FixFluxIn {
  double m[3][3], dv[4][3], vel[3], p, q[5], r1, r2, umf[3];
};

// F[c * 3 + n]: component c of the flux along direction n; false (F not set) for a point left to the FP64 arithmetic
template <bool VISC>
ATI_HD bool flux_point_fixed(const FixFluxIn &I, double *F) {
  using namespace fxf;
  unsigned all = umax(mag(I.p), umax(mag(I.q[0]), mag(I.q[4])));
#pragma unroll
  for (int n = 0; n < 3; n++) {
#pragma unroll
    for (int k = 0; k < 3; k++) all = umax(all, mag(I.m[n][k]));
    all = umax(all, umax(mag(I.q[1 + n]), umax(mag(I.vel[n]), mag(I.umf[n]))));
    if (VISC)
#pragma unroll
      for (int f = 0; f < 4; f++) all = umax(all, mag(I.dv[f][n]));
  }
  if (VISC) all = umax(all, umax(mag(I.r1), mag(I.r2)));
  if ((int)(all >> 20) > E_MAX) return false;
  Num M[3][3];
#pragma unroll
  for (int n = 0; n < 3; n++)
#pragma unroll
    for (int k = 0; k < 3; k++) M[n][k] = num(I.m[n][k]);
  // minus the stresses, t: xx yy zz xy yz zx, and w = u . t - r2 grad T - p u_inf
  Num t[6], w[3];
  const Num p = num(I.p);
  if (VISC) {
    auto grad = [&](int f, int k) {
      return dot<3>({M[0][k], M[1][k], M[2][k]}, {num(I.dv[f][0]), num(I.dv[f][1]), num(I.dv[f][2])});
    };
    const Num r1 = num(-I.r1), r1t = num(-I.r1 * (2.0 / 3.0)), r2 = num(-I.r2);
    const Num ux = grad(0, 0), vy = grad(1, 1), wz = grad(2, 2);
    {  // 2 u_x - 2/3 div u = 2/3 (2 u_x - v_y - w_z)
      const int E = imax(ux.e, imax(vy.e, wz.e)) + 2;
      const i64 a = shr(ux.x, E - ux.e), b = shr(vy.x, E - vy.e), c = shr(wz.x, E - wz.e);
      t[0] = mul(r1t, norm({2 * a - b - c, E}));
      t[1] = mul(r1t, norm({2 * b - a - c, E}));
      t[2] = mul(r1t, norm({2 * c - a - b, E}));
    }
    auto shear = [&](Num a, Num b) {
      const int E = imax(a.e, b.e) + 1;
      return mul(r1, norm({shr(a.x, E - a.e) + shr(b.x, E - b.e), E}));
    };
    t[3] = shear(grad(1, 0), grad(0, 1));
    t[4] = shear(grad(2, 1), grad(1, 2));
    t[5] = shear(grad(0, 2), grad(2, 0));
    const Num u[3] = {num(I.vel[0]), num(I.vel[1]), num(I.vel[2])};
    const int at[3][3] = {{0, 3, 5}, {3, 1, 4}, {5, 4, 2}};
#pragma unroll
    for (int k = 0; k < 3; k++)
      w[k] = norm(dot<5>({t[at[k][0]], t[at[k][1]], t[at[k][2]], norm(grad(3, k)), num(-I.umf[k])}, {u[0], u[1], u[2], r2, p}));
  } else {
#pragma unroll
    for (int k = 0; k < 3; k++) w[k] = mul(p, num(-I.umf[k]));
  }
  // contravariant velocities in the moving frame
  Num S[3];
  {
    const Num V[3] = {num(I.vel[0] + I.umf[0]), num(I.vel[1] + I.umf[1]), num(I.vel[2] + I.umf[2])};
#pragma unroll
    for (int n = 0; n < 3; n++) S[n] = norm(dot<3>({M[n][0], M[n][1], M[n][2]}, {V[0], V[1], V[2]}));
  }
  const Num r = num(I.q[0]);
#pragma unroll
  for (int n = 0; n < 3; n++) F[n] = to_double(mul(r, S[n]));
#pragma unroll
  for (int m = 0; m < 3; m++) {
    const Num q = num(I.q[1 + m]);
    if (VISC) {
      const int E = imax(p.e, t[m].e) + 1;
      const Num s = {shr(p.x, E - p.e) + shr(t[m].x, E - t[m].e), E};
      const Num row[3] = {m == 0 ? s : (m == 1 ? t[3] : t[5]), m == 0 ? t[3] : (m == 1 ? s : t[4]),
                          m == 0 ? t[5] : (m == 1 ? t[4] : s)};
#pragma unroll
      for (int n = 0; n < 3; n++)
        F[3 * (m + 1) + n] = to_double(dot<4>({S[n], M[n][0], M[n][1], M[n][2]}, {q, row[0], row[1], row[2]}));
    } else {
#pragma unroll
      for (int n = 0; n < 3; n++) F[3 * (m + 1) + n] = to_double(dot<2>({S[n], M[n][m]}, {q, p}));
    }
  }
  const Num h = num(I.q[4] + I.p);
#pragma unroll
  for (int n = 0; n < 3; n++)
    F[12 + n] = to_double(dot<4>({S[n], M[n][0], M[n][1], M[n][2]}, {h, w[0], w[1], w[2]}));
  return true;
}

}  // namespace ati
