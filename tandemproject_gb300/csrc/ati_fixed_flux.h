// ati_fixed_flux.h — the FP64 fast path's fluxes at one point in 64-bit fixed point (see ati_fixed.h for why).
//
// A group of inputs that enter sums together (the nine metrics, the velocity derivatives, the temperature derivatives,
// the velocities, ...) shares one exponent, its largest; an input becomes a signed integer below 2^60 in that unit.
// Sums of products run in integers (three 32 x 32 + 64 bit multiply-adds a product, the lowest partial product left
// out); sums over groups align to the larger unit first.  A flux component's error before its one rounding is some
// 2^-56 of the largest term that enters it, where FP64 rounds each of some ten operations at 2^-53: against extended
// precision, 0.4 to 0.8 of the FP64 arithmetic's error on flows at rest, slow and fast, equal where a component is a
// single product.
//
// The fluxes are formed as tensors in space and then contracted with the metrics (src/Main3D.f90:631-766):
//   rho V,  (rho u_m) V_k + p delta - tau,  (rhoE + p) V - p u_inf - r2 grad T - u . tau,   V = u + u_inf
#pragma once
#include <cstdint>
#include <cstring>

namespace ati {

#ifdef __CUDACC__
#define ATI_HD __host__ __device__ __forceinline__
#else
#define ATI_HD inline
#endif

namespace fxf {

using i64 = long long;
using u64 = unsigned long long;

ATI_HD i64 mad_wide(int a, int b, i64 c) {
#ifdef __CUDA_ARCH__
  i64 r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
#else
  return (i64)((u64)((i64)a * b) + (u64)c);
#endif
}
ATI_HD int hi_word(double f) {
#ifdef __CUDA_ARCH__
  return __double2hiint(f);
#else
  u64 b;
  std::memcpy(&b, &f, 8);
  return (int)(b >> 32);
#endif
}
ATI_HD unsigned lo_word(double f) {
#ifdef __CUDA_ARCH__
  return (unsigned)__double2loint(f);
#else
  u64 b;
  std::memcpy(&b, &f, 8);
  return (unsigned)b;
#endif
}
ATI_HD double from_words(int hi, unsigned lo) {
#ifdef __CUDA_ARCH__
  return __hiloint2double(hi, (int)lo);
#else
  const u64 b = (u64)(unsigned)hi << 32 | lo;
  double f;
  std::memcpy(&f, &b, 8);
  return f;
#endif
}
ATI_HD int imax(int a, int b) { return a > b ? a : b; }
ATI_HD int imin(int a, int b) { return a < b ? a : b; }
ATI_HD unsigned umax(unsigned a, unsigned b) { return a > b ? a : b; }

// a 64-bit value as hi 2^32 + lo, both signed
struct Split {
  int hi, lo;
};
ATI_HD Split split(i64 x) {
  const int lo = (int)(unsigned)x;
  return {(int)(x >> 32) + (int)((unsigned)lo >> 31), lo};
}

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

// exponents: a group's exponent e (biased, of its largest value) is kept in [E_MIN, E_MAX]; smaller groups lose what
// lies 60 bits below 2^-200, and a point with a larger or non-finite value is left to the FP64 arithmetic
constexpr int E_MIN = 1023 - 200, E_MAX = 1023 + 200;
constexpr int BITS = 60;
// |x| < 2^60, x 2^(unit) the value
ATI_HD int unit(int e) { return e - 1023 - (BITS - 1); }
ATI_HD unsigned mag(double f) { return (unsigned)hi_word(f) & 0x7fffffffu; }
ATI_HD i64 conv(double f, int e) {
  const int h = hi_word(f), r = imin(e - ((h >> 20) & 0x7ff), 63);
  const u64 m = (((u64)((unsigned)h & 0xfffffu) | 0x100000u) << 32 | lo_word(f)) << (BITS - 53);
  const i64 s = (i64)(h >> 31);
  return ((i64)(m >> r) ^ s) - s;
}
// x 2^u as a double (x = 0: zero)
ATI_HD double to_double(i64 x, int u) {
  const double d = (double)x;
  const int h = hi_word(d);
  return from_words(h == 0 ? 0 : h + u * (1 << 20), lo_word(d));
}
ATI_HD i64 shr(i64 x, int s) { return x >> imin(s, 63); }

}  // namespace fxf

// one point's inputs: metrics m[direction][component], derivatives dv[field u v w T][direction], velocity, pressure,
// state, r1 = mu J (the viscosity times the Jacobian), r2 = r1 / ((gamma - 1) Pr), frame velocity
struct FluxIn {
  double m[3][3], dv[4][3], vel[3], p, q[5], r1, r2, umf[3];
};

// F[c * 3 + n]: component c of the flux along direction n; false (F not set) for a point left to the FP64 arithmetic
template <bool VISC>
ATI_HD bool flux_point_fixed(const FluxIn &I, double *F) {
  using namespace fxf;
  unsigned gm = 0, gv = 0, gq = 0, gd = 0, gt = 0;
#pragma unroll
  for (int n = 0; n < 3; n++)
#pragma unroll
    for (int k = 0; k < 3; k++) gm = umax(gm, mag(I.m[n][k]));
#pragma unroll
  for (int k = 0; k < 3; k++) {
    gv = umax(gv, umax(mag(I.vel[k]), mag(I.umf[k])));
    gq = umax(gq, mag(I.q[1 + k]));
  }
  const unsigned gr = mag(I.q[0]), gp = umax(mag(I.p), mag(I.q[4]));
  unsigned all = umax(umax(gm, gv), umax(umax(gq, gr), gp));
  if (VISC) {
#pragma unroll
    for (int n = 0; n < 3; n++) {
      gd = umax(umax(gd, mag(I.dv[0][n])), umax(mag(I.dv[1][n]), mag(I.dv[2][n])));
      gt = umax(gt, mag(I.dv[3][n]));
    }
    all = umax(all, umax(umax(gd, gt), umax(mag(I.r1), mag(I.r2))));
  }
  if ((int)(all >> 20) > E_MAX) return false;
  auto expo = [](unsigned g) { return imax((int)(g >> 20), E_MIN); };
  const int em = expo(gm), ev = expo(gv), eq = expo(gq), er = expo(gr), ep = expo(gp);
  const int um = unit(em), uv = unit(ev);
  Split M[3][3];
#pragma unroll
  for (int n = 0; n < 3; n++)
#pragma unroll
    for (int k = 0; k < 3; k++) M[n][k] = split(conv(I.m[n][k], em));
  // velocities in the moving frame
  Split vel[3], umf[3], V[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const i64 a = conv(I.vel[k], ev), b = conv(I.umf[k], ev);
    vel[k] = split(a);
    umf[k] = split(-b);
    V[k] = split(a + b);
  }
  auto contract = [&](const Split *G, int ug, double *f) {
#pragma unroll
    for (int n = 0; n < 3; n++) {
      Dot d;
#pragma unroll
      for (int k = 0; k < 3; k++) d.add(M[n][k], G[k]);
      f[n] = to_double(d.value(3), um + ug + 61);
    }
  };
  Split G[3];
  {  // mass
    const Split r = split(conv(I.q[0], er));
#pragma unroll
    for (int k = 0; k < 3; k++) {
      Dot d;
      d.add(r, V[k]);
      G[k] = split(d.value(3));
    }
    contract(G, unit(er) + uv + 61, F);
  }
  const i64 p = conv(I.p, ep);
  // viscous stresses t: xx yy zz xy yz zx in units of 2^ut; heat flux r2 grad T
  i64 t[6] = {0, 0, 0, 0, 0, 0}, hq[3] = {0, 0, 0};
  int ut = 0, uh = 0;
  if (VISC) {
    const int ed = expo(gd), et = expo(gt), e1 = expo(mag(I.r1)), e2 = expo(mag(I.r2));
    auto grad = [&](int f, int e, int up, i64 *c) {
      Split d[3];
#pragma unroll
      for (int n = 0; n < 3; n++) d[n] = split(conv(I.dv[f][n], e));
#pragma unroll
      for (int k = 0; k < 3; k++) {
        Dot s;
#pragma unroll
        for (int n = 0; n < 3; n++) s.add(M[n][k], d[n]);
        c[k] = s.value(up);
      }
    };
    i64 u[3], v[3], w[3], T[3];
    grad(0, ed, 2, u);
    grad(1, ed, 2, v);
    grad(2, ed, 2, w);
    grad(3, et, 4, T);
    // two thirds of the divergence: 2/3 = 0x2AAAAAAA.AAAAAAAA 2^-30
    const Split dv = split(u[0] + v[1] + w[2]);
    i64 mid = mad_wide(0x2aaaaaab, dv.lo, (i64)1 << 29);
    mid = mad_wide(-0x55555555, dv.hi, mid);
    const i64 d5 = (mad_wide(0x2aaaaaab, dv.hi, 0) << 2) + (mid >> 30);
    const Split r1 = split(conv(I.r1, e1)), r2 = split(conv(I.r2, e2));
    auto scaled = [&](Split r, i64 x) {
      Dot s;
      s.add(r, split(x));
      return s.value(2);
    };
    t[0] = scaled(r1, 2 * u[0] - d5);
    t[1] = scaled(r1, 2 * v[1] - d5);
    t[2] = scaled(r1, 2 * w[2] - d5);
    t[3] = scaled(r1, v[0] + u[1]);
    t[4] = scaled(r1, w[1] + v[2]);
    t[5] = scaled(r1, u[2] + w[0]);
    ut = unit(e1) + um + unit(ed) + 62 + 62;
#pragma unroll
    for (int k = 0; k < 3; k++) hq[k] = scaled(r2, T[k]);
    uh = unit(e2) + um + unit(et) + 60 + 62;
  }
  {  // momentum: q_m V_k + p delta - tau
    const int us = VISC ? imax(unit(ep), ut) : unit(ep), uq = unit(eq) + uv + 61, uP = imax(us, uq);
    const int sp = uP - unit(ep), st = uP - ut, sq = uP - uq;
    const i64 pp = shr(p, sp);
    i64 ts[6];
    if (VISC) {
#pragma unroll
      for (int k = 0; k < 6; k++) ts[k] = shr(t[k], st);
    }
#pragma unroll
    for (int m = 0; m < 3; m++) {
      const Split q = split(conv(I.q[1 + m], eq));
#pragma unroll
      for (int k = 0; k < 3; k++) {
        Dot d;
        d.add(q, V[k]);
        i64 x = shr(d.value(3), sq);
        if (m == k) x += pp;
        if (VISC) x -= ts[m == k ? m : (m + k == 1 ? 3 : (m + k == 3 ? 4 : 5))];
        G[k] = split(x);
      }
      contract(G, uP, F + 3 * (m + 1));
    }
  }
  {  // energy: (rhoE + p) V - p u_inf - r2 grad T - u . tau
    const Split h = split(conv(I.q[4], ep) + p), ps = split(p);
    const int ua = unit(ep) + uv + 62, uc = VISC ? uv + ut + 62 : 0;
    const int uE = VISC ? imax(ua, imax(uh, uc)) : ua;
    Split ts[6];
    if (VISC) {
#pragma unroll
      for (int k = 0; k < 6; k++) ts[k] = split(t[k]);
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
      Dot d;
      d.add(h, V[k]);
      d.add(ps, umf[k]);
      i64 x = shr(d.value(2), uE - ua);
      if (VISC) {
        Dot c;
#pragma unroll
        for (int j = 0; j < 3; j++) c.add(vel[j], ts[j == k ? j : (j + k == 1 ? 3 : (j + k == 3 ? 4 : 5))]);
        x -= shr(hq[k], uE - uh) + shr(c.value(2), uE - uc);
      }
      G[k] = split(x);
    }
    contract(G, uE, F + 12);
  }
  return true;
}

}  // namespace ati
