// ati_fixed_prim.h — the FP64 fast path's primitives of one point in 64-bit fixed point (see ati_fixed_flux.h).
//
// u = rho u / rho, p = (gamma - 1) (rhoE - rho u . u / 2), T = gamma p / rho, mu = c T sqrt(T) / (T + S)
// (src/Main3D.f90:576-583).  Reciprocals and the reciprocal square root start from the 23-bit hardware approximations in
// FP32 and take two Newton-Raphson steps, x' = x + x (1 - a x) and y' = y + y (1 - a y^2) / 2, in fixed point.
#pragma once
#include <cmath>

#include "ati_fixed_flux.h"

namespace ati {
namespace fxf {

// density and energy from 2^-100 up (below, a state is not a flow's: FP64 operations)
constexpr int E_STATE_MIN = 1023 - 100;

// a constant as a normalised significand (2^59 <= |x| < 2^60) and its unit
struct Num {
  Split x;
  int u;
};
ATI_HD Num num(double f) {
  const int e = (int)(mag(f) >> 20);
  return {split(conv(f, e)), unit(e)};
}

ATI_HD float approx_rcp(float x) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return 1.0f / x;
#endif
}
ATI_HD float approx_rsqrt(float x) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return 1.0f / std::sqrt(x);
#endif
}
ATI_HD unsigned float_bits(float f) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(f);
#else
  unsigned u;
  std::memcpy(&u, &f, 4);
  return u;
#endif
}
ATI_HD float float_of(unsigned u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float f;
  std::memcpy(&f, &u, 4);
  return f;
#endif
}
// f in [0.5, 1] as an integer, 2^60 f
ATI_HD i64 seed60(float f) {
  const unsigned b = float_bits(f);
  return (i64)((u64)((b & 0x7fffffu) | 0x800000u) << (36 + (int)(b >> 23) - 126));
}

// a product in units of 2^(64-K) of the product's
ATI_HD i64 mul(Split a, Split b, int K) {
  Dot d;
  d.add(a, b);
  return d.value(K);
}

// 1/f for a positive normal f: x in (2^59, 2^60], 1/f = x 2^(-60 - (e - 1023)) with e the biased exponent of f
ATI_HD Split recip(double f) {
  const int h = hi_word(f);
  const Split a = split(conv(f, (h >> 20) & 0x7ff));  // 2^59 times the significand
  i64 x = seed60(approx_rcp(float_of(0x3f800000u | (((unsigned)h & 0xfffffu) << 3) | (lo_word(f) >> 29))));
#pragma unroll
  for (int it = 0; it < 2; it++) {
    const Split s = split(x);
    x += mul(s, split(((i64)1 << 62) - mul(a, s, 7)), 2);
  }
  return split(x);
}

}  // namespace fxf

// the scheme's constants, taken once per tile
struct PrimFx {
  fxf::Num gamm1, gam, c;
  double s;
  ATI_HD PrimFx(double gamm1_, double gam_, double srefp1dre, double srefoo)
      : gamm1(fxf::num(gamm1_)), gam(fxf::num(gam_)), c(fxf::num(srefp1dre)), s(srefoo) {}
};

// out = u, v, w, T, p, mu; false (out not set) for a point left to the FP64 arithmetic: a state that is not finite, not
// positive in density, energy or pressure, or outside the exponent range
ATI_HD bool prim_point_fixed(const PrimFx &C, const double q[5], double out[6]) {
  using namespace fxf;
  const unsigned gr = (unsigned)hi_word(q[0]), ge = (unsigned)hi_word(q[4]);  // (a negative value: beyond E_MAX)
  const unsigned gq = umax(mag(q[1]), umax(mag(q[2]), mag(q[3])));
  const int er = (int)(gr >> 20), ee = (int)(ge >> 20), eq = imax((int)(gq >> 20), E_MIN);
  if ((int)(umax(gr, umax(ge, gq)) >> 20) > E_MAX || imin(er, ee) < E_STATE_MIN) return false;
  const Split r = recip(q[0]);
  const int ur = -60 - (er - 1023), uq = unit(eq);
  const int uv = uq + ur + 60;
  Dot kin;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const int e = imax((int)(mag(q[1 + k]) >> 20), E_MIN), s = eq - e;  // each velocity in its own unit
    const i64 m = conv(q[1 + k], e), v = mul(split(m), r, 4);
    out[k] = to_double(v, uv - s);
    kin.add(split(shr(m, s)), split(shr(v, s)));
  }
  // rhoE - rho u . u / 2 in the larger unit
  const int ue = unit(ee), uk = uq + uv + 61, up = imax(ue, uk);
  const i64 d = shr(conv(q[4], ee), up - ue) - shr(kin.value(2), up - uk);
  if (d <= 0) return false;
  // (a constant's significand at 2^59.. of 2^60: the product keeps the unit's bits)
  const i64 p = mul(split(d), C.gamm1.x, 4);
  const int u1 = up + C.gamm1.u + 60;
  out[4] = to_double(p, u1);
  const i64 gp = mul(split(p), C.gam.x, 4);
  const i64 t = mul(split(gp), r, 4);
  const double T = to_double(t, u1 + C.gam.u + 60 + ur + 60);
  out[3] = T;
  const int et = (int)(mag(T) >> 20);
  if (t <= 0) return false;
  // sqrt(T) = a y, a = T 2^-2j in [1, 4): y = 1/sqrt(a)
  const int odd = (et - 1023) & 1;
  const i64 a58 = conv(T, et) >> (1 - odd);  // 2^58 a
  const Split a = split(a58);
  const unsigned fb = (((unsigned)hi_word(T) & 0xfffffu) << 3) | (lo_word(T) >> 29);
  i64 y = seed60(approx_rsqrt(float_of((0x3f800000u + ((unsigned)odd << 23)) | fb)));
#pragma unroll
  for (int it = 0; it < 2; it++) {
    const Split s = split(y);
    const Split y2 = split(mul(s, s, 4));
    y += mul(s, split(((i64)1 << 62) - mul(a, y2, 8)), 1);
  }
  const i64 root = mul(a, split(y), 4);  // 2^58 sqrt(a), below 2^59
  const double ts = T + C.s;
  const Split rs = recip(ts);
  const int es = (int)(mag(ts) >> 20);
  const i64 tt = mul(split(conv(T, et)), split(root), 4);                 // T sqrt(a)
  const i64 x = mul(split(mul(split(tt), rs, 4)), C.c.x, 4);
  out[5] = to_double(x, unit(et) + (-58 + ((et - 1023 - odd) >> 1)) + 60 + (-60 - (es - 1023)) + 60 + C.c.u + 60);
  return true;
}

}  // namespace ati
