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
ATI_HD i64 prod(Split a, Split b, int K) {
  Dot d;
  d.add(a, b);
  return d.value(K);
}

// 1/f for a positive normal f, its x in (2^59, 2^60]
ATI_HD Num recip(double f) {
  const int h = hi_word(f);
  const Num n = num(f);
  const Split a = split(n.x);  // 2^59 times the significand
  i64 x = seed60(approx_rcp(float_of(0x3f800000u | (((unsigned)h & 0xfffffu) << 3) | (lo_word(f) >> 29))));
#pragma unroll
  for (int it = 0; it < 2; it++) {
    const Split s = split(x);
    x += prod(s, split(((i64)1 << 62) - prod(a, s, 7)), 2);
  }
  return {x, -119 - n.e};  // (2^59 2^60 over the significand's integer)
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
  if ((int)(umax(gr, umax(ge, gq)) >> 20) > E_MAX || (int)(umin(gr, ge) >> 20) < E_STATE_MIN) return false;
  const Num r = recip(q[0]);
  const Num m[3] = {num(q[1]), num(q[2]), num(q[3])};
  const Num v[3] = {mul(m[0], r), mul(m[1], r), mul(m[2], r)};
#pragma unroll
  for (int k = 0; k < 3; k++) out[k] = to_double(v[k]);
  // rhoE - rho u . u / 2 in the larger unit
  const Num E = num(q[4]), kin = dot<3>({m[0], m[1], m[2]}, {v[0], v[1], v[2]});
  const int up = imax(E.e, kin.e - 1);
  const i64 d = shr(E.x, up - E.e) - shr(kin.x, up - (kin.e - 1));
  if (d <= 0) return false;
  const Num p = mul(Num{d, up}, C.gamm1);
  out[4] = to_double(p);
  const Num t = mul(mul(p, C.gam), r);
  const double T = to_double(t);
  out[3] = T;
  const int et = (int)(mag(T) >> 20);
  if (t.x <= 0) return false;
  // sqrt(T) = a y, a = T 2^-2j in [1, 4): y = 1/sqrt(a)
  const int odd = (et - 1023) & 1;
  const Num tn = num(T);
  const i64 a58 = tn.x >> (1 - odd);  // 2^58 a
  const Split a = split(a58);
  const unsigned fb = (((unsigned)hi_word(T) & 0xfffffu) << 3) | (lo_word(T) >> 29);
  i64 y = seed60(approx_rsqrt(float_of((0x3f800000u + ((unsigned)odd << 23)) | fb)));
#pragma unroll
  for (int it = 0; it < 2; it++) {
    const Split s = split(y);
    const Split y2 = split(prod(s, s, 4));
    y += prod(s, split(((i64)1 << 62) - prod(a, y2, 8)), 1);
  }
  const Num root = {prod(a, split(y), 4), -58 + ((et - 1023 - odd) >> 1)};  // sqrt(T), its x below 2^59
  out[5] = to_double(mul(mul(mul(tn, root), recip(T + C.s)), C.c));
  return true;
}

}  // namespace ati
