// ati_convert.h — conversions between FP32 and FP64 on the integer pipes.
//
// On GB300 the FP64 pipe does 1/55 of the FP32 work per clock and also executes
// the F2F conversion instructions, so the mixed path's RK update and filter,
// which add FP32 increments to the FP64 state, spend much of their time there.
// widen() does the exact conversion with integer and bit operations, straight
// from the IEEE-754 binary32/binary64 layouts; zero is handled, and subnormals,
// infinities and NaNs fall back to the instruction.  It gives the instruction's
// result bit for bit (checked on the device by ati_check_conversions).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

namespace ati {

// float -> double, exact: re-bias the exponent (127 -> 1023) and pad the significand
__device__ __forceinline__ double widen(float f) {
  const unsigned u = __float_as_uint(f);
  const unsigned e = (u >> 23) & 0xffu, m = u & 0x7fffffu, s = u & 0x80000000u;
  if (e - 1u < 254u) return __hiloint2double((int)(s | ((e + 896u) << 20) | (m >> 3)), (int)(m << 29));
  if ((u << 1) == 0u) return __hiloint2double((int)s, 0);  // signed zero
  return (double)f;  // subnormal, infinity, NaN
}

// 1/a and 1/sqrt(a) for the FP64 fast build, for positive normal a: the
// hardware approximations (PTX rcp.approx.ftz.f64, rsqrt.approx.ftz.f64) refined
// by two Newton-Raphson steps each, x' = x + x (1 - a x) and
// y' = y + y (1 - a y^2) / 2, each of which squares the relative error.  The
// results are within a few ulp of the correctly rounded ones (the bound is
// checked against the division and the square root on the device by
// ati_check_recip); they take about half the FP64 operations of the IEEE
// division and square root.
__device__ __forceinline__ double recip_nr(double a) {
  double x;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(a));
  double e = fma(-a, x, 1.0);
  x = fma(x, e, x);
  e = fma(-a, x, 1.0);
  return fma(x, e, x);
}
__device__ __forceinline__ double rsqrt_nr(double a) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
#pragma unroll
  for (int it = 0; it < 2; it++) {
    const double e = fma(-(a * y), y, 1.0);
    y = fma(y, 0.5 * e, y);
  }
  return y;
}

// (an instruction the compiler cannot predicate: the block that holds it stays behind a branch)
__device__ __forceinline__ void keep_branch() { asm volatile("nanosleep.u32 0;"); }

// K conversions at a time, the values outside the integer forms' range behind one branch (zeros, subnormals, infinities
// and NaNs on the way in; results outside the normal float range on the way out).  After a plain test the compiler
// predicates the conversion instruction, and a predicated-off F2F still takes its turn in the FP64 pipe: the mixed
// filter sweeps spent 3.8 FP64 instructions a point and field, 1.4 of them its own additions.  Results are the
// instruction's, bit for bit (checked on the device by ati_check_conversions).
// Narrowing rounds to nearest even: the significand's top 23 bits and a carry decided by the 29 bits dropped, which may
// run into the exponent, as the rounding requires (up to infinity).
template <int K>
__device__ __forceinline__ void narrow_all(const double (&v)[K], float (&o)[K]) {
  bool odd = false;
#pragma unroll
  for (int k = 0; k < K; k++) {
    const unsigned hi = (unsigned)__double2hiint(v[k]), lo = (unsigned)__double2loint(v[k]);
    odd |= (hi & 0x7fffffffu) - (897u << 20) >= (254u << 20);
    const unsigned m = __funnelshift_l(lo, hi, 3);  // the significand's top 23 bits under the exponent's low bits
    const unsigned up = (lo & 0x1fffffffu) + 0x0fffffffu + (m & 1u);  // bit 29: round up (ties to even)
    o[k] = __uint_as_float((m - (896u << 23) + (up >> 29)) | (hi & 0x80000000u));
  }
  if (odd) {
    keep_branch();
#pragma unroll
    for (int k = 0; k < K; k++) o[k] = (float)v[k];
  }
}
template <int K>
__device__ __forceinline__ void widen_all(const float (&v)[K], double (&o)[K]) {
  bool odd = false;
#pragma unroll
  for (int k = 0; k < K; k++) {
    const unsigned u = __float_as_uint(v[k]), a = u & 0x7fffffffu;
    odd |= a - 0x00800000u >= 0x7f000000u;
    o[k] = __hiloint2double((int)((u & 0x80000000u) | ((a >> 3) + (896u << 20))), (int)(u << 29));
  }
  if (odd) {
    keep_branch();
#pragma unroll
    for (int k = 0; k < K; k++) o[k] = (double)v[k];
  }
}

// conversion between the engine types: FP32 -> FP64 on the integer pipes; the other direction is the conversion
// instruction here, and the kernels whose time it was (filters, fluxes, divergence, primitives) call narrow_all
template <typename TO, typename TI>
__device__ __forceinline__ TO cvt(TI v) {
  if constexpr (std::is_same<TO, TI>::value) return v;
  else if constexpr (std::is_same<TO, double>::value && std::is_same<TI, float>::value) return widen(v);
  else return (TO)v;
}

}  // namespace ati
