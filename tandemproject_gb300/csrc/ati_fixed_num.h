// ati_fixed_num.h — arithmetic shared by the 64-bit fixed-point kernels (lines, fluxes, primitives), for device and host.
#pragma once
#include <cstdint>
#include <cstring>

namespace ati {

#ifndef ATI_HD
#ifdef __CUDACC__
#define ATI_HD __host__ __device__ __forceinline__
#else
#define ATI_HD inline
#endif
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
ATI_HD i64 mul_wide(int a, int b) { return (i64)a * b; }
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
ATI_HD unsigned mag(double f) { return (unsigned)hi_word(f) & 0x7fffffffu; }
ATI_HD int imax(int a, int b) { return a > b ? a : b; }
ATI_HD int imin(int a, int b) { return a < b ? a : b; }
ATI_HD unsigned umax(unsigned a, unsigned b) { return a > b ? a : b; }
ATI_HD unsigned umin(unsigned a, unsigned b) { return a < b ? a : b; }

// a 64-bit value as hi 2^32 + lo, both signed
struct Split {
  int hi, lo;
};
ATI_HD Split split(i64 x) {
  const int lo = (int)(unsigned)x;
  return {(int)(x >> 32) + (int)((unsigned)lo >> 31), lo};
}

ATI_HD i64 shr(i64 x, int s) {
#ifdef __CUDA_ARCH__
  i64 r;
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(s));  // (a shift beyond 63 is one by 63)
  return r;
#else
  return x >> imin(s, 63);
#endif
}
ATI_HD int clz(unsigned x) {
#ifdef __CUDA_ARCH__
  return __clz((int)x);
#else
  return x ? __builtin_clz(x) : 32;
#endif
}
ATI_HD i64 shl(i64 x, int s) {
#ifdef __CUDA_ARCH__
  i64 r;
  asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(s));  // (a shift beyond 63 gives 0)
  return r;
#else
  return s > 63 ? 0 : (i64)((u64)x << s);
#endif
}

}  // namespace fxf

}  // namespace ati
