// ati_fixed.cu — 64-bit fixed-point line sweeps of the FP64 fast path (see ati_fixed.h).
//
// k_sweep_fix is the segmented line solve of k_sweep_seg (ati_kernels.cu) in integers: 32 consecutive lines of one
// block and one field staged whole in shared memory as a [point][line] tile, one warp per segment of about 48 points,
// lane l line l, segment carries handed on by one warp (src/Subroutines3D.f90:84-206).
//
// Scale of a line.  M: the largest exponent on the line.  The values become integers F = f 2^(61-M) (|F| < 2^62).  G: the
// largest |F(i+1) - F(i)|, with the difference across the ends of a periodic line.  F is then shifted so that G < 2^gbits,
// gbits from the operator's amplification: the shift may push high bits of F out, since the operator reads differences
// only, and those are exact modulo 2^64.  A coefficient product keeps all but its lowest partial product (about one
// unit), so a row's rounding error is some 2^-57 of the line's largest difference, where FP64 rounds at 2^-53 of each
// row's values: on lines of all kinds tried (random, smooth, nearly uniform, boundary layers, peaks) a derivative's error
// against extended precision is 0.1 to 0.9 of the FP64 solve's (periodic lines: 0.6 to 1.7, where the closure weights'
// own rounding, which the two treat differently, sets it).
//
// Bound: integer issue.  A row takes some 185 warp instructions, 33 of them 64-bit multiply-adds of 4 clocks, at 15 to 19
// warps an SM (the tiles fill the shared memory): 45-55 % of the issue slots, the FP64 pipe 31 % busy with the
// conversions in and out, DRAM at 20-30 %.  On 8.85 M points (4.5 fields a launch, 2070 MHz): xi 795 -> 453 us, eta
// 754 -> 383, zeta 764 -> 385 a derivative launch, the xi and eta filters 1093 -> 544 and 954 -> 467, against the FP64
// sweeps (k_sweep_xc, k_sweep_g), which keep the FP64 pipe 86-91 % busy.
#include <cuda_runtime.h>

#include <cstdint>

#include "ati_fixed.h"

namespace ati {
namespace fast {
namespace {

using i64 = long long;
using u64 = unsigned long long;

__device__ __forceinline__ i64 mad_wide(int a, int b, i64 c) {
  i64 r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}

// a 64-bit value as hi 2^32 + lo with both signed
struct Split {
  int hi, lo;
};
__device__ __forceinline__ Split split(i64 x) {
  const int lo = (int)(unsigned)x;
  return {(int)(x >> 32) + (int)((unsigned)lo >> 31), lo};
}

// a sum of coefficient products, BITS fraction bits in the coefficients' high words: hi counts units of 2^(32-BITS),
// mid units of 2^-BITS
template <int BITS = FX_BITS>
struct Acc {
  i64 hi, mid;
  __device__ Acc() : hi(0), mid((i64)1 << (BITS - 1)) {}
  __device__ __forceinline__ void add(int chi, int clo, Split x) {
    mid = mad_wide(chi, x.lo, mid);
    mid = mad_wide(clo, x.hi, mid);
    hi = mad_wide(chi, x.hi, hi);
  }
  __device__ __forceinline__ i64 value() const { return (i64)((u64)hi << (32 - BITS)) + (mid >> BITS); }
};

// the line ends' sums, whose coefficients take FX_END_BITS: the lowest partial products are kept too
struct AccEnd : Acc<FX_END_BITS> {
  __device__ __forceinline__ void add(int chi, int clo, Split x) {
    Acc<FX_END_BITS>::add(chi, clo, x);
    mid += mad_wide(clo, x.lo, (i64)1 << 31) >> 32;
  }
};

// f 2^x to the nearest integer, x20 = x 2^20 added to the exponent field; values that this leaves below 2^-900 of the
// line's scale (thr: the smallest high word that stays normal) are zero
__device__ __forceinline__ i64 to_fixed(double f, int x20, unsigned thr) {
  const int hi = __double2hiint(f);
  const bool z = ((unsigned)hi & 0x7fffffffu) < thr;
  return __double2ll_rn(__hiloint2double(z ? 0 : hi + x20, __double2loint(f)));  // (a zero high word: a subnormal)
}

// v 2^x as a double; x moves the exponent of the converted integer (the line's scale keeps it in the normal range)
__device__ __forceinline__ double from_fixed(i64 v, int x20) {
  const double d = (double)v;
  const int hi = __double2hiint(d);
  return __hiloint2double(hi == 0 ? 0 : hi + x20, __double2loint(d));
}

template <int NN>
__device__ __forceinline__ bool line_of(const BlockDev &B, int t, int64_t &base, int64_t &stride, int &jk) {
  const int nx = B.lxi + 1, ny = B.let + 1, nz = B.lze + 1;
  if (NN == 1) {
    base = B.off + (int64_t)t * nx; stride = 1; jk = t;
    return t < ny * nz;
  } else if (NN == 2) {
    const int xi = t % nx, ze = t / nx;
    base = B.off + (int64_t)ze * nx * ny + xi; stride = nx; jk = xi * nz + ze;
    return t < nx * nz;
  }
  base = B.off + t; stride = (int64_t)nx * ny; jk = t;
  return t < nx * ny;
}

__device__ __forceinline__ void cp_async8(void *smem, const void *gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}

constexpr int RS = SEG_LINES + 1;  // tile row stride in doubles: rows and columns of a tile are free of bank conflicts

// scales: lines whose largest exponent lies outside [EM_LO, EM_HI] go through ldexp on the way in and out
constexpr int EM_LO = 256, EM_HI = 1900;

// (96 registers a thread: measured 481, 417, 397 us at the 128 the compiler takes unbounded, 453, 383, 385 at 96 and 486,
// 404, 401 at 80, xi, eta and zeta derivatives of 8.85 M points)
template <int NN, bool FILT>
__global__ void __maxnreg__(96) k_sweep_fix(const __grid_constant__ FixArgs a) {
  extern __shared__ __align__(16) unsigned char fx_smem[];
  const int nwarp = (int)(blockDim.x >> 5);
  const LTile LT = a.lt[blockIdx.x];
  const BlockDev &B = a.blk[LT.b];
  const int f = blockIdx.y;
  const int lane = (int)(threadIdx.x & 31), w = (int)(threadIdx.x >> 5);
  const int L = NN == 1 ? B.lxi + 1 : (NN == 2 ? B.let + 1 : B.lze + 1);
  const int t0 = LT.t0, nx = B.lxi + 1;
  const int nl = t0 >= B.nbsize[NN] ? 0
                 : (NN == 2 && a.rowtiles) ? min(SEG_LINES, nx - t0 % nx)
                                           : min(SEG_LINES, (int)B.nbsize[NN] - t0);
  // shared memory: per segment and line the two values passed on and received, the exponent and difference maxima,
  // then the tile
  longlong2 *cf = reinterpret_cast<longlong2 *>(fx_smem), *cx = cf + nwarp * SEG_LINES;
  unsigned *smax = reinterpret_cast<unsigned *>(cx + nwarp * SEG_LINES);
  double *tile = reinterpret_cast<double *>(smax + nwarp * SEG_LINES);
  int64_t base = 0, stride = 1;
  int jk = 0;
  line_of<NN>(B, t0 + lane, base, stride, jk);
  const double *in = a.io.in + f * a.io.in_fs;

  // 1. stage the lines
  if constexpr (NN == 1) {
    const double *src0 = in + B.off + (int64_t)t0 * L;
    for (int ln = w; ln < nl; ln += nwarp) {
      const double *src = src0 + (int64_t)ln * L + lane;
      double *dst = tile + lane * RS + ln;
#pragma unroll 4
      for (int i = lane; i < L; i += 32, src += 32, dst += 32 * RS) cp_async8(dst, src);
    }
  } else {
    if (lane < nl) {
      const double *src = in + base + (int64_t)w * stride;
      const int64_t step = (int64_t)nwarp * stride;
      double *dst = tile + w * RS + lane;
#pragma unroll 4
      for (int i = w; i < L; i += nwarp, src += step, dst += nwarp * RS) cp_async8(dst, src);
    }
  }
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();

  const int S = seg_count(L);
  const bool act = w < S && lane < nl;
  const int s0 = seg_start(w, L, S), s1 = seg_start(w + 1, L, S);
  double *col = tile + lane;
  i64 *icol = reinterpret_cast<i64 *>(tile) + lane;
  const int *rows = a.rows + (int64_t)B.fac_off[NN] * FX_RT;
  const int *et = reinterpret_cast<const int *>(a.ends + ((int64_t)LT.b * 3 + NN - 1) * FX_ET);
  const bool per = !FILT && NN == 3 && B.ndf[0][NN] == 1;  // both faces periodic onto this block

  // 2. the line's largest exponent; a segment also reads the first row of the next one and, at the ends of a
  // periodic line, the other end
  unsigned mx = 0;
  double fnext = 0, fwrap = 0;
  if (act) {
#pragma unroll 4
    for (int i = s0; i < s1; i++) mx = max(mx, (unsigned)__double2hiint(col[i * RS]) & 0x7fffffffu);
    if (w < S - 1) fnext = col[s1 * RS];
    if (per && w == S - 1) fwrap = col[0];
    smax[w * SEG_LINES + lane] = mx;
  }
  __syncthreads();
  int em = 1023, pre = 0;  // pre: the line is scaled by 2^pre on the way in (very small or very large values)
  bool bad = false;        // a value that is not finite: the whole line's results are NaN, as the recurrence gives
  if (act) {
    for (int k = 0; k < S; k++) mx = max(mx, smax[k * SEG_LINES + lane]);
    em = (int)(mx >> 20);
    bad = em == 0x7ff;
    if (bad || mx == 0) {
      em = 1023;  // (mx 0: values below 2^-1042 at most, taken as zero)
    } else if (em < EM_LO || em > EM_HI) {
      pre = em < EM_LO ? 900 : -200;
      em = (__double2hiint(ldexp(__hiloint2double((int)mx, -1), pre)) >> 20) & 0x7ff;
    }
    // (loops of their own, here and at the results: inside the common loops the compiler would predicate the
    // scaling and issue its FP64 operations for every row)
    if (pre) {
      for (int i = s0; i < s1; i++) col[i * RS] = ldexp(col[i * RS], pre);
      fnext = ldexp(fnext, pre);
      fwrap = ldexp(fwrap, pre);
    }
  }
  __syncthreads();

  // 3. fixed point, in place, and the largest difference of neighbours
  if (act) {
    const int c20 = (1023 + 61 - em) * (1 << 20);
    const unsigned thr = (unsigned)max(em - 900, 1) << 20;  // (em is at least EM_LO)
    auto conv = [&](double v) { return to_fixed(v, c20, thr); };
    u64 acc = 0;
    auto grow = [&](i64 x, i64 y) {
      const i64 d = x - y;
      acc |= (u64)(d ^ (d >> 63));
    };
    i64 Fp = conv(col[s0 * RS]);
    icol[s0 * RS] = Fp;
#pragma unroll 4
    for (int i = s0 + 1; i < s1; i++) {
      const i64 v = conv(col[i * RS]);
      icol[i * RS] = v;
      grow(v, Fp);
      Fp = v;
    }
    if (w < S - 1) grow(conv(fnext), Fp);
    if (per && w == S - 1) grow(conv(fwrap), Fp);
    smax[w * SEG_LINES + lane] = 64 - __clzll((i64)acc);  // bits of the largest difference
  }
  __syncthreads();
  int sl = 0;  // the line's shift to the left
  int x20 = 0, xex = 0;
  if (act) {
    unsigned m = 0;
    for (int k = 0; k < S; k++) m = max(m, smax[k * SEG_LINES + lane]);
    const int s = a.gbits - (int)m;
    sl = max(s, 0);
    if (s < 0)  // differences as large as the values
      for (int i = s0; i < s1; i++) icol[i * RS] >>= -s;
    // a unit of the scaled line is 2^(em - 1023 - 61 - s - k)
    xex = em - 1084 - s - a.kscale - pre;
    x20 = xex << 20;
  }
  __syncthreads();
  const bool odd = bad || pre != 0;
  auto odd_result = [&](i64 v) { return bad ? __hiloint2double(0x7ff80000, 0) : ldexp((double)v, xex); };
  auto ld = [&](int i) -> i64 { return (i64)((u64)icol[i * RS] << sl); };
  auto rd4 = [](const int *p) { return __ldg(reinterpret_cast<const int4 *>(p)); };
  auto rd2 = [](const int *p) { return __ldg(reinterpret_cast<const int2 *>(p)); };

  // 4. what a segment reads outside its own rows, before any row is overwritten: the closure rows, the first window
  // and the three rows after the segment
  const int ilo = max(s0, 4), ihi = min(s1, L - 3);
  i64 sbs[3] = {0, 0, 0}, sbe[3] = {0, 0, 0}, sb3 = 0;
  i64 a0 = 0, a1 = 0, a2 = 0, a3 = 0, a4 = 0, a5 = 0, h0 = 0, h1 = 0, h2 = 0;
  auto stencil = [&](int4 t0_, int2 t1_, i64 x0, i64 x1, i64 x2, i64 x3, i64 x4, i64 x5, i64 x6, Acc<> &q) {
    if constexpr (!FILT) {
      q.add(t0_.x, t0_.y, split(x4 - x2));
      q.add(t0_.z, t0_.w, split(x5 - x1));
      q.add(t1_.x, t1_.y, split(x6 - x0));
    } else {
      const i64 c = x3 + x3;
      q.add(t0_.x, t0_.y, split(x4 + x2 - c));
      q.add(t0_.z, t0_.w, split(x5 + x1 - c));
      q.add(t1_.x, t1_.y, split(x6 + x0 - c));
    }
  };
  if (act) {
    auto ends = [&](int side, i64 *sb) {
      // rows 0-2 from either end; p(q): the q-th point from that end
      auto p = [&](int q) { return ld(side ? L - 1 - q : q); };
      if (per) {
        // rows 0 and 1: sums over both ends of the line (the closure of src/Subroutines3D.f90:16-80 taken here)
        const int *c = et + 2 * (54 + 48 * side);
        // point q of the sums: 0..11 from this end, then the other end's points inwards
        auto pt = [&](int q) { return q < 12 ? p(q) : p(L - 1 - (q - 12)); };
        i64 r0 = 0, r1 = 0;
#pragma unroll 1
        for (int q = 0; q < 24; q += 4) {
          Acc<> A, D;
          // difference q: neighbours, but number 11 goes from this end's first point to the other end's
#pragma unroll
          for (int u = 0; u < 4; u++) {
            const Split d = split(q + u == 11 ? pt(12) - pt(0) : pt(q + u + 1) - pt(q + u));
            const int2 ca = rd2(c + 2 * (q + u)), cd = rd2(c + 2 * (24 + q + u));
            A.add(ca.x, ca.y, d);
            D.add(cd.x, cd.y, d);
          }
          r0 += A.value();
          r1 += D.value();
        }
        sb[0] = r0;
        sb[1] = r1;
        // row 2: the interior stencil with its farthest point from the other end
        const int i = side ? L - 3 : 2;
        const int *t = rows + (int64_t)i * FX_RT;
        Acc<> A;
        stencil(rd4(t), rd2(t + 4), side ? ld(L - 6) : ld(L - 2), ld(i - 2), ld(i - 1), ld(i), ld(i + 1), ld(i + 2),
                side ? ld(1) : ld(5), A);
        sb[2] = A.value();
      } else {
        i64 pt[7];
#pragma unroll
        for (int q = 0; q < 7; q++) pt[q] = p(q);
#pragma unroll
        for (int r = 0; r < 3; r++) {
          AccEnd A;
#pragma unroll
          for (int q = 0; q < 6; q++) {
            const int2 c = rd2(et + 2 * (18 * side + 6 * r + q));
            A.add(c.x, c.y, split(pt[q < r ? q : q + 1] - pt[r]));
          }
          sb[r] = A.value();
        }
      }
    };
    if (w == 0) {
      ends(0, sbs);
      AccEnd A;
      const i64 c = FILT ? 2 * ld(3) : 0;
#pragma unroll
      for (int d = 1; d <= 3; d++) {
        const int2 k = rd2(et + 2 * (149 + d));
        A.add(k.x, k.y, split(FILT ? ld(3 + d) + ld(3 - d) - c : ld(3 + d) - ld(3 - d)));
      }
      sb3 = A.value();
    }
    if (w == S - 1) ends(1, sbe);
    if (ilo < ihi) {
      a0 = ld(ilo - 3); a1 = ld(ilo - 2); a2 = ld(ilo - 1); a3 = ld(ilo); a4 = ld(ilo + 1); a5 = ld(ilo + 2);
    }
    if (w < S - 1) { h0 = ld(s1); h1 = ld(s1 + 1); h2 = ld(s1 + 2); }
  }
  __syncthreads();

  // 5. forward elimination of the segment from zero incoming values, in place
  if (act) {
    i64 u2 = 0, u1 = 0;
    auto put = [&](int i, i64 v) {
      icol[i * RS] = v;
      u2 = u1;
      u1 = v;
    };
    auto end_row = [&](int i, i64 sb, int at) {
      AccEnd A;
      const int2 c0 = rd2(et + 2 * at), c1 = rd2(et + 2 * at + 2);
      A.add(c0.x, c0.y, split(u2));
      A.add(c1.x, c1.y, split(u1));
      put(i, sb + A.value());
    };
    // (a row's coefficients are loaded a row ahead: with most of the SM's memory taken by the tiles the tables come
    // from L2)
    int4 c0, c1;
    int2 c2;
    const int *t = rows;
    auto load = [&]() { c0 = rd4(t); c1 = rd4(t + 4); c2 = rd2(t + 8); };
    auto inner = [&](i64 x6) {
      const int4 e0 = c0, e1 = c1;
      const int2 e2 = c2;
      t += FX_RT;
      load();
      Acc<> q;
      stencil(e0, make_int2(e1.x, e1.y), a0, a1, a2, a3, a4, a5, x6, q);
      q.add(e1.z, e1.w, split(u2));
      q.add(e2.x, e2.y, split(u1));
      a0 = a1; a1 = a2; a2 = a3; a3 = a4; a4 = a5; a5 = x6;
      return q.value();
    };
    int i = s0;
    for (; i < min(s1, 3); i++) end_row(i, i == 0 ? sbs[0] : (i == 1 ? sbs[1] : sbs[2]), 36 + 2 * i);
    if (i == 3) {
      end_row(3, sb3, 153);
      i = 4;
    }
    const int iown = min(ihi, s1 - 3);
    t = rows + (int64_t)i * FX_RT;
    load();
#pragma unroll 4
    for (; i < iown; i++) put(i, inner(ld(i + 3)));
    for (; i < ihi; i++) {  // windows reaching into the next segment
      const int d = i + 3 - s1;
      put(i, inner(d == 0 ? h0 : (d == 1 ? h1 : h2)));
    }
    for (; i < s1; i++) end_row(i, i == L - 1 ? sbe[0] : (i == L - 2 ? sbe[1] : sbe[2]), 42 + 2 * (L - 1 - i));
    cf[w * SEG_LINES + lane] = make_longlong2(u2, u1);
  }
  const bool multi = S > 1;
  constexpr int CB = FILT ? FX_CBITS_FILTER : FX_BITS;
  if (multi) {
    __syncthreads();
    // 6. incoming values of every segment, carried by the first warp
    if (w == 0 && lane < nl) {
      i64 x2 = 0, x1 = 0;
      cx[lane] = make_longlong2(0, 0);
      for (int k = 1; k < S; k++) {
        const int e = seg_start(k, L, S);
        const longlong2 c = cf[(k - 1) * SEG_LINES + lane];
        const int4 t2 = rd4(rows + (int64_t)(e - 2) * FX_RT + 24), t1 = rd4(rows + (int64_t)(e - 1) * FX_RT + 24);
        const Split p2 = split(x2), p1 = split(x1);
        Acc<> A, D;
        A.add(t2.x, t2.y, p2);
        A.add(t2.z, t2.w, p1);
        D.add(t1.x, t1.y, p2);
        D.add(t1.z, t1.w, p1);
        x2 = c.x + A.value();
        x1 = c.y + D.value();
        cx[k * SEG_LINES + lane] = make_longlong2(x2, x1);
      }
    }
    __syncthreads();
  }
  double *out = a.io.out + f * a.io.out_fs;
  double *out2 = FILT && a.io.out2 ? a.io.out2 + f * a.io.out_fs : nullptr;
  double *drv = (!FILT && a.io.drva) ? a.drva + B.face_off[NN] * 10 : nullptr;
  const int64_t nbs = B.nbsize[NN];
  const int m = a.io.m0 + f;
  constexpr bool DIRECT = NN != 1 && !FILT;  // one-segment lines write their results from the back substitution
  // 7. back substitution of the segment's own forward values from zero values beyond its end; one-segment
  // derivatives along eta and zeta go straight to DRAM from there
  Split x2{0, 0}, x1{0, 0};  // the segment's incoming forward values
  if (act) {
    i64 q1 = 0, q2 = 0;
    const int *t = rows + (int64_t)(s1 - 1) * FX_RT;
    double *po = out + base + (int64_t)(s1 - 1) * stride;
    auto sweep = [&](auto direct) {
      constexpr bool DI = decltype(direct)::value;
      auto emit = [&](int i, i64 q) {
        if constexpr (DI) {
          *po = from_fixed(q, x20);
          po -= stride;
        } else {
          icol[i * RS] = q;
        }
        q2 = q1;
        q1 = q;
      };
      int i = s1 - 1;
      const int ib = max(s0, 3);
      int4 cn = rd4(t + 12);
#pragma unroll 4
      for (; i >= ib; i--) {
        const int4 c = cn;
        t -= FX_RT;
        cn = rd4(t + 12);
        Acc<> A;
        A.add(c.z, c.w, split(q2));
        A.add(c.x, c.y, split(q1));
        emit(i, icol[i * RS] + A.value());
      }
      for (; i >= s0; i--) {
        AccEnd A;
        const int2 c0 = rd2(et + 2 * (48 + 2 * i)), c1 = rd2(et + 2 * (49 + 2 * i));
        A.add(c0.x, c0.y, split(q1));
        A.add(c1.x, c1.y, split(q2));
        emit(i, icol[i * RS] + A.value());
      }
    };
    if (multi) {
      sweep(std::false_type{});
      const longlong2 x = cx[w * SEG_LINES + lane];
      x2 = split(x.x);
      x1 = split(x.y);
      const int4 r0 = rd4(rows + (int64_t)s0 * FX_RT + 16), r1 = rd4(rows + (int64_t)(s0 + 1) * FX_RT + 16);
      Acc<CB> A, D;
      A.add(r0.x, r0.y, x2);
      A.add(r0.z, r0.w, x1);
      D.add(r1.x, r1.y, x2);
      D.add(r1.z, r1.w, x1);
      cf[w * SEG_LINES + lane] = make_longlong2(q1 + A.value(), q2 + D.value());  // rows s0, s0+1
    } else if constexpr (DIRECT) {
      if (odd) x20 = 0;
      sweep(std::true_type{});
      if (odd)
        for (int i = 0; i < L; i++) {
          double *o = out + base + (int64_t)i * stride;
          *o = bad ? __hiloint2double(0x7ff80000, 0) : ldexp(*o, xex);
        }
      if (drv) {  // the line ends, read back from this thread's own stores
        drv[jk + nbs * (m - 1)] = out[base];                                    // drva(jk,m,0) = sb(is)
        drv[jk + nbs * ((m - 1) + 5)] = out[base + (int64_t)(L - 1) * stride];  // drva(jk,m,1) = sb(ie)
      }
    } else {
      sweep(std::false_type{});
    }
  }
  if (multi) {
    __syncthreads();
    // 8. values beyond every segment's end, carried backwards
    if (w == 0 && lane < nl) {
      i64 y1 = 0, y2 = 0;
      cx[(S - 1) * SEG_LINES + lane] = make_longlong2(0, 0);
      for (int k = S - 2; k >= 0; k--) {
        const int e = seg_start(k + 1, L, S);
        const longlong2 c = cf[(k + 1) * SEG_LINES + lane];
        const int4 t0_ = rd4(rows + (int64_t)e * FX_RT + 20), t1_ = rd4(rows + (int64_t)(e + 1) * FX_RT + 20);
        const Split p1 = split(y1), p2 = split(y2);
        Acc<CB> A, D;
        A.add(t0_.x, t0_.y, p1);
        A.add(t0_.z, t0_.w, p2);
        D.add(t1_.x, t1_.y, p1);
        D.add(t1_.z, t1_.w, p2);
        y1 = c.x + A.value();
        y2 = c.y + D.value();
        cx[k * SEG_LINES + lane] = make_longlong2(y1, y2);
      }
    }
    __syncthreads();
  }
  // 9. results: eta/zeta rows straight to DRAM, xi lines through the tile
  if (act && (multi || !DIRECT)) {
    Split y1{0, 0}, y2{0, 0};
    if (multi) {
      const longlong2 y = cx[w * SEG_LINES + lane];
      y1 = split(y.x);
      y2 = split(y.y);
    }
    const int *t = rows + (int64_t)s0 * FX_RT + 16;
    int4 rn = rd4(t), gn = rd4(t + 4);
    auto value = [&](int i) {
      const int4 r = rn, g = gn;
      t += FX_RT;
      rn = rd4(t);
      gn = rd4(t + 4);
      Acc<CB> A;
      A.add(r.x, r.y, x2);
      A.add(r.z, r.w, x1);
      A.add(g.x, g.y, y1);
      A.add(g.z, g.w, y2);
      return icol[i * RS] + A.value();
    };
    double *po = out + base + (int64_t)s0 * stride;
    double r = 0;
    auto put = [&](int i) {
      if constexpr (NN == 1) {
        col[i * RS] = r;
      } else {
        if (FILT) {  // rr = rr + sb (src/Subroutines3D.f90:200-202)
          r = in[po - out] + r;
          if (out2) out2[po - out] = r;
        }
        *po = r;
        po += stride;
      }
    };
    int i = s0;
    if (odd) {
      for (; i < s1; i++) {
        r = odd_result(value(i));
        if (i == 0 && drv) drv[jk + nbs * (m - 1)] = r;
        put(i);
      }
    } else {
      if (i == 0) {
        r = from_fixed(value(i), x20);
        if (drv) drv[jk + nbs * (m - 1)] = r;  // drva(jk,m,0) = sb(is)
        put(i);
        i++;
      }
#pragma unroll 4
      for (; i < s1; i++) {
        r = from_fixed(value(i), x20);
        put(i);
      }
    }
    if (w == S - 1 && drv) drv[jk + nbs * ((m - 1) + 5)] = r;  // drva(jk,m,1) = sb(ie)
  }
  if constexpr (NN == 1) {
    __syncthreads();
    const int64_t o0 = B.off + (int64_t)t0 * L;
    auto wr = [&](int64_t p, double v, double q) {
      const double r = FILT ? q + v : v;  // rr = rr + sb (src/Subroutines3D.f90:200-202)
      out[p] = r;
      if (out2) out2[p] = r;
    };
    for (int ln = w; ln < nl; ln += nwarp) {
      const int64_t lb = o0 + (int64_t)ln * L;
      int i = lane;
      for (; i + 96 < L; i += 128) {  // the filter runs in place: four inputs read before any is stored
        double q0 = 0, q1 = 0, q2 = 0, q3 = 0;
        if (FILT) { q0 = in[lb + i]; q1 = in[lb + i + 32]; q2 = in[lb + i + 64]; q3 = in[lb + i + 96]; }
        wr(lb + i, tile[i * RS + ln], q0);
        wr(lb + i + 32, tile[(i + 32) * RS + ln], q1);
        wr(lb + i + 64, tile[(i + 64) * RS + ln], q2);
        wr(lb + i + 96, tile[(i + 96) * RS + ln], q3);
      }
      for (; i < L; i += 32) wr(lb + i, tile[i * RS + ln], FILT ? in[lb + i] : 0.0);
    }
  }
}

size_t fixed_smem(int nwarp, int maxlen) {
  return (size_t)nwarp * SEG_LINES * (2 * sizeof(longlong2) + sizeof(unsigned)) + (size_t)maxlen * RS * sizeof(double);
}

template <typename K>
cudaError_t max_smem(K kernel) {
  int dev = 0, optin = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  cudaFuncAttributes fa{};
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, kernel);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes);
}

}  // namespace

cudaError_t fixed_init() {
  cudaError_t e = max_smem(k_sweep_fix<1, false>);
  if (e == cudaSuccess) e = max_smem(k_sweep_fix<2, false>);
  if (e == cudaSuccess) e = max_smem(k_sweep_fix<3, false>);
  if (e == cudaSuccess) e = max_smem(k_sweep_fix<1, true>);
  if (e == cudaSuccess) e = max_smem(k_sweep_fix<2, true>);
  return e;
}

void sweep_fixed(const Eng<double> &e, cudaStream_t st, int nn, bool filt, const SweepIO<double, double> &io) {
  FixArgs a;
  a.blk = e.blk;
  a.rows = e.fxr[filt];
  a.ends = e.fxe[filt];
  a.io = io;
  a.drva = e.drva;
  a.gbits = e.fx_gbits[filt];
  a.kscale = e.fx_k[filt];
  a.rowtiles = e.eta_rowtiles;
  for (int c = 0; c < e.nsegc[nn]; c++) {  // one launch per class of equal segment counts
    const SegClass &C = e.segc[nn][c];
    if (C.n == 0) continue;
    a.lt = e.lts[nn] + C.off;
    const int nt = SEG_LINES * seg_count(C.maxlen);
    const size_t smem = fixed_smem(seg_count(C.maxlen), C.maxlen);
    const dim3 g(C.n, io.nf);
    // The directions' and classes' sweeps of a stage run at once, and an SM runs kernels side by side only at one split
    // of its memory between L1 and shared memory: on a small handle, whose sweeps together fit the GPU, each asks for
    // the largest share, so that none waits for an SM to drain (a step of 0.23 M points 1170 -> 967 us; of 0.6 to 1.9 M
    // the same; of 3.5 M, where each sweep fills the GPU and the tables want the L1, 8139 -> 8230 us).
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    at.val.sharedMemCarveout = cudaSharedmemCarveoutMaxShared;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = g;
    cfg.blockDim = nt;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = e.N < (1 << 20) ? 1 : 0;
    auto launch = [&](auto *k) { (void)cudaLaunchKernelEx(&cfg, k, a); };
    if (!filt) {
      if (nn == 1) launch(k_sweep_fix<1, false>);
      else if (nn == 2) launch(k_sweep_fix<2, false>);
      else launch(k_sweep_fix<3, false>);
    } else {
      if (nn == 1) launch(k_sweep_fix<1, true>);
      else launch(k_sweep_fix<2, true>);
    }
  }
}

}  // namespace fast
}  // namespace ati
