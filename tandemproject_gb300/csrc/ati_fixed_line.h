// ati_fixed_line.h — one line's solve in 64-bit fixed point, segment by segment, for device (ati_fixed.cu) and host.
//
// A line of L points is cut into segments (seg_count), a segment into groups of about eight rows (fx_groups).
// A thread has one segment; the phases below run for all segments of a line with a barrier between them
// (src/Subroutines3D.f90:84-206).
//
// Scales.  The values of a group are integers F = f 2^(61 - M), M the group's largest exponent.  The solve's values in a
// group are integers in units of 2^(W - gbits), W chosen as the sweep enters the group: the largest difference of
// neighbouring values that the group's rows read, or the values carried in from the rows before, whichever is larger.
// So the scale follows the solution along the line as a floating-point number's does, and the error of a row is relative
// to what enters it there, not to the line's largest value.  F enters the solve modulo 2^64 in the group's units (only
// differences are used); a coefficient product keeps all but its lowest partial product (about one unit).
//
// Errors against extended precision, point by point over lines of a kind, in units of the FP64 sweeps' on the same lines:
// smooth fields of one size or falling by up to a third of a bit a row 0.1 to 0.7 on average and up to 2 at single points,
// rough ones 0.4 to 0.7 (the filter 1.00: both round one product); beside a tanh layer a wave 2^-20 of it 0.4 on average,
// up to 4 in the last rows of the layer's tail, whose values fall by 5.8 bits within a group.
#pragma once
#include <cmath>

#include "ati_fixed_num.h"
#include "ati_fixed_tab.h"

namespace ati {
namespace fxl {

using namespace fxf;

struct I2 {
  int x, y;
};
struct I4 {
  int x, y, z, w;
};
ATI_HD I2 rd2(const int *p) {
#ifdef __CUDA_ARCH__
  const int2 v = __ldg(reinterpret_cast<const int2 *>(p));
  return {v.x, v.y};
#else
  return {p[0], p[1]};
#endif
}
ATI_HD I4 rd4(const int *p) {
#ifdef __CUDA_ARCH__
  const int4 v = __ldg(reinterpret_cast<const int4 *>(p));
  return {v.x, v.y, v.z, v.w};
#else
  return {p[0], p[1], p[2], p[3]};
#endif
}

// a sum of coefficient products, BITS fraction bits in the coefficients' high words: hi counts units of 2^(32-BITS),
// mid units of 2^-BITS
template <int BITS = FX_BITS>
struct Acc {
  i64 hi, mid;
  ATI_HD Acc(int chi, int clo, Split x) : hi(mul_wide(chi, x.hi)), mid(mad_wide(clo, x.hi, mul_wide(chi, x.lo))) {}
  ATI_HD void add(int chi, int clo, Split x) {
    mid = mad_wide(chi, x.lo, mid);
    mid = mad_wide(clo, x.hi, mid);
    hi = mad_wide(chi, x.hi, hi);
  }
  // (rounded down: half a unit low on average, a quarter after a solve)
  ATI_HD i64 value() const { return (i64)((u64)hi << (32 - BITS)) + (mid >> BITS); }
};
// the line ends' sums, whose coefficients take FX_END_BITS: the lowest partial products are kept too
struct AccEnd : Acc<FX_END_BITS> {
  ATI_HD static i64 low(int clo, Split x) { return mad_wide(clo, x.lo, (i64)1 << 31) >> 32; }
  ATI_HD AccEnd(int chi, int clo, Split x) : Acc<FX_END_BITS>(chi, clo, x) { mid += low(clo, x); }
  ATI_HD void add(int chi, int clo, Split x) {
    Acc<FX_END_BITS>::add(chi, clo, x);
    mid += low(clo, x);
  }
};

ATI_HD i64 move(i64 x, int s) { return shr(shl(x, imax(s, 0)), imax(-s, 0)); }  // x 2^s
// |a|, |b| < 2^bits (at least 32)
ATI_HD int bits2(i64 a, i64 b) {
  const int h = (int)(a >> 32), k = (int)(b >> 32);
  return 64 - clz((unsigned)((h ^ (h >> 31)) | (k ^ (k >> 31))));
}
// queues of up to six numbers of ten bits
ATI_HD int low10(u64 p) { return (int)p & 1023; }
ATI_HD void push_back(u64 &p, int v) { p = p >> 10 | (u64)v << 50; }  // (the first of n ends at bit 60 - 10 n)
ATI_HD void push_front(u64 &p, int v) { p = p << 10 | (u64)v; }

// f 2^(1084 - m), towards zero, for |f| below 2^(m + 1 - 1023), m at least 64 (subnormals are zero).  In integers: the
// conversion instruction takes the FP64 pipe, 64 clocks a warp, and the results' conversions need it.
ATI_HD i64 to_fixed(double f, int m) {
  const int h = hi_word(f), s = h >> 31;
  const u64 x = (u64)(((unsigned)h & 0xfffffu) | 0x100000u) << 32 | lo_word(f);
  const i64 v = shr((i64)(x << 9), m - ((h >> 20) & 0x7ff));
  return (v ^ (i64)s) - (i64)s;
}
// v 2^x as a double; x moves the exponent of the converted integer (the scales keep it in the normal range)
ATI_HD double from_fixed(i64 v, int x20) {
  const double d = (double)v;
  const int hi = hi_word(d);
  return from_words(hi == 0 ? 0 : hi + x20, lo_word(d));
}

// lines whose largest exponent lies outside [EM_LO, EM_HI] go through ldexp on the way in and out
constexpr int EM_LO = 256, EM_HI = 1900;
constexpr int W_MIN = 100;      // smallest W: results stay in the normal range
constexpr int NONE = -4096;     // the scale of a carried zero

// two carried values in units of 2^(W - gbits)
struct Pair {
  i64 a, b;
  int W;
};
// the sums of two pairs, brought to just below 2^FX_CARRY
ATI_HD Pair sum(Pair c, Pair p) {
  const int E = imax(c.W, p.W) + 1;
  const i64 a = shr(c.a, E - c.W) + shr(p.a, E - p.W), b = shr(c.b, E - c.W) + shr(p.b, E - p.W);
  const int s = bits2(a, b) - FX_CARRY;
  return {move(a, -s), move(b, -s), E + s};
}
// incoming forward values x of a segment and its own last two c to those of the next one, whose first row is e
ATI_HD Pair carry_forward(const int *rows, int e, Pair c, Pair x) {
  const I4 t2 = rd4(rows + (e - 2) * FX_RT + 24), t1 = rd4(rows + (e - 1) * FX_RT + 24);
  const Split p2 = split(x.a), p1 = split(x.b);
  Acc<> A(t2.x, t2.y, p2), D(t1.x, t1.y, p2);
  A.add(t2.z, t2.w, p1);
  D.add(t1.z, t1.w, p1);
  return sum(c, {A.value(), D.value(), x.W - rows[(e - 1) * FX_RT + 11]});
}
// values y beyond a segment's end and its own first two c (rows e, e+1) to those beyond the end of the one before
ATI_HD Pair carry_backward(const int *rows, int e, Pair c, Pair y) {
  const I4 t0 = rd4(rows + e * FX_RT + 20), t1 = rd4(rows + (e + 1) * FX_RT + 20);
  const Split p1 = split(y.a), p2 = split(y.b);
  Acc<> A(t0.x, t0.y, p1), D(t1.x, t1.y, p1);
  A.add(t0.z, t0.w, p2);
  D.add(t1.z, t1.w, p2);
  return sum(c, {A.value(), D.value(), y.W - (rows[e * FX_RT + 10] >> 16)});
}

// What other segments read of a segment: the exponents of its groups' values (M), and (edge) of largest differences:
// [0] into the first three rows, [1] and [2] in the first two groups, [3] in the last three rows, [4] and [5] in the last
// two groups
struct Scales {
  u64 M, edge;
};

// FILT: the filter, else the derivative; PER: the lines may be periodic onto themselves; RS: the tile's row stride
template <bool FILT, bool PER, int RS>
struct Segment {
  const int *rows, *et;  // row table, end table of the line
  double *col;           // the line's column: values, then integers
  int L, S, w, s0, s1, ng, fin;  // fin: the last group's first row
  bool per;              // periodic onto itself (PER)
  FixScale fs;
  int em, pre;           // the line's largest exponent, and the power of two it was scaled by (very small or large values)
  bool bad;              // a value that is not finite: the whole line's results are NaN, as the recurrence gives
  Scales sc;
  u64 Wp;                // the groups' W; before the elimination the largest difference that the group's rows read
  double fnext, fwrap;
  i64 a[3];              // the first window's first rows
  i64 tail[3];           // the next segment's first rows; the line's last three right-hand sides, from its end
  i64 rs[3];             // a periodic line's first three right-hand sides
  int W0, We, Mn;

  ATI_HD Segment(const int *rows_, const int *et_, double *col_, int L_, int S_, int w_, bool per_, FixScale fs_)
      : rows(rows_), et(et_), col(col_), L(L_), S(S_), w(w_), s0(seg_start(w_, L_, S_)), s1(seg_start(w_ + 1, L_, S_)),
        ng(fx_groups(s1 - s0)),
        fin(s0 + fx_group_start(ng - 1, ng, s1 - s0)), per(PER && per_), fs(fs_) {}

  ATI_HD int first(int g) const { return g == ng - 1 ? fin : s0 + FX_GR * g; }
  ATI_HD int end(int g) const { return g == ng - 1 ? s1 : (g == ng - 2 ? fin : s0 + FX_GR * (g + 1)); }
  ATI_HD i64 get(int i) const {
#ifdef __CUDA_ARCH__
    return reinterpret_cast<const i64 *>(col)[i * RS];
#else
    i64 v;
    std::memcpy(&v, col + i * RS, 8);
    return v;
#endif
  }
  ATI_HD void set(int i, i64 v) {
#ifdef __CUDA_ARCH__
    reinterpret_cast<i64 *>(col)[i * RS] = v;
#else
    std::memcpy(col + i * RS, &v, 8);
#endif
  }
  // exponents of a group's values, halved in the queue (F below 2^62 at an even exponent, 2^61 at an odd one)
  ATI_HD int M(u64 p) const { return imax(2 * low10(p) + 1 + pre, 64); }
  // W, and exponents of differences, counted down from the line's largest value's
  ATI_HD int W(u64 p) const { return em + 12 - low10(p); }
  ATI_HD int put_W(int W_) const { return imin(imax(em + 12 - W_, 0), 1023); }
  ATI_HD int floor_W(int W) const { return imax(W, imax(W_MIN, em - 1000)); }
  // shift from a value's integers to units of W
  ATI_HD int in(int M_, int W_) const { return M_ - W_ - 61 + fs.gbits; }
  // exponent of a result's unit
  ATI_HD int out(int W_) const { return W_ - 1023 - fs.gbits - fs.k - pre; }

  // 1. the groups' largest exponents; what a segment reads of the next one, and at the ends of a periodic line
  ATI_HD unsigned maxima() {
    unsigned mx = 0;
    sc.M = 0;
    for (int g = 0, i = s0; g < ng; g++) {
      const int i1 = end(g);
      unsigned m = 0;
      if (i1 - i >= FX_GR) {
#pragma unroll
        for (int q = 0; q < FX_GR; q++) m = umax(m, mag(col[(i + q) * RS]));
        i += FX_GR;
      }
#pragma unroll 1
      for (; i < i1; i++) m = umax(m, mag(col[i * RS]));
      push_back(sc.M, (int)(m >> 21));
      mx = umax(mx, m);
    }
    sc.M >>= 60 - 10 * ng;
    fnext = w < S - 1 ? col[s1 * RS] : 0.0;
    fwrap = per && w == S - 1 ? col[0] : 0.0;
    return mx;
  }

  // 2. values to integers, in place, and the largest differences of neighbours; mx: the line's maximum
  ATI_HD void convert(unsigned mx) {
    em = (int)(mx >> 20);
    bad = em == 0x7ff;
    pre = 0;
    if (bad || mx == 0) {
      em = 1023;  // (mx 0: values below 2^-1042 at most, taken as zero)
    } else if (em < EM_LO || em > EM_HI) {
      // (a loop of its own, here and at the results: inside the common loops the compiler would predicate the scaling
      // and issue its FP64 operations for every row)
      pre = em < EM_LO ? 900 : -200;
      em = (hi_word(ldexp(from_words((int)mx, 0xffffffffu), pre)) >> 20) & 0x7ff;
      for (int i = s0; i < s1; i++) col[i * RS] = ldexp(col[i * RS], pre);
      fnext = ldexp(fnext, pre);
      fwrap = ldexp(fwrap, pre);
    }
    Wp = 0;
    double before = 0;
    int tb = NONE, db = NONE;  // of the group before: the last three rows' differences, all that its rows read so far
    int d0 = NONE, d1 = NONE, h0 = NONE, dl = NONE, dm = NONE;  // of the first and the last groups
    u64 mp = sc.M;
    // (two values apart in scale: the exponent above that of their difference)
    auto cross = [](double x, double y) { return ((hi_word(x - y) >> 20) & 0x7ff) + 1; };
    for (int g = 0; g < ng; g++) {
      const int m = M(mp), i0 = first(g), i1 = end(g);
      mp >>= 10;
      // (differences by their high words; h: of the first two inside, t1 and t2 the last two, c: all)
      auto step = [](i64 x, i64 y) {
        const int q = (int)((x - y) >> 32);
        return (unsigned)(q ^ (q >> 31));
      };
      unsigned h = 0, t1 = 0, t2 = 0, c = 0;
      const double last = before;
      double v0;
      i64 Fp;
      int i = i0;
      if (i1 - i0 >= FX_GR) {  // (the loads and the conversions of a whole group at once)
        double v[FX_GR];
        i64 F[FX_GR];
#pragma unroll
        for (int q = 0; q < FX_GR; q++) v[q] = col[(i0 + q) * RS];
#pragma unroll
        for (int q = 0; q < FX_GR; q++) F[q] = to_fixed(v[q], m);
#pragma unroll
        for (int q = 0; q < FX_GR; q++) set(i0 + q, F[q]);
        h = step(F[1], F[0]) | step(F[2], F[1]);
        t1 = step(F[FX_GR - 2], F[FX_GR - 3]);
        t2 = step(F[FX_GR - 1], F[FX_GR - 2]);
        c = h | t1 | t2;
#pragma unroll
        for (int q = 3; q < FX_GR - 2; q++) c |= step(F[q], F[q - 1]);
        v0 = v[0];
        before = v[FX_GR - 1];
        Fp = F[FX_GR - 1];
        i += FX_GR;
      } else {
        v0 = before = col[i0 * RS];
        Fp = to_fixed(v0, m);
        set(i0, Fp);
        i++;
      }
#pragma unroll 1
      for (; i < i1; i++) {
        before = col[i * RS];
        const i64 F = to_fixed(before, m);
        set(i, F);
        t1 = t2;
        t2 = step(F, Fp);
        c |= t2;
        Fp = F;
        if (i == i0 + 2) h = c;
      }
      const int d = g > 0 ? cross(v0, last) : 0;
      // the exponent above the largest difference of rows a..b with the row before each; acc: their high words.  (Differences
      // below 2^32 are looked at again: a line of nearly one value.)
      auto expo = [&](unsigned acc, int a, int b) {
        if (acc) return 32 + (32 - clz(acc)) + m - 61;
        unsigned lo = 0;
        for (int i = a; i <= b; i++) {
          const i64 q = get(i) - get(i - 1);
          lo |= (unsigned)(q ^ (q >> 63));
        }
        return (32 - clz(lo)) + m - 61;
      };
      const int dh = imax(d, expo(h, i0 + 1, i0 + 2));
      int dt = expo(t1 | t2, i1 - 2, i1 - 1);
      if (g == ng - 1) {
        if (w < S - 1) dt = imax(dt, cross(fnext, before));
        if (per && w == S - 1) dt = imax(dt, cross(fwrap, before));
      }
      const int d_ = imax(imax(dh, dt), expo(c, i0 + 1, i1 - 1));
      if (g > 0) push_back(Wp, put_W(imax(db, dh)));
      else h0 = dh;
      d1 = g == 1 ? d_ : d1;
      d0 = g == 0 ? d_ : d0;
      dm = dl;
      dl = d_;
      db = imax(tb, d_);
      tb = dt;
    }
    push_back(Wp, put_W(db));
    Wp >>= 60 - 10 * ng;
    sc.edge = 0;
    push_front(sc.edge, put_W(dm));
    push_front(sc.edge, put_W(dl));
    push_front(sc.edge, put_W(tb));
    push_front(sc.edge, put_W(d1));
    push_front(sc.edge, put_W(d0));
    push_front(sc.edge, put_W(h0));
  }

  // 3. what a segment reads outside its own rows, before any row is overwritten.  scales(s): the groups of segment s
  template <class F>
  ATI_HD void reads(F &&scales) {
    int Mp = 0, Tb = NONE, Hn = NONE;  // last group of the segment before, first one of the next
    Mn = 0;
    if (w > 0) {
      const Scales q = scales(w - 1);
      Mp = M(q.M >> 10 * (fx_groups(s0 - seg_start(w - 1, L, S)) - 1));
      Tb = W(q.edge >> 30);
    }
    if (w < S - 1) {
      const Scales q = scales(w + 1);
      Mn = M(q.M);
      Hn = W(q.edge);
    }
    int wf = imax(W(Wp), Tb), we = imax(W(Wp >> 10 * (ng - 1)), Hn);
    Scales qs = sc, qe = sc;
    if (per && (w == 0 || w == S - 1)) {  // the closure rows read both ends
      qs = scales(0);
      qe = scales(S - 1);
      const int d = imax(imax(W(qs.edge >> 10), W(qs.edge >> 20)), imax(W(qe.edge >> 40), W(qe.edge >> 50)));
      if (w == 0) wf = imax(wf, d);
      if (w == S - 1) we = imax(we, d);
    }
    if (w == S - 1 && !per) we += fs.spare;
    if (ng == 1 || (per && S == 1)) wf = we = imax(wf, we);
    W0 = floor_W(wf);
    We = floor_W(we);
    const int i = w == 0 ? 4 : s0;  // the first inner row
#pragma unroll
    for (int q = 0; q < 3; q++) a[q] = move(get(i - 3 + q), in(w > 0 ? Mp : M(sc.M), W0));
#pragma unroll
    for (int q = 0; q < 3; q++) tail[q] = w < S - 1 ? get(s1 + q) : 0;
    if (per && (w == 0 || w == S - 1)) periodic(qs, qe);
  }
  // the first (side 0) or last three rows of a line, from its first seven points p from that end
  ATI_HD void one_sided(int side, const i64 (&p)[7], i64 (&sb)[3]) const {
    const int *c = et + 36 * side;
#pragma unroll
    for (int r = 0; r < 3; r++) {
      const I4 t = rd4(c + 12 * r), u = rd4(c + 12 * r + 4), v = rd4(c + 12 * r + 8);
      auto d = [&](int q) { return split(p[q < r ? q : q + 1] - p[r]); };
      AccEnd A(t.x, t.y, d(0));
      A.add(t.z, t.w, d(1));
      A.add(u.x, u.y, d(2));
      A.add(u.z, u.w, d(3));
      A.add(v.x, v.y, d(4));
      A.add(v.z, v.w, d(5));
      sb[r] = A.value();
    }
  }
  // Rows 0-2 from the ends of a periodic line: 0 and 1 are sums over both its ends (the closure of
  // src/Subroutines3D.f90:16-80 taken here), 2 the interior stencil with its farthest point from the other end.  The two
  // ends' sums take the same differences of neighbours: the first segment forms its own, the last one its own, a line of
  // one segment both (W0 = We there).
  ATI_HD void periodic(Scales qs, Scales qe) {
    const int e0 = seg_start(1, L, S), sl = seg_start(S - 1, L, S), n0 = fx_groups(e0), nl = fx_groups(L - sl);
    const int W_ = w == 0 ? W0 : We;
    // the scales of the first two and last two groups, the rows of the outer ones
    const int m0 = in(M(qs.M), W_), m1 = n0 > 1 ? in(M(qs.M >> 10), W_) : m0;
    const int k0 = in(M(qe.M >> 10 * (nl - 1)), W_), k1 = nl > 1 ? in(M(qe.M >> 10 * (nl - 2)), W_) : k0;
    const int near = fx_group_start(1, n0, e0), size = L - sl - fx_group_start(nl - 1, nl, L - sl);
    auto lo = [&](int q) { return move(get(q), q < near ? m0 : m1); };          // row q
    auto hi = [&](int q) { return move(get(L - 1 - q), q < size ? k0 : k1); };  // row L-1-q
    const bool first = w == 0, last = w == S - 1;
    // sums of the start's and the end's rows 0 and 1
    i64 s0_ = 0, s1_ = 0, e0_ = 0, e1_ = 0, x = lo(0), y = hi(0);
    const int *c = et + 2 * 54;
    const Split wrap = split(y - x), back = split(x - y);
#pragma unroll 1
    for (int q = 0; q < 12; q += 2) {
      const int k = 2 * q;
      const I4 a0 = rd4(c + k), b0 = rd4(c + 24 + k), a1 = rd4(c + 48 + k), b1 = rd4(c + 72 + k);
      // rows q..q+2 from the start (n, u) and from the end (o, v); number 11 of the nearer end's is the step across
      const i64 xn = lo(q + 1), yn = hi(q + 1), xm = lo(q + 2), ym = hi(q + 2);
      const Split n = split(xn - x), o = split(yn - y), u = split(xm - xn), v = split(ym - yn);
      x = xm;
      y = ym;
      if (first) {
        const Split f = q == 10 ? wrap : u;
        Acc<> A(a0.x, a0.y, n), B(a1.x, a1.y, n);
        A.add(b0.x, b0.y, o);
        B.add(b1.x, b1.y, o);
        A.add(a0.z, a0.w, f);
        B.add(a1.z, a1.w, f);
        A.add(b0.z, b0.w, v);
        B.add(b1.z, b1.w, v);
        s0_ += A.value();
        s1_ += B.value();
      }
      if (last) {
        const Split f = q == 10 ? back : v;
        Acc<> A(a0.x, a0.y, o), B(a1.x, a1.y, o);
        A.add(b0.x, b0.y, n);
        B.add(b1.x, b1.y, n);
        A.add(a0.z, a0.w, f);
        B.add(a1.z, a1.w, f);
        A.add(b0.z, b0.w, u);
        B.add(b1.z, b1.w, u);
        e0_ += A.value();
        e1_ += B.value();
      }
    }
    auto times = [&](int at, i64 v) {
      const I2 k = rd2(et + 2 * at);
      return Acc<>(k.x, k.y, split(v)).value();
    };
    auto third = [&](int i, i64 x0, i64 x1, i64 x2, i64 x3, i64 x4, i64 x5, i64 x6) {
      const I2 t = rd2(rows + i * FX_RT + 4);
      return stencil(rd4(rows + i * FX_RT), t.x, t.y, x0, x1, x2, x3, x4, x5, x6).value();
    };
    if (first) {
      rs[0] = times(102, s0_);
      rs[1] = times(103, s1_);
      rs[2] = third(2, hi(1), lo(0), lo(1), lo(2), lo(3), lo(4), lo(5));
    }
    if (last) {
      tail[0] = times(104, e0_);
      tail[1] = times(105, e1_);
      tail[2] = third(L - 3, hi(5), hi(4), hi(3), hi(2), hi(1), hi(0), lo(1));
    }
  }
  ATI_HD static Acc<> stencil(I4 c0, int c1x, int c1y, i64 x0, i64 x1, i64 x2, i64 x3, i64 x4, i64 x5, i64 x6) {
    const i64 c = FILT ? x3 + x3 : 0;
    Acc<> q(c0.x, c0.y, split(FILT ? x4 + x2 - c : x4 - x2));
    q.add(c0.z, c0.w, split(FILT ? x5 + x1 - c : x5 - x1));
    q.add(c1x, c1y, split(FILT ? x6 + x0 - c : x6 - x0));
    return q;
  }

  // 4. forward elimination of the segment from zero incoming values, in place; its last two values
  ATI_HD Pair forward() {
    i64 u2 = 0, u1 = 0;
    int W_ = W0, i = s0;
    auto put = [&](i64 v) {
      set(i, v);
      u2 = u1;
      u1 = v;
      i++;
    };
    auto end_row = [&](i64 sb, int at) {
      const I2 c0 = rd2(et + 2 * at), c1 = rd2(et + 2 * at + 2);
      AccEnd A(c0.x, c0.y, split(u2));
      A.add(c1.x, c1.y, split(u1));
      put(sb + A.value());
    };
    const int in0 = w == 0 ? 4 : s0, ihi = imin(s1, L - 3);  // the inner rows
    u64 mp = sc.M, wp = Wp;
    int m = M(mp);  // the group's exponent
    if (!per && w == S - 1) {
      const int s = in(M(sc.M >> 10 * (ng - 1)), We);
      i64 p[7];
#pragma unroll
      for (int q = 0; q < 7; q++) p[q] = move(get(L - 1 - q), s);
      one_sided(1, p, tail);
    }
    i64 a3 = 0, a4 = 0, a5 = 0;
    auto window = [&](int r) {
      const int s = in(m, W_);
      a3 = move(get(r), s); a4 = move(get(r + 1), s); a5 = move(get(r + 2), s);
    };
    window(in0);
    if (w == 0) {
      const int s = in(m, W_);
      i64 p[7];
#pragma unroll
      for (int q = 0; q < 7; q++) p[q] = move(get(q), s);
      const i64 c = 2 * p[3];
      const I4 k = rd4(et + 2 * 150);
      const I2 k3 = rd2(et + 2 * 152);
      auto d = [&](int q) { return split(FILT ? p[3 + q] + p[3 - q] - c : p[3 + q] - p[3 - q]); };
      AccEnd A(k.x, k.y, d(1));
      A.add(k.z, k.w, d(2));
      A.add(k3.x, k3.y, d(3));
      i64 sb[3];
      if (!per) one_sided(0, p, sb);
      end_row(per ? rs[0] : sb[0], 36);
      end_row(per ? rs[1] : sb[1], 38);
      end_row(per ? rs[2] : sb[2], 40);
      end_row(A.value(), 153);
    }
    // (a row's coefficients are loaded a row ahead: with most of the SM's memory taken by the tiles the tables come
    // from L2)
    const int *t = rows + in0 * FX_RT;
    I4 c0 = rd4(t), c1 = rd4(t + 4);
    I2 c2 = rd2(t + 8);
    i64 a0 = a[0], a1 = a[1], a2 = a[2];  // with a3.. the window, in units of the group
    auto inner = [&](i64 x6) {
      const I4 e0 = c0, e1 = c1;
      const I2 e2 = c2;
      t += FX_RT;
      c0 = rd4(t); c1 = rd4(t + 4); c2 = rd2(t + 8);
      Acc<> q = stencil(e0, e1.x, e1.y, a0, a1, a2, a3, a4, a5, x6);
      q.add(e1.z, e1.w, split(u2));
      q.add(e2.x, e2.y, split(u1));
      a0 = a1; a1 = a2; a2 = a3; a3 = a4; a4 = a5; a5 = x6;
      put(q.value());
    };
    Wp = 0;  // (from here on the last group's first)
    i64 r0 = 0, r1 = 0, r2 = 0;  // the group before's last three values
    for (int g = 0; g < ng; g++) {
      const bool last = g == ng - 1;
      const int g1 = end(g);
      if (g > 0) {
        const int most = last && w == S - 1 && !per ? fs.carry_end : fs.carry, mb = m;
        const int Wn = floor_W(imax(last ? We : W(wp), W_ + bits2(u2, u1) - most));
        mp >>= 10;
        m = M(mp);
        if (Wn != W_) {  // (else the window is in these units already)
          u2 = move(u2, W_ - Wn);
          u1 = move(u1, W_ - Wn);
          W_ = Wn;
          const int s = in(mb, W_);
          a0 = move(r0, s); a1 = move(r1, s); a2 = move(r2, s);
          window(i);
        }
      }
      wp >>= 10;
      push_front(Wp, put_W(W_));
      if (!last) { r0 = get(g1 - 3); r1 = get(g1 - 2); r2 = get(g1 - 1); }
      const int so = in(m, W_), sl = imax(so, 0), sr = imax(-so, 0), sn = in(last ? Mn : M(mp >> 10), W_);
      const int e = imin(g1 - 3, ihi);
      if (e - i == FX_GR - 3) {
#pragma unroll
        for (int q = 0; q < FX_GR - 3; q++) inner(shr(shl(get(i + 3), sl), sr));
      } else {
#pragma unroll 4
        while (i < e) inner(shr(shl(get(i + 3), sl), sr));
      }
      if (last && w == S - 1) {
        const int d = We - W_;
        end_row(move(tail[2], d), 46);
        end_row(move(tail[1], d), 44);
        end_row(move(tail[0], d), 42);
      } else {  // windows reaching into the next group
#pragma unroll
        for (int q = 0; q < 3; q++) inner(move(last ? tail[q] : get(i + 3), sn));
      }
    }
    return {u2, u1, W_};
  }

  // 5. back substitution of the segment's own forward values from zero values beyond its end; emit(row, value, W); its
  // first two values
  template <class E>
  ATI_HD Pair backward(E &&emit) {
    i64 q1 = 0, q2 = 0;
    int W_ = NONE;
    const int *t = rows + (s1 - 1) * FX_RT + 12;
    I4 cn = rd4(t);
    u64 wp = Wp;
    Wp = 0;  // (the first group's first)
    for (int g = ng - 1; g >= 0; g--) {
      const int Wu = W(wp), i0 = first(g);
      wp >>= 10;
      const int Wn = g == ng - 1 ? Wu : imax(Wu, W_ + bits2(q1, q2) - fs.carry);
      if (Wn != W_) {
        q1 = move(q1, W_ - Wn);
        q2 = move(q2, W_ - Wn);
        W_ = Wn;
      }
      const int d = W_ - Wu;
      push_front(Wp, put_W(W_));
      int i = end(g) - 1;
      const int ib = imax(i0, 3);
      auto row = [&](I4 k, int r) {
        Acc<> A(k.z, k.w, split(q2));
        A.add(k.x, k.y, split(q1));
        const i64 q = shr(get(r), d) + A.value();
        emit(r, q, W_);
        q2 = q1;
        q1 = q;
      };
#pragma unroll 4
      for (; i >= ib; i--) {
        const I4 c = cn;
        t -= FX_RT;
        cn = rd4(t);
        row(c, i);
      }
      for (; i >= i0; i--) {
        const I2 c0 = rd2(et + 2 * (48 + 2 * i)), c1 = rd2(et + 2 * (49 + 2 * i));
        AccEnd A(c0.x, c0.y, split(q1));
        A.add(c1.x, c1.y, split(q2));
        const i64 q = shr(get(i), d) + A.value();
        emit(i, q, W_);
        q2 = q1;
        q1 = q;
      }
    }
    return {q1, q2, W_};
  }
  // ... with the incoming forward values x (rows s0, s0+1)
  ATI_HD Pair with_incoming(Pair c, Pair x) const {
    const int *t = rows + s0 * FX_RT;
    const I4 r0 = rd4(t + 16), r1 = rd4(t + FX_RT + 16);
    const Split x2 = split(x.a), x1 = split(x.b);
    Acc<> A(r0.x, r0.y, x2), B(r1.x, r1.y, x2);
    A.add(r0.z, r0.w, x1);
    B.add(r1.z, r1.w, x1);
    return sum(c, {A.value(), B.value(), x.W - (int)(short)t[10]});
  }

  // 6. results: emit(row, value, W)
  template <class E>
  ATI_HD void results(Pair x, Pair y, E &&emit) {
    const int *t = rows + s0 * FX_RT;
    I4 rn = rd4(t + 16), gn = rd4(t + 20);
    int i = s0;
    for (int g = 0; g < ng; g++) {
      const int word = t[10], last = end(g), Wb = W(Wp);
      Wp >>= 10;
      const int wx = x.W - (int)(short)word, wy = y.W - (word >> 16);
      const int Wo = imax(Wb + 1, imax(wx, wy)), d = Wo - Wb;
      const Split x2 = split(shr(x.a, Wo - wx)), x1 = split(shr(x.b, Wo - wx));
      const Split y1 = split(shr(y.a, Wo - wy)), y2 = split(shr(y.b, Wo - wy));
      auto row = [&](I4 r, I4 q, int k) {
        Acc<> A(r.x, r.y, x2);
        A.add(r.z, r.w, x1);
        A.add(q.x, q.y, y1);
        A.add(q.z, q.w, y2);
        emit(k, shr(get(k), d) + A.value(), Wo);
      };
#pragma unroll 4
      for (; i < last; i++) {
        const I4 r = rn, q = gn;
        t += FX_RT;
        rn = rd4(t + 16);
        gn = rd4(t + 20);
        row(r, q, i);
      }
    }
  }
};

}  // namespace fxl
}  // namespace ati
