// Errors of the fixed-point line solve (csrc/ati_fixed_line.h, compiled for the host) and of the FP64 sweeps' arithmetic
// against extended precision.  Arguments: operator (0 derivative, 1 filter), periodic, points, kind of line, log2 of the
// kind's scale, number of lines, seed.  Output: the largest and the mean over the line's points of the ratio of the two
// root mean square errors over the lines, then the ratio over all points and lines, then the largest integer of the solve
// in bits (63: overflow).  Or "scales", operator, filter cut-off: the scales (0: left to FP64), and per line length the
// largest value that a group's rows can reach, in bits.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "ati_fixed_line.h"
#include "ati_scheme.h"

#if defined(__x86_64__)
typedef __float128 quad;
#else
typedef long double quad;
#endif
using namespace ati;

static SchemeHost H;

// LU factors and solve of the pentadiagonal rows in extended precision
template <class T>
static std::vector<T> solve(const std::vector<T> &rhs, bool filt, bool per) {
  const int L = (int)rhs.size();
  const auto &al = (filt ? H.albef : H.albed)[per];
  const T a = filt ? H.alphf : 0.5862704032801503, b = filt ? H.betf : 0.09549533555017055;
  std::vector<std::vector<T>> A(L, std::vector<T>(5, 0));
  std::vector<T> x = rhs;
  for (int i = 0; i < L; i++)
    for (int q = 0; q < 5; q++)
      A[i][q] = i < 3 ? (T)al[i][q] : (i > L - 4 ? (T)al[L - 1 - i][4 - q] : (q == 2 ? (T)1 : (q % 2 ? a : b)));
  for (int i = 0; i < L; i++)
    for (int d = 1; d <= 2 && i + d < L; d++) {
      const T m = A[i + d][2 - d] / A[i][2];
      for (int q = 0; q <= 2; q++) A[i + d][2 - d + q] -= m * A[i][2 + q];
      x[i + d] -= m * x[i];
    }
  for (int i = L - 1; i >= 0; i--) {
    for (int d = 1; d <= 2 && i + d < L; d++) x[i] -= A[i][2 + d] * x[i + d];
    x[i] /= A[i][2];
  }
  return x;
}

// right-hand sides of the three rows from either end and of inner rows, in T: the kernels' operations (line_ends)
template <class T>
static T fm(T a, T b, T c) { return a * b + c; }
static double fm(double a, double b, double c) { return std::fma(a, b, c); }
template <class T>
static void end_rows(const std::vector<double> &f, bool filt, bool per, bool far, T sb[3]) {
  const Scheme &S = H.s;
  const int L = (int)f.size();
  auto p = [&](int q) { return (T)f[far ? L - 1 - q : q]; };
  const T sg = far && !filt ? -1 : 1;
  if (per) {
    for (int r = 0; r < 2; r++) {
      T s = 0, o = 0;
      // (in extended precision on differences: the weights' sum, zero but for their own rounding, is left out)
      const T c = sizeof(T) > 8 ? p(0) : (T)0;
      for (int q = 0; q <= LMD; q++) s = fm((T)S.pbci[0][r][q], p(q) - c, s);
      for (int q = 0; q <= LMD; q++) o = fm((T)S.pbco[0][r][q], p(L - 2 - q) - c, o);
      sb[r] = sg * (s + o);
    }
    sb[2] = sg * fm((T)S.ac, p(5) - p(L - 2), fm((T)S.ab, p(4) - p(0), S.aa * (p(3) - p(1))));
  } else if (!filt) {
    for (int r = 0; r < 3; r++) {
      T s = 0;
      for (int q = 0, n = 0; q < 7; q++)
        if (q != r) s = fm((T)S.abc[r][n++], p(q) - p(r), s);
      sb[r] = sg * s;
    }
  } else {
    const T w0 = p(0), res = fm((T)S.fex[3], w0 - p(3), fm((T)S.fex[2], w0 - p(2), S.fex[1] * (w0 - p(1))));
    T w[7];
    for (int q = 0; q < 4; q++) w[3 + q] = p(q);
    for (int q = 1; q <= 3; q++) w[3 - q] = fm(res, (T)S.ffx[q], w0);
    auto at = [&](int i) { return i > 3 ? p(i) : w[3 + i]; };
    for (int r = 0; r < 3; r++) {
      const T ra = 2 * p(r);
      sb[r] = fm((T)S.fcm[r], at(r + 3) + at(r - 3) - ra,
                 fm((T)S.fbm[r], at(r + 2) + at(r - 2) - ra, S.fam[r] * (at(r + 1) + at(r - 1) - ra)));
    }
  }
}

static std::vector<quad> exact(const std::vector<double> &f, bool filt, bool per) {
  const Scheme &S = H.s;
  const int L = (int)f.size();
  std::vector<quad> r(L);
  quad s[3], e[3];
  end_rows<quad>(f, filt, per, false, s);
  end_rows<quad>(f, filt, per, true, e);
  for (int i = 0; i < L; i++) {
    if (i < 3) r[i] = s[i];
    else if (i > L - 4) r[i] = e[L - 1 - i];
    else if (filt)
      r[i] = S.fa * ((quad)f[i - 1] + f[i + 1] - 2 * (quad)f[i]) + S.fb * ((quad)f[i - 2] + f[i + 2] - 2 * (quad)f[i]) +
             S.fc * ((quad)f[i - 3] + f[i + 3] - 2 * (quad)f[i]);
    else r[i] = S.aa * ((quad)f[i + 1] - f[i - 1]) + S.ab * ((quad)f[i + 2] - f[i - 2]) + S.ac * ((quad)f[i + 3] - f[i - 3]);
  }
  return solve<quad>(r, filt, per);
}

// the FP64 fast path's sweeps: scaled-factor rows, products contracted
static std::vector<double> fp64(const std::vector<double> &f, const std::vector<double> &fac, bool filt, bool per) {
  const Scheme &S = H.s;
  const int L = (int)f.size();
  std::vector<double> u(L);
  double s[3], e[3];
  end_rows<double>(f, filt, per, false, s);
  end_rows<double>(f, filt, per, true, e);
  auto c2 = [&](int i) { return fac[i * 5 + 2]; };
  for (int i = 0; i < L; i++) {
    const double l0 = i >= 2 ? c2(i) * fac[i * 5] / c2(i - 2) : 0, l1 = i >= 1 ? c2(i) * fac[i * 5 + 1] / c2(i - 1) : 0;
    const double A = c2(i) * (filt ? S.fa : S.aa), B = c2(i) * (filt ? S.fb : S.ab), C = c2(i) * (filt ? S.fc : S.ac);
    double sb;
    if (i < 3) sb = c2(i) * s[i];
    else if (i > L - 4) sb = c2(i) * e[L - 1 - i];
    else if (!filt) sb = std::fma(C, f[i + 3] - f[i - 3], std::fma(B, f[i + 2] - f[i - 2], A * (f[i + 1] - f[i - 1])));
    else
      sb = std::fma(-2 * (A + B + C), f[i],
                    std::fma(C, f[i + 3] + f[i - 3], std::fma(B, f[i + 2] + f[i - 2], A * (f[i + 1] + f[i - 1]))));
    u[i] = std::fma(-l1, i >= 1 ? u[i - 1] : 0, std::fma(-l0, i >= 2 ? u[i - 2] : 0, sb));
  }
  for (int i = L - 2; i >= 0; i--) {
    u[i] = std::fma(-fac[i * 5 + 3], u[i + 1], u[i]);
    if (i + 2 < L) u[i] = std::fma(-fac[i * 5 + 4], u[i + 2], u[i]);
  }
  return u;
}

static long long worst = 0;
static void note(long long v) { worst = std::max(worst, v < 0 ? ~v : v); }

template <bool FILT>
static std::vector<double> fixed(const std::vector<double> &f, const std::vector<int> &rows, const std::vector<int> &ends,
                                 const FixScale &fs, bool per) {
  using Seg = fxl::Segment<FILT, !FILT, 1>;
  const int L = (int)f.size(), S = seg_count(L);
  std::vector<double> col = f, out(L);
  std::vector<Seg> seg;
  for (int w = 0; w < S; w++) seg.emplace_back(rows.data() + FX_PAD * FX_RT, ends.data(), col.data(), L, S, w, per, fs);
  unsigned mx = 0;
  for (auto &s : seg) mx = std::max(mx, s.maxima());
  for (auto &s : seg) s.convert(mx);
  for (auto &s : seg) s.reads([&](int w) { return seg[w].sc; });
  std::vector<fxl::Pair> c(S), x(S), y(S);
  for (int w = 0; w < S; w++) c[w] = seg[w].forward();
  for (int i = 0; i < L; i++) note(seg[0].get(i));
  const int *rw = rows.data() + FX_PAD * FX_RT;
  x[0] = y[S - 1] = {0, 0, fxl::NONE};
  for (int w = 1; w < S; w++) x[w] = fxl::carry_forward(rw, seg_start(w, L, S), c[w - 1], x[w - 1]);
  for (int w = 0; w < S; w++) {
    c[w] = seg[w].backward([&](int i, long long v, int) { seg[w].set(i, v); note(v); });
    c[w] = seg[w].with_incoming(c[w], x[w]);
  }
  for (int w = S - 2; w >= 0; w--) y[w] = fxl::carry_backward(rw, seg_start(w + 1, L, S), c[w + 1], y[w + 1]);
  for (auto &s : seg)
    s.results(x[s.w], y[s.w], [&](int i, long long v, int W) {
      note(v);
      out[i] = s.bad ? NAN : (s.pre ? std::ldexp((double)v, s.out(W)) : fxl::from_fixed(v, s.out(W) * (1 << 20)));
    });
  return out;
}

static int scales(bool filt, double fltk) {
  ati_config_t cfg{};
  cfg.fltk = cfg.fltkbc = fltk;
  build_scheme(cfg, H);
  const FixOp op = fix_operator(H, filt);
  printf("%d %d %d %d %d\n", op.gbits, op.k, op.carry, op.spare, op.carry_end);
  for (int L : {13, 15, 16, 22, 49, 97, 241, 800})
    for (int per = 0; per <= (filt ? 0 : 1) && op.gbits; per++) {
      const FixBounds b = fix_bounds(H, filt, L, per != 0);
      double top = 0;
      for (int z = 0; z < 2; z++) {
        const bool end = z && !per;  // an open line's last group
        const double sc = std::ldexp(1.0, op.gbits + op.k - (end ? op.spare : 0)), c = std::ldexp(1.0, end ? op.carry_end : op.carry);
        top = std::max({top, b.forward[z] * sc + b.forward_carry[z] * c, b.backward[z] * sc + b.backward_carry[z] * c});
      }
      printf("%d %d %.4f\n", L, per, std::log2(top));
    }
  return 0;
}

int main(int argc, char **argv) {
  if (argc == 4 && !std::strcmp(argv[1], "scales")) return scales(atoi(argv[2]) != 0, atof(argv[3]));
  if (argc < 8) return 2;
  const bool filt = atoi(argv[1]) != 0, per = atoi(argv[2]) != 0;
  const int L = atoi(argv[3]), kind = atoi(argv[4]), scale = atoi(argv[5]), n = atoi(argv[6]);
  ati_config_t cfg{};
  cfg.fltk = argc > 8 ? atof(argv[8]) : 0.85;
  cfg.fltkbc = cfg.fltk;
  build_scheme(cfg, H);
  const FixOp op = fix_operator(H, filt);
  if (!op.gbits) return 3;
  std::vector<double> fac((size_t)L * 5);
  const auto &al = filt ? H.albef : H.albed;
  penta_factors(al[per], al[per], filt ? H.alphf : 0.5862704032801503, filt ? H.betf : 0.09549533555017055, L, fac.data());
  std::vector<int> rows((size_t)(L + 2 * FX_PAD) * FX_RT, 0), ends(2 * FX_ET, 0);
  if (!fix_line(H, op, filt, L, per, fac.data(), rows.data() + FX_PAD * FX_RT, ends.data())) return 4;
  std::mt19937_64 g(atoi(argv[7]));
  std::uniform_real_distribution<double> U(-1.0, 1.0);
  std::vector<double> sx(L, 0), sd(L, 0), f(L);
  for (int it = 0; it < n; it++) {
    const double ph = 3.2 * U(g), ph2 = 3.2 * U(g), k1 = 1 + (int)(3 * std::fabs(U(g))), amp = 1 + 0.5 * U(g);
    const double w = 6.283185307179586 / (L - 1), small = std::ldexp(1.0, -scale);
    const int at = (int)((L - 1) * (0.5 + 0.3 * U(g)));
    for (int i = 0; i < L; i++) {
      const double wave = std::sin(k1 * w * i + ph) + 0.3 * std::sin(3 * w * i + ph2);
      switch (kind) {
        case 0: f[i] = std::ldexp(1.0 + 0.01 * wave, scale); break;                        // a smooth field of one size
        case 1: f[i] = std::ldexp(wave, scale); break;                                     // ... through zero
        case 2: f[i] = amp * std::exp2(-scale * i * (1.0 / (L - 1))) * (1 + 0.2 * wave); break;  // falling along the line
        case 3: f[i] = amp * std::exp2(-scale * (L - 1 - i) * (1.0 / (L - 1))) * (1 + 0.2 * wave); break;  // rising
        case 4: f[i] = amp * std::tanh((i - at) / 4.0) + small * wave; break;              // a layer beside a small wave
        case 5: f[i] = small * wave * (i == at ? 1.0 / small : 1.0); break;                // one large value
        case 6: f[i] = std::ldexp(U(g), scale); break;                                     // rough
        case 7: f[i] = U(g) * std::exp2(-scale * std::fabs(U(g))); break;                  // rough, of all sizes
        case 8: f[i] = (i & 1 ? 1 : -1) * std::ldexp(1.0, -scale * (i / 8 % 2)); break;    // steps as large as the values
        case 9: f[i] = i < at ? 1.0 : small * U(g); break;                                 // a jump to a quiet part
        case 10: {  // falling to both sides of a point, round the line's ends
          const int d = std::abs(i - at);
          f[i] = amp * std::exp2(-2.0 * scale * std::min(d, L - 1 - d) / (L - 1)) * (1 + 0.2 * wave);
          break;
        }
        default: f[i] = std::ldexp(1.0, scale); break;                                     // constant
      }
    }
    const std::vector<quad> X = exact(f, filt, per);
    const std::vector<double> A = filt ? fixed<true>(f, rows, ends, op, per) : fixed<false>(f, rows, ends, op, per);
    const std::vector<double> B = fp64(f, fac, filt, per);
    for (int i = 0; i < L; i++) {
      const double a = (double)(A[i] - X[i]), b = (double)(B[i] - X[i]);
      sx[i] += a * a;
      sd[i] += b * b;
    }
    if (getenv("DUMP") && it == 0)
      for (int i = 0; i < L; i++) printf("%d %.17g %.6g %.3g %.3g\n", i, f[i], (double)X[i], A[i] - (double)X[i], B[i] - (double)X[i]);
  }
  double top = 0, mean = 0, px = 0, pd = 0;
  int m = 0;
  for (int i = 0; i < L; i++) {
    px += sx[i];
    pd += sd[i];
    if (sd[i] == 0 && sx[i] == 0) continue;
    const double r = std::sqrt(sx[i] / sd[i]);
    if (getenv("ROWS")) printf("row %d %.3e %.3e %.2f\n", i, std::sqrt(sx[i] / n), std::sqrt(sd[i] / n), r);
    top = std::max(top, r);
    mean += r;
    m++;
  }
  int bits = 0;
  while (bits < 63 && (worst >> bits)) bits++;
  printf("%.3f %.3f %.3f %d\n", top, m ? mean / m : 0.0, pd > 0 ? std::sqrt(px / pd) : 0.0, bits);
  return 0;
}
