// ati_fixed_tab.cpp — tables of the fixed-point line sweeps (see ati_fixed_tab.h, ati_fixed_line.h).
#include "ati_fixed_tab.h"

#include <algorithm>
#include <cmath>
#include <cstring>

#include "ati_scheme.h"

namespace ati {
namespace {

constexpr double kAlpha = 0.5862704032801503, kBeta = 0.09549533555017055;

// the operator's interior stencil and the LU factors of a line
void stencil_of(const SchemeHost &H, bool filt, double ks[3]) {
  const Scheme &S = H.s;
  ks[0] = filt ? S.fa : S.aa;
  ks[1] = filt ? S.fb : S.ab;
  ks[2] = filt ? S.fc : S.ac;
}
std::vector<double> factors_of(const SchemeHost &H, bool filt, int L, bool per) {
  std::vector<double> fc((size_t)L * 5);
  const auto &al = filt ? H.albef : H.albed;
  penta_factors(al[per], al[per], filt ? H.alphf : kAlpha, filt ? H.betf : kBeta, L, fc.data());
  return fc;
}

// right-hand-side rows 0-2 of a line end as weights on its first seven points (one-sided ends)
void end_weights(const Scheme &S, bool filt, double E[3][7]) {
  std::memset(E, 0, sizeof(double) * 21);
  if (!filt) {
    for (int r = 0; r < 3; r++)
      for (int q = 0, n = 0; q < 7; q++) {
        if (q == r) continue;
        E[r][q] += S.abc[r][n];
        E[r][r] -= S.abc[r][n];
        n++;
      }
    return;
  }
  // the extrapolated points rv(n) = w0 - ffx(n) sum_q fex(q) (w(q) - w0) of src/Subroutines3D.f90:160-170
  double rv[4][7];
  std::memset(rv, 0, sizeof(rv));
  for (int n = 1; n <= 3; n++) {
    rv[n][0] = 1.0;
    for (int q = 1; q <= 3; q++) {
      rv[n][q] -= S.ffx[n] * S.fex[q];
      rv[n][0] += S.ffx[n] * S.fex[q];
    }
  }
  auto pt = [&](int r, double c, int at) {  // c times point at of the line (negative: extrapolated)
    if (at >= 0) E[r][at] += c;
    else
      for (int q = 0; q < 7; q++) E[r][q] += c * rv[-at][q];
  };
  for (int r = 0; r < 3; r++) {
    const double c[3] = {S.fam[r], S.fbm[r], S.fcm[r]};
    for (int d = 1; d <= 3; d++) {
      pt(r, c[d - 1], r - d);
      pt(r, c[d - 1], r + d);
      pt(r, -2.0 * c[d - 1], r);
    }
  }
}

// the recurrences' coefficients of row i
struct Rows {
  const double *f;
  int L;
  double c2(int i) const { return f[i * 5 + 2]; }
  double m0(int i) const { return i >= 2 ? -c2(i) * f[i * 5] / c2(i - 2) : 0.0; }
  double m1(int i) const { return i >= 1 ? -c2(i) * f[i * 5 + 1] / c2(i - 1) : 0.0; }
  double n1(int i) const { return i <= L - 2 ? -f[i * 5 + 3] : 0.0; }
  double n2(int i) const { return i <= L - 3 ? -f[i * 5 + 4] : 0.0; }
};

// the largest value of a row with weights c over all lines whose neighbours differ by at most 1 (on a periodic line also
// across its ends): the sum of the magnitudes of the weights on the differences
double amplitude(const std::vector<double> &c, bool per) {
  const int L = (int)c.size();
  double best = 0, s = 0;
  for (int j = L - 1; j >= 1; j--) best += std::fabs(s += c[j]);
  if (!per) return best;
  // points up to m reached from point 0, the others from the far end (any m bounds the row; three are tried)
  for (int m = L / 4; m < L - 1; m += L / 4) {
    double t = 0, v = 0;
    for (int j = m; j >= 1; j--) t += std::fabs(v += c[j]);
    v = 0;
    for (int j = m + 1; j < L - 1; j++) t += std::fabs(v += c[j]);
    best = std::min(best, t + std::fabs(v + c[L - 1]));
  }
  return best;
}

// the power of two that brings the largest of n numbers to [1/2, 1)
int to_one(const double *v, int n) {
  double m = 0;
  for (int q = 0; q < n; q++) m = std::max(m, std::fabs(v[q]));
  int e = 0;
  std::frexp(m, &e);
  return m > 0 ? std::min(std::max(-e, -30), 1000) : 0;
}

}  // namespace

FixBounds fix_bounds(const SchemeHost &H, bool filt, int L, bool per) {
  const Scheme &S = H.s;
  double ks[3], E[3][7];
  stencil_of(H, filt, ks);
  end_weights(S, filt, E);
  const std::vector<double> fc = factors_of(H, filt, L, per);
  const Rows F{fc.data(), L};
  std::vector<std::vector<double>> R(L, std::vector<double>(L, 0.0));
  for (int i = 0; i < L; i++) {
    auto &r = R[i];
    const int e = i < 3 ? i : (i > L - 4 ? L - 1 - i : -1);
    const double sg = !filt && i > 2 ? -1.0 : 1.0;  // a derivative changes sign under reflection
    auto at = [&](int q) -> double & { return r[i < 3 ? q : L - 1 - q]; };
    if (e < 0) {
      for (int d = 1; d <= 3; d++) {
        r[i + d] += ks[d - 1];
        r[i - d] += filt ? ks[d - 1] : -ks[d - 1];
        if (filt) r[i] -= 2 * ks[d - 1];
      }
    } else if (per && e < 2) {
      for (int q = 0; q <= LMD; q++) {
        at(q) += sg * S.pbci[0][e][q];
        at(L - 2 - q) += sg * S.pbco[0][e][q];
      }
    } else if (per) {
      at(3) += sg * ks[0]; at(1) -= sg * ks[0]; at(4) += sg * ks[1]; at(0) -= sg * ks[1];
      at(5) += sg * ks[2]; at(L - 2) -= sg * ks[2];
    } else {
      for (int q = 0; q < 7; q++) at(q) += sg * E[e][q];
    }
    for (double &v : r) v *= F.c2(i);
  }
  FixBounds out;
  const int nseg = seg_count(L);
  for (int k = 0; k < nseg; k++) {
    const int s0 = seg_start(k, L, nseg), s1 = seg_start(k + 1, L, nseg), ng = fx_groups(s1 - s0);
    for (int g = 0; g < ng; g++) {
      const int a = s0 + fx_group_start(g, ng, s1 - s0), b = s0 + fx_group_start(g + 1, ng, s1 - s0), n = b - a;
      std::vector<std::vector<double>> U(n + 2, std::vector<double>(L, 0.0));
      // responses to u(a-2) = 1, u(a-1) = 1, b(b) = 1, b(b+1) = 1
      std::vector<double> p(n + 2, 0.0), q(n + 2, 0.0), x(n + 2, 0.0), y(n + 2, 0.0);
      double p2 = k + g > 0, p1 = 0, q2 = 0, q1 = k + g > 0;
      const int z = b == L;
      auto top = [](double &m, double v) { m = std::max(m, v); };
      for (int i = a; i < b; i++) {
        const int r = i - a;
        const double m0 = F.m0(i), m1 = F.m1(i);
        p[r] = m0 * p2 + m1 * p1;
        q[r] = m0 * q2 + m1 * q1;
        p2 = p1; p1 = p[r]; q2 = q1; q1 = q[r];
        for (int j = 0; j < L; j++) U[r][j] = R[i][j] + (r >= 2 ? m0 * U[r - 2][j] : 0) + (r >= 1 ? m1 * U[r - 1][j] : 0);
        const double v = amplitude(U[r], per);
        top(out.forward[z], v);
        if (i >= 2 && i <= L - 5) top(out.inner[z], v);
        top(out.forward_carry[z], std::fabs(p[r]) + std::fabs(q[r]));
      }
      x[n] = y[n + 1] = b < L;
      for (int i = b - 1; i >= a; i--) {
        const int r = i - a;
        const double n1 = F.n1(i), n2 = F.n2(i);
        for (auto *V : {&p, &q, &x, &y}) (*V)[r] += n1 * (*V)[r + 1] + n2 * (*V)[r + 2];
        for (int j = 0; j < L; j++) U[r][j] += n1 * U[r + 1][j] + n2 * U[r + 2][j];
        top(out.backward[z], amplitude(U[r], per));
        top(out.backward_carry[z], std::fabs(p[r]) + std::fabs(q[r]) + std::fabs(x[r]) + std::fabs(y[r]));
      }
    }
  }
  return out;
}

bool fix_line(const SchemeHost &H, const FixOp &op, bool filt, int L, bool per, const double *fac, int *o, int *e) {
  const Scheme &S = H.s;
  double ks[3], E[3][7];
  stencil_of(H, filt, ks);
  end_weights(S, filt, E);
  const Rows F{fac, L};
  const double sc = (double)(1 << op.k), g32 = std::ldexp(1.0, op.gbits - 32), limit = 8.9e18;
  // a coefficient of a value of up to x largest differences; mid: its group's largest middle sum so far
  auto pairc = [&](double c, int *p, double x, double &mid, int bits = FX_BITS) {
    if (!(std::ldexp(std::fabs(c), bits) < 2147483000.0)) return false;
    const double hi = std::nearbyint(std::ldexp(c, bits));
    const double lo = std::min(std::nearbyint(std::ldexp(std::ldexp(c, bits) - hi, 32)), 2147483647.0);
    p[0] = (int)hi;
    p[1] = (int)lo;
    mid += std::fabs(hi) * 2147483648.0 + std::fabs(lo) * (x * g32 + 1.0);
    return mid < limit;
  };
  const double carry = std::ldexp(1.0, FX_CARRY - op.gbits);
  bool fits = true;
  for (int i = 0; i < L; i++) {
    int *r = o + (size_t)i * FX_RT;
    double f = 0, b = 0;
    if ((i >= 4 && i <= L - 4) || per) {
      for (int q = 0; q < 3; q++) fits = fits && pairc(F.c2(i) * ks[q] * sc, r + 2 * q, 2.0 * (q + 1), f);
      if (i >= 4 && i <= L - 4) fits = fits && pairc(F.m0(i), r + 6, op.vinner, f) && pairc(F.m1(i), r + 8, op.vinner, f);
    }
    if (i >= 3) fits = fits && pairc(F.n1(i), r + 12, op.vback, b) && pairc(F.n2(i), r + 14, op.vback, b);
  }
  const int nseg = seg_count(L);
  std::vector<double> R, T, G, W;
  for (int k = 0; k < nseg; k++) {  // segment responses
    const int s0 = seg_start(k, L, nseg), s1 = seg_start(k + 1, L, nseg), n = s1 - s0, ng = fx_groups(n);
    for (auto *V : {&R, &T, &G, &W}) V->assign(n + 2, 0.0);
    if (k > 0) {
      double g2 = 1, g1 = 0, h2 = 0, h1 = 1;
      for (int i = s0; i < s1; i++) {
        R[i - s0] = F.m0(i) * g2 + F.m1(i) * g1;
        T[i - s0] = F.m0(i) * h2 + F.m1(i) * h1;
        g2 = g1; g1 = R[i - s0]; h2 = h1; h1 = T[i - s0];
      }
      const double v[4] = {g2, h2, g1, h1};
      const int ex = to_one(v, 4);
      double mid[2] = {0, 0};
      for (int q = 0; q < 4; q++)
        fits = fits && pairc(std::ldexp(v[q], ex), o + (size_t)(s1 - 2 + q / 2) * FX_RT + 24 + 2 * (q % 2), carry, mid[q / 2]);
      o[(size_t)(s1 - 1) * FX_RT + 11] = ex;
    }
    if (k < nseg - 1) G[n] = W[n + 1] = 1.0;
    for (int q = n - 1; q >= 0; q--)
      for (auto *V : {&R, &T, &G, &W}) (*V)[q] += F.n1(s0 + q) * (*V)[q + 1] + F.n2(s0 + q) * (*V)[q + 2];
    for (int g = 0; g < ng; g++) {
      const int a = fx_group_start(g, ng, n), b = fx_group_start(g + 1, ng, n);
      const int ex = std::min(to_one(&R[a], b - a), to_one(&T[a], b - a)), ey = std::min(to_one(&G[a], b - a), to_one(&W[a], b - a));
      for (int q = a; q < b; q++) {
        int *r = o + (size_t)(s0 + q) * FX_RT;
        double mid = 0;
        fits = fits && pairc(std::ldexp(R[q], ex), r + 16, carry, mid) && pairc(std::ldexp(T[q], ex), r + 18, carry, mid) &&
               pairc(std::ldexp(G[q], ey), r + 20, carry, mid) && pairc(std::ldexp(W[q], ey), r + 22, carry, mid);
        r[10] = (int)((unsigned)ey << 16 | ((unsigned)ex & 0xffffu));
      }
    }
  }
  const double sg = filt ? 1.0 : -1.0;
  auto endc = [&](double c, int at, double x, double &mid) { return pairc(c, e + 2 * at, x, mid, FX_END_BITS); };
  for (int r = 0; r < 3; r++) {
    double ms = 0, me = 0, f = 0, g = 0, b = 0;
    for (int q = 0, n = 0; q < 7; q++) {
      if (q == r) continue;
      const double x = std::abs(q - r);
      fits = fits && endc(F.c2(r) * E[r][q] * sc, 6 * r + n, x, ms) &&
             endc(sg * F.c2(L - 1 - r) * E[r][q] * sc, 18 + 6 * r + n, x, me);
      n++;
    }
    fits = fits && endc(F.m0(r), 36 + 2 * r, op.vfwd, f) && endc(F.m1(r), 37 + 2 * r, op.vfwd, f);
    fits = fits && endc(F.m0(L - 1 - r), 42 + 2 * r, op.vfwd, g) && endc(F.m1(L - 1 - r), 43 + 2 * r, op.vfwd, g);
    fits = fits && endc(F.n1(r), 48 + 2 * r, op.vback, b) && endc(F.n2(r), 49 + 2 * r, op.vback, b);
  }
  // row 3: next to one-sided rows its c2 is large
  double m3 = 0, f3 = 0;
  for (int q = 0; q < 3; q++) fits = fits && endc(F.c2(3) * ks[q] * sc, 150 + q, 2.0 * (q + 1), m3);
  fits = fits && endc(F.m0(3), 153, op.vfwd, f3) && endc(F.m1(3), 154, op.vfwd, f3);
  for (int r = 0; r < 2 && per; r++) {
    // weights on f(q) - f(0) and f(L-2-q) - f(0) as weights on the neighbour differences
    double w[24] = {0};
    constexpr double big = 2.0;  // (the sums' own rounding, before their last product)
    for (int q = 0; q <= LMD; q++) {
      for (int j = 0; j < q; j++) w[j] += big * S.pbci[0][r][q];
      w[11] += big * S.pbco[0][r][q];
      for (int j = 0; j <= q; j++) w[12 + j] += big * S.pbco[0][r][q];
    }
    double sum = 0;
    for (int q = 0; q < 12; q += 2) {
      double mid = 0;
      for (int u = q; u < q + 2; u++) {  // (summed two rows of both ends at a time)
        fits = fits && pairc(w[u], e + 2 * (54 + 24 * r + u), u == 11 ? 12.0 : 1.0, mid) &&
               pairc(w[12 + u], e + 2 * (54 + 24 * r + 12 + u), 1.0, mid);
        sum += std::fabs(w[u]) + std::fabs(w[12 + u]);
      }
    }
    double mid[2] = {0, 0};
    fits = fits && pairc(F.c2(r) * sc / big, e + 2 * (102 + r), sum, mid[0]) &&
           pairc(-F.c2(L - 1 - r) * sc / big, e + 2 * (104 + r), sum, mid[1]);
  }
  return fits;
}

FixOp fix_operator(const SchemeHost &H, bool filt) {
  // the lines that the bounds and the sums are checked on: every cut into groups, one to five segments, both kinds
  struct Line {
    int L;
    bool per;
    std::vector<double> fac;
  };
  std::vector<Line> lines;
  auto line = [&](int L) {
    for (int per = 0; per <= (filt ? 0 : 1); per++) lines.push_back({L, per != 0, factors_of(H, filt, L, per != 0)});
  };
  for (int L = FX_LMIN; L <= 31; L++) line(L);
  for (int L : {48, 49, 50, 57, 63, 97, 120}) line(L);
  FixBounds B;
  for (const Line &l : lines) {
    const FixBounds b = fix_bounds(H, filt, l.L, l.per);
    for (int z = 0; z < 2; z++) {
      const int y = l.per ? 0 : z;  // (a periodic line's last group is like the others)
      B.forward[y] = std::max(B.forward[y], b.forward[z]);
      B.inner[y] = std::max(B.inner[y], b.inner[z]);
      B.forward_carry[y] = std::max(B.forward_carry[y], b.forward_carry[z]);
      B.backward[y] = std::max(B.backward[y], b.backward[z]);
      B.backward_carry[y] = std::max(B.backward_carry[y], b.backward_carry[z]);
    }
  }
  FixOp op;
  // the extra scale: a small operator (the filter) uses the range a derivative would
  while (op.k < 8 && std::max(B.forward[0], B.backward[0]) * (2 << op.k) <= 14.0) op.k++;
  const double sc = 1.03125 * (1 << op.k);  // (other line lengths, rounding)
  auto fits = [&] {
    const double c = std::ldexp(1.0, op.carry - op.gbits), d = std::ldexp(1.0, -op.spare);
    const double ce = std::ldexp(1.0, op.carry_end - op.gbits), most = std::ldexp(0.93, 63 - op.gbits);
    op.vfwd = std::max(B.forward[0] * sc + B.forward_carry[0] * c, B.forward[1] * sc * d + B.forward_carry[1] * ce);
    op.vinner = std::max(B.inner[0] * sc + B.forward_carry[0] * c, B.inner[1] * sc * d + B.forward_carry[1] * ce);
    op.vback = std::max(B.backward[0] * sc + B.backward_carry[0] * c, B.backward[1] * sc * d + B.backward_carry[1] * ce);
    if (!(std::max(op.vfwd, op.vback) < most)) return false;
    std::vector<int> ro((size_t)lines.back().L * FX_RT), eo(2 * FX_ET);
    for (const Line &l : lines)
      if (!fix_line(H, op, filt, l.L, l.per, l.fac.data(), ro.data(), eo.data())) return false;
    return true;
  };
  // The unit's size sets the error, 2^-gbits of the differences that a group reads or 2^-carry of the values carried in,
  // which are some twice the differences where a line is smooth: first the smallest of both, then of the first.
  for (int unit = 59; unit >= 54; unit--)
    for (op.gbits = 60; op.gbits >= unit; op.gbits--)
      for (op.carry = 60; op.carry >= unit + 1; op.carry--)
        for (op.spare = 0; op.spare <= 2; op.spare++)
          for (op.carry_end = op.carry; op.carry_end >= unit; op.carry_end--)
            if (fits()) return op;
  return FixOp{};
}

}  // namespace ati
