// Errors of flux_point_fixed (csrc/ati_fixed_flux.h, compiled for the host) and of the FP64 flux arithmetic against
// extended precision.  Arguments: viscous, then log2 of the ratio of the largest to the smallest direction's metrics, of
// u to w, of the largest to the smallest velocity derivative, of p to the dynamic pressure scale, seed.  Output: for each
// of the fifteen components the root mean square error of the two, in units of the sum of the magnitudes of the terms the
// component at that point is made of, and their ratio.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "ati_fixed_flux.h"

#if defined(__x86_64__)
typedef __float128 quad;
#else
typedef long double quad;
#endif

using ati::FixFluxIn;

static quad mag(quad x) { return x < 0 ? -x : x; }
// F, and A: the same sums of magnitudes
static void exact(const FixFluxIn &I, bool visc, quad *F, quad *A) {
  quad c[4][3] = {}, t[3][3] = {}, w[3], C[4][3] = {}, T[3][3] = {}, W[3];
  if (visc) {
    for (int f = 0; f < 4; f++)
      for (int k = 0; k < 3; k++)
        for (int n = 0; n < 3; n++) {
          c[f][k] += (quad)I.m[n][k] * I.dv[f][n];
          C[f][k] += mag((quad)I.m[n][k] * I.dv[f][n]);
        }
    const quad div = c[0][0] + c[1][1] + c[2][2], Div = C[0][0] + C[1][1] + C[2][2];
    for (int a = 0; a < 3; a++)
      for (int b = 0; b < 3; b++) {
        t[a][b] = I.r1 * (a == b ? 2 * c[a][a] - 2 * div / 3 : c[a][b] + c[b][a]);
        T[a][b] = I.r1 * (a == b ? 2 * C[a][a] + 2 * Div / 3 : C[a][b] + C[b][a]);
      }
  }
  for (int k = 0; k < 3; k++) {
    w[k] = (quad)I.p * I.umf[k];
    W[k] = mag(w[k]);
    if (visc) {
      w[k] += I.r2 * c[3][k];
      W[k] += I.r2 * C[3][k];
      for (int j = 0; j < 3; j++) {
        w[k] += I.vel[j] * t[j][k];
        W[k] += mag(I.vel[j]) * T[j][k];
      }
    }
  }
  for (int n = 0; n < 3; n++) {
    quad s = 0, e = 0, S = 0, E = 0;
    for (int k = 0; k < 3; k++) {
      s += I.m[n][k] * ((quad)I.vel[k] + I.umf[k]);
      e += I.m[n][k] * w[k];
      S += mag(I.m[n][k] * ((quad)I.vel[k] + I.umf[k]));
      E += mag(I.m[n][k]) * W[k];
    }
    F[n] = I.q[0] * s;
    A[n] = I.q[0] * S;
    for (int m = 0; m < 3; m++) {
      quad x = I.q[1 + m] * s + (quad)I.m[n][m] * I.p;
      quad y = mag(I.q[1 + m]) * S + mag((quad)I.m[n][m] * I.p);
      for (int k = 0; k < 3; k++) {
        x -= I.m[n][k] * t[m][k];
        y += mag(I.m[n][k]) * T[m][k];
      }
      F[3 * (m + 1) + n] = x;
      A[3 * (m + 1) + n] = y;
    }
    F[12 + n] = ((quad)I.q[4] + I.p) * s - e;
    A[12 + n] = ((quad)I.q[4] + I.p) * S + E;
  }
}

// the FP64 kernels' operations (stress_point and flux_fast_point), products contracted as the compiler does
static double dot3(double a, double x, double b, double y, double c, double z) {
  return std::fma(c, z, std::fma(b, y, a * x));
}
static void fp64(const FixFluxIn &I, bool visc, double *F) {
  double c[4][3], t[9] = {0};
  if (visc) {
    for (int f = 0; f < 4; f++)
      for (int k = 0; k < 3; k++)
        c[f][k] = dot3(I.m[0][k], I.dv[f][0], I.m[1][k], I.dv[f][1], I.m[2][k], I.dv[f][2]);
    const double d5 = 2.0 / 3.0 * (c[0][0] + c[1][1] + c[2][2]);
    for (int k = 0; k < 3; k++) t[k] = I.r1 * std::fma(2.0, c[k][k], -d5);
    t[3] = I.r1 * (c[1][0] + c[0][1]);
    t[4] = I.r1 * (c[2][1] + c[1][2]);
    t[5] = I.r1 * (c[0][2] + c[2][0]);
    const double *u = I.vel;
    t[6] = std::fma(u[2], t[5], std::fma(u[1], t[3], std::fma(u[0], t[0], I.r2 * c[3][0])));
    t[7] = std::fma(u[2], t[4], std::fma(u[1], t[1], std::fma(u[0], t[3], I.r2 * c[3][1])));
    t[8] = std::fma(u[2], t[2], std::fma(u[1], t[4], std::fma(u[0], t[5], I.r2 * c[3][2])));
  }
  const int at[3][3] = {{0, 3, 5}, {3, 1, 4}, {5, 4, 2}};
  double V[3], w[3];
  for (int k = 0; k < 3; k++) {
    V[k] = I.vel[k] + I.umf[k];
    w[k] = visc ? std::fma(I.p, I.umf[k], t[6 + k]) : I.p * I.umf[k];
  }
  const double h = I.q[4] + I.p;
  for (int n = 0; n < 3; n++) {
    const double *M = I.m[n];
    const double s = dot3(M[0], V[0], M[1], V[1], M[2], V[2]);
    F[n] = I.q[0] * s;
    for (int m = 0; m < 3; m++) {
      if (visc) {
        double g[3];
        for (int k = 0; k < 3; k++) g[k] = k == m ? I.p - t[m] : -t[at[m][k]];
        F[3 * (m + 1) + n] = std::fma(M[2], g[2], std::fma(M[1], g[1], std::fma(M[0], g[0], I.q[1 + m] * s)));
      } else {
        F[3 * (m + 1) + n] = std::fma(M[m], I.p, I.q[1 + m] * s);
      }
    }
    F[12 + n] = std::fma(h, s, -dot3(M[0], w[0], M[1], w[1], M[2], w[2]));
  }
}

int main(int argc, char **argv) {
  if (argc != 7) return 2;
  const bool visc = atoi(argv[1]) != 0;
  const int rm = atoi(argv[2]), rw = atoi(argv[3]), rd = atoi(argv[4]), rp = atoi(argv[5]);
  std::mt19937_64 g(atoi(argv[6]));
  std::uniform_real_distribution<double> U(-1.0, 1.0);
  const int n = 20000;
  double sx[15] = {0}, sd[15] = {0};
  for (int it = 0; it < n; it++) {
    FixFluxIn I;
    // directions xi and zeta along x and z, eta across, as in a stretched layer next to a wall: each direction's metrics
    // of its own size, its own component the largest
    const double md[3] = {1.0, std::ldexp(1.0, rm), std::ldexp(1.0, rm / 2)};
    for (int d = 0; d < 3; d++)
      for (int k = 0; k < 3; k++) I.m[d][k] = md[d] * U(g) * (k == d ? 1.0 : 0.2);
    const double vs[3] = {0.3, 0.1, std::ldexp(0.3, -rw)};
    for (int k = 0; k < 3; k++) {
      I.vel[k] = vs[k] * U(g);
      I.umf[k] = k == 0 ? 0.24 : (k == 1 ? 0.01 * U(g) : 0.0);
    }
    const double ds[4] = {1.0, 0.3, std::ldexp(1.0, -rw), 1.0};
    for (int f = 0; f < 4; f++)
      for (int d = 0; d < 3; d++) I.dv[f][d] = 0.01 * ds[f] * U(g) * (d == 1 ? 1.0 : std::ldexp(1.0, -rd));
    const double rho = 1.0 + 0.1 * U(g);
    I.p = std::ldexp(1.0 / 1.4, rp) * (1.0 + 0.1 * U(g));
    I.q[0] = rho;
    double ke = 0;
    for (int k = 0; k < 3; k++) {
      I.q[1 + k] = rho * I.vel[k];
      ke += 0.5 * I.q[1 + k] * I.vel[k];
    }
    I.q[4] = I.p / 0.4 + ke;
    I.r1 = 1e-4 * (1.0 + 0.1 * U(g)) / md[1];
    I.r2 = 3.4 * I.r1;
    quad X[15], scale[15];
    double A[15], B[15];
    exact(I, visc, X, scale);
    if (!(visc ? ati::flux_point_fixed<true>(I, A) : ati::flux_point_fixed<false>(I, A))) return 3;
    fp64(I, visc, B);
    for (int c = 0; c < 15; c++) {
      const double ea = (double)((A[c] - X[c]) / scale[c]), eb = (double)((B[c] - X[c]) / scale[c]);
      sx[c] += ea * ea;
      sd[c] += eb * eb;
    }
  }
  for (int c = 0; c < 15; c++)
    printf("%d %.3e %.3e %.3f\n", c, std::sqrt(sx[c] / n), std::sqrt(sd[c] / n), std::sqrt(sx[c] / sd[c]));
  return 0;
}
