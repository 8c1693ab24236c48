// The float64 collision in fixed point (csrc/sw_f64.cuh), compiled for the host, and the same
// collision in long double, for tests/test_f64_fixed.py.
#include "sw_f64.cuh"

namespace {
const int C[19][3] = {{0, 0, 0}, {1, 0, 0}, {-1, 0, 0}, {0, 1, 0}, {0, -1, 0}, {0, 0, 1}, {0, 0, -1},
                      {1, 1, 0}, {-1, -1, 0}, {1, -1, 0}, {-1, 1, 0}, {1, 0, 1}, {-1, 0, -1}, {1, 0, -1},
                      {-1, 0, 1}, {0, 1, 1}, {0, -1, -1}, {0, 1, -1}, {0, -1, 1}};
}

// n cells f[n][19]; out[n][19], mom[n][4] = rho, u; ok[n] = 1 where the fixed-point form takes the cell
extern "C" void fx_cells(const double *f, int n, const double *tau0, const double *c18, double *out, double *mom,
                         unsigned char *ok) {
  for (int k = 0; k < n; ++k) {
    double in[19], res[19];
    for (int i = 0; i < 19; ++i) in[i] = f[19 * k + i];
    sw::fx::Moments m;
    ok[k] = sw::fx::collide(in, tau0[k], tau0[k] * tau0[k], c18[k], res, m);
    if (!ok[k]) continue;
    for (int i = 0; i < 19; ++i) out[19 * k + i] = res[i];
    mom[4 * k] = m.rho;
    for (int a = 0; a < 3; ++a) mom[4 * k + 1 + a] = m.vel(a);
  }
}

// lbm3d.py:103-155 in long double: err[n][19] = got - exact, mom_err[n][4] likewise
extern "C" void long_cells(const double *f, int n, const double *tau0, const double *c18, const double *got,
                           const double *got_mom, double *err, double *mom_err) {
  typedef long double L;
  for (int k = 0; k < n; ++k) {
    L rho = 0, m[3] = {0, 0, 0}, p[3][3] = {}, u[3], q = 0;
    for (int i = 0; i < 19; ++i) {
      const L v = f[19 * k + i];
      rho += v;
      for (int a = 0; a < 3; ++a) {
        m[a] += v * C[i][a];
        for (int b = 0; b < 3; ++b) p[a][b] += v * (C[i][a] * C[i][b]);
      }
    }
    for (int a = 0; a < 3; ++a) u[a] = m[a] / rho;
    for (int a = 0; a < 3; ++a)
      for (int b = 0; b < 3; ++b) {
        p[a][b] -= (a == b ? rho / 3 : 0) + m[a] * u[b];
        q += p[a][b] * p[a][b];
      }
    const L t0 = tau0[k], tau = (t0 + std::sqrt(t0 * t0 + (L)c18[k] * std::sqrt(q) / rho)) / 2, keep = 1 - 1 / tau;
    for (int i = 0; i < 19; ++i) {
      const L w = i == 0 ? 1.0L / 3 : i < 7 ? 1.0L / 18 : 1.0L / 36;
      L cu = 0, qn = 0;
      for (int a = 0; a < 3; ++a) {
        cu += 3 * u[a] * C[i][a];
        for (int b = 0; b < 3; ++b) qn += (C[i][a] * C[i][b] - (a == b ? 1.0L / 3 : 0)) * p[a][b];
      }
      const L usq = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
      err[19 * k + i] = (double)(got[19 * k + i] - w * (rho * (1 + cu + cu * cu / 2 - 1.5L * usq) + 4.5L * keep * qn));
    }
    mom_err[4 * k] = (double)(got_mom[4 * k] - rho);
    for (int a = 0; a < 3; ++a) mom_err[4 * k + 1 + a] = (double)(got_mom[4 * k + 1 + a] - u[a]);
  }
}
