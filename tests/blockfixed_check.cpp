// Host check of hc_blockfixed.h: the block fixed-point collision and velocity
// against long double, beside the same expressions in double.
#include <cmath>
#include <cstdio>
#include <limits>
#include <random>

#include "hc_blockfixed.h"

static const int C[19][3] = {{0, 0, 0},  {-1, 0, 0}, {0, -1, 0}, {0, 0, -1}, {-1, -1, 0}, {-1, 1, 0}, {-1, 0, -1},
                             {-1, 0, 1}, {0, -1, -1}, {0, -1, 1}, {1, 0, 0},  {0, 1, 0},   {0, 0, 1},  {1, 1, 0},
                             {1, -1, 0}, {1, 0, 1},  {1, 0, -1}, {0, 1, 1},  {0, 1, -1}};
static int norm1(int i) { return std::abs(C[i][0]) + std::abs(C[i][1]) + std::abs(C[i][2]); }
template <typename R>
static R weight(int i) {
  return norm1(i) == 0 ? R(1) / 3 : (norm1(i) == 1 ? R(1) / 18 : R(1) / 36);
}

template <typename R>
static void collide(const double f[19], const double F[3], double omega, R out[19], R u[3]) {
  R rb = 0, j[3] = {0, 0, 0};
  for (int i = 0; i < 19; ++i) {
    rb += f[i];
    for (int a = 0; a < 3; ++a) j[a] += (R)C[i][a] * (R)f[i];
  }
  const R rho = 1 + rb, om = omega;
  R uu = 0, uF = 0;
  for (int a = 0; a < 3; ++a) u[a] = (j[a] + R(0.5) * (R)F[a]) / rho;
  for (int a = 0; a < 3; ++a) {
    uu += u[a] * u[a];
    uF += u[a] * (R)F[a];
  }
  for (int i = 0; i < 19; ++i) {
    R cu = 0, cF = 0;
    for (int a = 0; a < 3; ++a) {
      cu += (R)C[i][a] * u[a];
      cF += (R)C[i][a] * (R)F[a];
    }
    const R w = weight<R>(i), eq = w * (rb + rho * (3 * cu + R(4.5) * cu * cu - R(1.5) * uu));
    out[i] = (1 - om) * (R)f[i] + om * eq + (1 - R(0.5) * om) * w * (3 * (cF - uF) + 9 * cu * cF);
  }
}

struct Error {
  double worst = 0, square = 0;
  long long n = 0;
  void add(long double x, long double exact, long double scale) {
    const double e = (double)(fabsl(x - exact) / scale / 0x1p-53L);
    worst = std::fmax(worst, e);
    square += e * e;
    n++;
  }
  double rms() const { return std::sqrt(square / n); }
};

int main() {
  std::mt19937_64 g(5);
  std::uniform_real_distribution<double> U(-1, 1);
  // velocities of 2e-2 down to 1e-10, densities off one by as much, forces over
  // six decades (and none), populations off equilibrium by a tenth
  for (int mode = 0; mode < 8; ++mode) {
    Error fixed, dbl, fixed_u, dbl_u;
    for (int t = 0; t < 100000; ++t) {
      const double amp = std::pow(10.0, -1.7 - 1.2 * mode), force = t % 4 ? std::pow(10.0, -6.5 + 3.0 * U(g)) : 0.0;
      const double v[3] = {amp * U(g), amp * U(g), amp * U(g)}, drho = amp * U(g);
      const double F[3] = {force * U(g), force * U(g), force * U(g)};
      const double om = t % 5 ? 0.6 + 1.3 * (0.5 + 0.5 * U(g)) : 1.0;
      double f[19];
      for (int i = 0; i < 19; ++i) {
        double cu = 0, uu = 0;
        for (int a = 0; a < 3; ++a) {
          cu += C[i][a] * v[a];
          uu += v[a] * v[a];
        }
        const double w = weight<double>(i);
        f[i] = w * (drho + (1 + drho) * (3 * cu + 4.5 * cu * cu - 1.5 * uu)) + 0.1 * amp * w * U(g);
      }
      long double e[19], eu[3];
      double d[19], du[3], x[19], u[3];
      collide<long double>(f, F, om, e, eu);
      collide<double>(f, F, om, d, du);
      if (!hcfix::collide(f, F[0], F[1], F[2], hcfix::relax_constants(om), [&](int i, double r) { x[i] = r; }) ||
          !hcfix::velocity(f, F[0], F[1], F[2], u[0], u[1], u[2])) {
        printf("refused at scale %g\n", amp);
        return 1;
      }
      long double scale = 0, su = 0;
      for (int i = 0; i < 19; ++i) scale = fmaxl(scale, fabsl(e[i]));
      for (int a = 0; a < 3; ++a) su = fmaxl(su, fabsl(eu[a]));
      for (int i = 0; i < 19; ++i) {
        fixed.add(x[i], e[i], scale);
        dbl.add(d[i], e[i], scale);
      }
      for (int a = 0; a < 3; ++a) {
        fixed_u.add(u[a], eu[a], su);
        dbl_u.add(du[a], eu[a], su);
      }
    }
    printf("scale %d: collision rms %.3f worst %.1f (double %.3f, %.1f); velocity rms %.3f worst %.1f (double %.3f, %.1f)\n",
           mode, fixed.rms(), fixed.worst, dbl.rms(), dbl.worst, fixed_u.rms(), fixed_u.worst, dbl_u.rms(),
           dbl_u.worst);
    // no further off than double arithmetic, and within 32 last places of the largest
    if (!(fixed.rms() <= dbl.rms()) || !(fixed_u.rms() <= dbl_u.rms()) || fixed.worst > 32) return 1;
  }
  // a lattice at rest stays at rest; subnormal populations stay nothing
  for (double tiny : {0.0, -0.0, 5e-324, -1e-310}) {
    double f[19], x[19];
    for (double& v : f) v = tiny;
    if (!hcfix::collide(f, 0.0, 0.0, 0.0, hcfix::relax_constants(0.8), [&](int i, double r) { x[i] = r; })) return 1;
    for (double v : x)
      if (!(std::fabs(v) < 1e-240)) return 1;
  }
  // what does not fit the bounds is refused, and nothing is stored
  const double inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
  struct {
    int i;
    double v;
  } bad[] = {{1, 0.4}, {13, -0.5}, {0, 1.5}, {0, -0.6}, {0, -2.5}, {5, inf}, {7, -inf}, {9, nan}, {0, 1e300}};
  for (auto& b : bad) {
    double f[19] = {};
    f[b.i] = b.v;
    bool stored = false;
    if (hcfix::collide(f, 0.0, 0.0, 0.0, hcfix::relax_constants(1.0), [&](int, double) { stored = true; }) || stored) {
      printf("not refused: f[%d] = %g\n", b.i, b.v);
      return 1;
    }
  }
  double f[19] = {}, u[3];
  if (hcfix::velocity(f, nan, 0.0, 0.0, u[0], u[1], u[2]) || hcfix::velocity(f, 0.0, -inf, 0.0, u[0], u[1], u[2])) return 1;
  // conversions: doubles of up to 53 bits within 58 of the top come back
  for (int k = 0; k < 1000000; ++k) {
    const int top = 300 + (int)(g() % 1500), drop = (int)(g() % 6);
    const double v = std::ldexp(1.0 + 0.5 * (1 + U(g)), top - 1023 - drop) * (k % 2 ? 1 : -1);
    if (hcfix::from_fixed(hcfix::to_fixed(v, top), top) != v) {
      printf("%.17g does not come back\n", v);
      return 1;
    }
  }
  printf("ok\n");
  return 0;
}
