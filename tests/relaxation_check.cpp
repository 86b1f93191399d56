// Host check of the block fixed-point collision over the relaxation times that a
// handle accepts, from just above 1/2 to far beyond those in use: every population
// within 32 last places of the node's largest (the bound of blockfixed_check.cpp)
// of long double.
#include <cmath>
#include <cstdio>
#include <random>

#include "hc_blockfixed.h"

static const int C[19][3] = {{0, 0, 0},  {-1, 0, 0}, {0, -1, 0}, {0, 0, -1}, {-1, -1, 0}, {-1, 1, 0}, {-1, 0, -1},
                             {-1, 0, 1}, {0, -1, -1}, {0, -1, 1}, {1, 0, 0},  {0, 1, 0},   {0, 0, 1},  {1, 1, 0},
                             {1, -1, 0}, {1, 0, 1},  {1, 0, -1}, {0, 1, 1},  {0, 1, -1}};

int main() {
  std::mt19937_64 g(11);
  std::uniform_real_distribution<double> U(-1, 1);
  for (double tau : {0.5 + 1e-15, 0.5001, 0.6, 1.0, 1.0 + 1e-15, 1.001, 3.0, 1e3, 1e8, 1e15, 9e15, 1.7e16, 2e16, 1e30, 1e300}) {
    const double om = 1.0 / tau;
    const hcfix::Relax k = hcfix::relax_constants(om);
    for (int t = 0; t < 20000; ++t) {
      double f[19], x[19];
      const double F[3] = {1e-5 * U(g), 1e-5 * U(g), 1e-5 * U(g)};
      long double rb = 0, j[3] = {}, u[3], uu = 0, uF = 0, scale = 0;
      for (int i = 0; i < 19; ++i) {
        f[i] = 1e-3 * U(g);
        rb += f[i];
        for (int a = 0; a < 3; ++a) j[a] += (long double)C[i][a] * f[i];
      }
      for (int a = 0; a < 3; ++a) {
        u[a] = (j[a] + 0.5L * F[a]) / (1 + rb);
        uu += u[a] * u[a];
        uF += u[a] * F[a];
      }
      if (!hcfix::collide(f, F[0], F[1], F[2], k, [&](int i, double v) { x[i] = v; })) return 1;
      long double worst = 0;
      for (int i = 0; i < 19; ++i) {
        const int n = std::abs(C[i][0]) + std::abs(C[i][1]) + std::abs(C[i][2]);
        const long double w = n == 0 ? 1.0L / 3 : (n == 1 ? 1.0L / 18 : 1.0L / 36);
        long double cu = 0, cF = 0;
        for (int a = 0; a < 3; ++a) {
          cu += C[i][a] * u[a];
          cF += (long double)C[i][a] * F[a];
        }
        const long double e = (1 - (long double)om) * f[i] +
                              om * w * (rb + (1 + rb) * (3 * cu + 4.5L * cu * cu - 1.5L * uu)) +
                              (1 - 0.5L * om) * w * (3 * (cF - uF) + 9 * cu * cF);
        scale = fmaxl(scale, fabsl(e));
        worst = fmaxl(worst, fabsl(x[i] - e));
      }
      if (!(worst <= 32 * 0x1p-53L * scale)) {
        printf("tau %.17g: off by %.3Lg of a largest %.3Lg\n", tau, worst, scale);
        return 1;
      }
    }
  }
  printf("ok\n");
  return 0;
}
