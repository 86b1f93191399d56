// Host check of the block fixed-point collision over whole runs: small lattices
// (a closed box with a moving lid, a periodic box with an obstacle, a periodic box,
// and shear between walls) stepped with it, with the same equations in double, and
// in long double.  Its velocities and populations may not be further off than
// double's in any set-up: what one collision rounds alike in every step (a constant
// of the relaxation) adds up, which the errors of single collisions do not show.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "hc_blockfixed.h"

static const int C[19][3] = {{0, 0, 0},  {-1, 0, 0}, {0, -1, 0}, {0, 0, -1}, {-1, -1, 0}, {-1, 1, 0}, {-1, 0, -1},
                             {-1, 0, 1}, {0, -1, -1}, {0, -1, 1}, {1, 0, 0},  {0, 1, 0},   {0, 0, 1},  {1, 1, 0},
                             {1, -1, 0}, {1, 0, 1},  {1, 0, -1}, {0, 1, 1},  {0, 1, -1}};
static const int D[3] = {12, 14, 11};
static const int N = 12 * 14 * 11;
enum Kind { LID, OBSTACLE, PERIODIC, SHEAR };

template <typename R>
static R weight(int i) {
  const int n = std::abs(C[i][0]) + std::abs(C[i][1]) + std::abs(C[i][2]);
  return n == 0 ? R(1) / 3 : (n == 1 ? R(1) / 18 : R(1) / 36);
}
template <typename R>
static void moments(const R* f, R& rb, R j[3]) {
  rb = j[0] = j[1] = j[2] = 0;
  for (int i = 0; i < 19; ++i) {
    rb += f[i];
    for (int a = 0; a < 3; ++a) j[a] += C[i][a] * f[i];
  }
}
template <typename R>
static void collide(R* f, const double F[3], double omega) {
  R rb, j[3], u[3], uu = 0, uF = 0;
  moments(f, rb, j);
  const R rho = 1 + rb, om = omega;
  for (int a = 0; a < 3; ++a) {
    u[a] = (j[a] + R(0.5) * R(F[a])) / rho;
    uu += u[a] * u[a];
    uF += u[a] * R(F[a]);
  }
  for (int i = 0; i < 19; ++i) {
    R cu = 0, cF = 0;
    for (int a = 0; a < 3; ++a) {
      cu += C[i][a] * u[a];
      cF += C[i][a] * R(F[a]);
    }
    const R w = weight<R>(i);
    f[i] = (1 - om) * f[i] + om * (w * (rb + rho * (3 * cu + R(4.5) * cu * cu - R(1.5) * uu))) +
           (1 - R(0.5) * om) * w * (3 * (cF - uF) + 9 * cu * cF);
  }
}
static bool solid(Kind kind, int x, int y, int z) {
  return kind == OBSTACLE && (x - 6) * (x - 6) + (y - 7) * (y - 7) + (z - 5) * (z - 5) < 7;
}

template <typename R>
static bool run(Kind kind, double omega, int steps, bool fixed, std::vector<R>& f, std::vector<R>& u) {
  std::mt19937_64 g(7);
  std::uniform_real_distribution<double> U(-1, 1);
  f.assign(19 * N, R(0));
  std::vector<R> next(f);
  std::vector<double> F(3 * N, 0.0);
  const bool force = kind == OBSTACLE || kind == PERIODIC;
  for (int n = 0; n < N && force; ++n)
    for (int a = 0; a < 3; ++a) F[3 * n + a] = 1e-6 * U(g) + (a == 0 ? 2e-6 : 0.0);
  for (int n = 0; n < N && kind == PERIODIC; ++n) {
    const double v[3] = {0.01 * U(g), 0.01 * U(g), 0.01 * U(g)}, drho = 1e-3 * U(g);
    for (int i = 0; i < 19; ++i)
      f[19 * n + i] = weight<double>(i) * (drho + 3 * (C[i][0] * v[0] + C[i][1] * v[1] + C[i][2] * v[2]));
  }
  const hcfix::Relax k = hcfix::relax_constants(omega);
  auto at = [](int x, int y, int z) { return (x * D[1] + y) * D[2] + z; };
  for (int t = 0; t < steps; ++t) {
    for (int n = 0; n < N; ++n) {
      if (solid(kind, n / (D[1] * D[2]), n / D[2] % D[1], n % D[2])) continue;
      R* p = &f[19 * n];
      if (!fixed) {
        collide(p, &F[3 * n], omega);
        continue;
      }
      double in[19], out[19];
      for (int i = 0; i < 19; ++i) in[i] = (double)p[i];
      if (!hcfix::collide(in, F[3 * n], F[3 * n + 1], F[3 * n + 2], k, [&](int i, double v) { out[i] = v; })) return false;
      for (int i = 0; i < 19; ++i) p[i] = out[i];
    }
    for (int x = 0; x < D[0]; ++x)
      for (int y = 0; y < D[1]; ++y)
        for (int z = 0; z < D[2]; ++z) {
          if (solid(kind, x, y, z)) continue;
          for (int i = 0; i < 19; ++i) {
            int q[3] = {x - C[i][0], y - C[i][1], z - C[i][2]};
            bool wall = false;
            const bool lid = q[1] >= D[1] && (kind == LID || kind == SHEAR);
            for (int a = 0; a < 3; ++a) {
              const bool out = q[a] < 0 || q[a] >= D[a];
              if (out && (kind == LID || (kind == SHEAR && a == 1))) wall = true;
              q[a] = (q[a] + D[a]) % D[a];
            }
            wall = wall || solid(kind, q[0], q[1], q[2]);
            const int o = i == 0 ? 0 : (i <= 9 ? i + 9 : i - 9), n = at(x, y, z);
            next[19 * n + i] = wall ? f[19 * n + o] + (lid ? 6 * weight<R>(i) * C[i][0] * R(0.02) : R(0))
                                    : f[19 * at(q[0], q[1], q[2]) + i];
          }
        }
    f.swap(next);
  }
  u.assign(3 * N, R(0));
  for (int n = 0; n < N; ++n) {
    if (fixed) {
      double in[19], v[3];
      for (int i = 0; i < 19; ++i) in[i] = (double)f[19 * n + i];
      if (!hcfix::velocity(in, 0.0, 0.0, 0.0, v[0], v[1], v[2])) return false;
      for (int a = 0; a < 3; ++a) u[3 * n + a] = v[a];
    } else {
      R rb, j[3];
      moments(&f[19 * n], rb, j);
      for (int a = 0; a < 3; ++a) u[3 * n + a] = j[a] / (1 + rb);
    }
  }
  return true;
}

static double distance(const std::vector<double>& a, const std::vector<long double>& e) {
  long double d = 0, s = 0;
  for (size_t i = 0; i < a.size(); ++i) {
    d += (a[i] - e[i]) * (a[i] - e[i]);
    s += e[i] * e[i];
  }
  return (double)sqrtl(d / s);
}

int main() {
  const char* name[4] = {"lid", "obstacle", "periodic", "shear"};
  int worse = 0;
  for (int kind = 0; kind < 4; ++kind)
    for (double tau : {0.55, 0.8, 1.1, 1.8})
      for (int steps : {40, 160}) {
        std::vector<long double> ef, eu;
        std::vector<double> df, du, xf, xu;
        run((Kind)kind, 1.0 / tau, steps, false, ef, eu);
        run((Kind)kind, 1.0 / tau, steps, false, df, du);
        if (!run((Kind)kind, 1.0 / tau, steps, true, xf, xu)) return 2;
        const double d = distance(du, eu), x = distance(xu, eu), pd = distance(df, ef), px = distance(xf, ef);
        const bool bad = !(x <= d) || !(px <= pd);
        worse += bad;
        printf("%-8s tau %.2f, %3d steps: velocity %.2e (double %.2e), populations %.2e (%.2e)%s\n", name[kind], tau,
               steps, x, d, px, pd, bad ? "  further off" : "");
      }
  printf("further off in %d\n", worse);
  return worse != 0;
}
