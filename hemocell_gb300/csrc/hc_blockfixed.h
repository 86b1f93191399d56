// The FP64 collision and moments in block fixed point.
//
// This GPU's FP64 pipe (two lanes an SM and cycle: 16 cycles a warp instruction)
// bounded the plain form's lattice kernels at a fifth of the memory bandwidth,
// while its 32-bit integer units issue four warp instructions a cycle.  A node's
// 19 populations and its force share one exponent, that of the largest of them:
// each becomes a 64-bit integer in units of 2^(top - 57), where 2^top is at most
// the largest magnitude.  All of them are then held to half such a unit: 58 bits of
// the largest, as many fewer of a smaller one as it is smaller (below a 32nd of the
// largest fewer than a double's 53), and sums are exact.  Double arithmetic, whose
// moments round to 2^-53 of the largest and enter every population, is no closer:
// whole runs are a tenth as far off (tests/lattice_error_check.cpp).  Sums, the pair
// terms and the relaxation run on those integers; the scalars of a node (1/rho, u,
// the even part, the force's shares) stay in FP64: 27 FP64 instructions a node
// instead of 143.
//
// Bounds: |v| < 2^(top + 1) for every population and force component, so the
// moments stay below 19, a below 6, b below 4 and the results below 25 of those
// units times 2^58 for |u| < 1/4, which fit 63 bits.  A node with |u| >= 1/4,
// rho outside [1/2, 2) or a value that is not finite is refused, and the caller
// takes the FP64 collision.
//
// Host and device compile the same code; a CPU test measures its error and the
// FP64 collision's against long double.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#include "hc_newton.h"
#include "hc_posbits.h"

namespace hcfix {

HC_POS_HD uint64_t shift_right(uint64_t m, int n) {  // 0 for n >= 64
#ifdef __CUDA_ARCH__
  uint64_t r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(m), "r"(n));
  return r;
#else
  return n > 63 ? 0 : m >> n;
#endif
}
HC_POS_HD int64_t mul_high(int64_t a, int64_t b) {
#ifdef __CUDA_ARCH__
  return __mul64hi(a, b);
#else
  return (int64_t)(((__int128)a * b) >> 64);
#endif
}
HC_POS_HD int leading_zeros(uint64_t x) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)x);
#else
  return x ? __builtin_clzll(x) : 64;
#endif
}
HC_POS_HD double reciprocal(double x) {
#ifdef __CUDA_ARCH__
  return hcnewton::recip(x);
#else
  return 1.0 / x;
#endif
}

HC_POS_HD int exponent(double v) {  // biased
  uint32_t hi, lo;
  hcpos::double_words(v, hi, lo);
  return (int)((hi >> 20) & 0x7ffu);
}
HC_POS_HD uint32_t magnitude_word(double v) {  // grows with |v|; above 0x7ff00000 for a NaN
  uint32_t hi, lo;
  hcpos::double_words(v, hi, lo);
  return hi & 0x7fffffffu;
}

// v in units of 2^(top - 1023 - 57), to the nearest (truncation would take a
// little off every value, every step); top is a biased exponent and
// |v| < 2^(top - 1023 + 6).  A subnormal v counts as its leading bit alone would
// and is below any unit in use.
HC_POS_HD int64_t to_fixed(double v, int top) {
  uint32_t hi, lo;
  hcpos::double_words(v, hi, lo);
  const uint32_t mh = (hi << 11) | (lo >> 21) | 0x80000000u;
  const uint64_t m = ((uint64_t)mh << 32) | (lo << 11);
  const int64_t x = (int64_t)((shift_right(m, 5 + top - (int)((hi >> 20) & 0x7ffu)) + 1) >> 1);
  const int64_t s = (int64_t)((int32_t)hi >> 31);
  return (x ^ s) - s;
}
// the double nearest to x units (ties away from zero)
HC_POS_HD double from_fixed(int64_t x, int top) {
  const int64_t s = x >> 63;
  const uint64_t a = (uint64_t)((x ^ s) - s);
  const int lz = leading_zeros(a);
  const uint64_t m = a << (lz & 63);
  const uint64_t r = (m >> 11) + ((m >> 10) & 1u);
  const uint64_t bits = ((uint64_t)(uint32_t)(top + 5 - lz) << 52) + r;
  return hcpos::double_from_words(a ? (uint32_t)(bits >> 32) | ((uint32_t)(s >> 32) & 0x80000000u) : 0u,
                                  a ? (uint32_t)bits : 0u);
}

// units small enough for every later exponent to stay normal
constexpr int kLeastTop = 200;
constexpr int kVelocityTop = 1016;   // u in units of 2^-64, |u| < 1/4
constexpr int kRelaxationTop = 1018;  // 1 - omega, which rounds to 1 for a large tau, in units of 2^-62

// The common exponent of the populations and the force; 2047 when one of them
// is not finite.
HC_POS_HD int block_top(const double f[19], double Fx, double Fy, double Fz) {
  uint32_t m = magnitude_word(Fx);
  const uint32_t my = magnitude_word(Fy), mz = magnitude_word(Fz);
  m = m > my ? m : my;
  m = m > mz ? m : mz;
#ifdef __CUDACC__
#pragma unroll
#endif
  for (int i = 0; i < 19; ++i) {
    const uint32_t w = magnitude_word(f[i]);
    m = m > w ? m : w;
  }
  const int top = (int)(m >> 20);
  return top > kLeastTop ? top : kLeastTop;
}

struct Moments {
  int64_t mass, Jx, Jy, Jz;  // rhoBar and j in units
  double rhoBar, jx, jy, jz;
};
HC_POS_HD Moments fixed_moments(const int64_t x[19], int top) {
  int64_t d[10], p[10];
#ifdef __CUDACC__
#pragma unroll
#endif
  for (int i = 1; i <= 9; ++i) {
    d[i] = x[i + 9] - x[i];
    p[i] = x[i + 9] + x[i];
  }
  const int64_t r = x[0] + ((p[1] + p[2]) + (p[3] + p[4])) + ((p[5] + p[6]) + (p[7] + p[8])) + p[9];
  const int64_t jx = (d[1] + d[4]) + (d[5] + d[6]) + d[7], jy = (d[2] + d[4]) - d[5] + (d[8] + d[9]),
                jz = (d[3] + d[6]) - d[7] + (d[8] - d[9]);
  return {r, jx, jy, jz, from_fixed(r, top), from_fixed(jx, top), from_fixed(jy, top), from_fixed(jz, top)};
}

// omega-dependent constants of the collision (see hcd::CollideK)
struct Relax {
  double om, gF, aF;  // omega, -3 (1 - omega/2), (1 - omega/2) / 8
  int32_t bhi, blo;   // omega 3/36 in units of 2^-63: bhi 2^31 + blo, blo >= 0
  int64_t om1;        // 1 - omega in units of 2^-62
};
// omega / 12 in units of 2^-63, to the nearest: omega = m 2^(e - 53) with a whole m
inline int64_t omega_twelfth(double om) {
  int e;
  const uint64_t m = (uint64_t)ldexp(frexp(om, &e), 53);
  const int up = 10 + e;
  if (up <= -64) return 0;
  return (int64_t)(((up >= 0 ? (unsigned __int128)m << up : (unsigned __int128)(m >> -up)) + 6) / 12);
}
// J omega / 12 to the nearest, |J| < 2^62: with J = j1 2^32 + j0 the quotient
// (j1 2^32 + j0) (bhi 2^31 + blo) / 2^63 takes four 32-bit products
HC_POS_HD int64_t momentum_share(int64_t J, const Relax& k) {
  const int32_t j1 = (int32_t)(J >> 32);
  const uint32_t j0 = (uint32_t)J;
  const int64_t low = (int64_t)j1 * k.blo + (int64_t)(((uint64_t)j0 * (uint32_t)k.blo >> 32) + (1u << 30));
  const int64_t mid = (int64_t)((uint64_t)low << 1) + (int64_t)((uint64_t)j0 * (uint32_t)k.bhi);
  return (int64_t)j1 * k.bhi + (mid >> 32);
}
inline Relax relax_constants(double om) {
  const double hs = 1.0 - 0.5 * om;
  const int64_t b = omega_twelfth(om);
  return {om, -3.0 * hs, 0.125 * hs, (int32_t)(b >> 31), (int32_t)(b & 0x7fffffff),
          to_fixed(1.0 - om, kRelaxationTop)};
}

// The Guo-forced BGK collision of the pair terms P + Q, P - Q (see
// collide_store): store(i, value) receives the 19 post-collision populations.
// Returns false, having stored nothing, where the bounds do not hold.
template <typename Store>
HC_POS_HD bool collide(const double f[19], double Fx, double Fy, double Fz, const Relax& k, const Store& store) {
  const int top = block_top(f, Fx, Fy, Fz);
  if (top >= 2047) return false;
  int64_t x[19];
#ifdef __CUDACC__
#pragma unroll
#endif
  for (int i = 0; i < 19; ++i) x[i] = to_fixed(f[i], top);
  const Moments M = fixed_moments(x, top);
  const double rho = 1.0 + M.rhoBar;
  if (magnitude_word(rho) - 0x3fe00000u >= 0x00200000u || rho < 0.0) return false;  // [1/2, 2)
  const double inv = reciprocal(rho);
  const double mx = fma(0.5, Fx, M.jx), my = fma(0.5, Fy, M.jy), mz = fma(0.5, Fz, M.jz);
  const double ux = mx * inv, uy = my * inv, uz = mz * inv;
  const uint32_t quarter = 0x3fd00000u;
  if (magnitude_word(ux) >= quarter || magnitude_word(uy) >= quarter || magnitude_word(uz) >= quarter) return false;
  const double mu = fma(mx, ux, fma(my, uy, mz * uz)), uF = fma(ux, Fx, fma(uy, Fy, uz * Fz));
  const double even = fma(k.gF, uF, k.om * fma(-1.5, mu, M.rhoBar));
  // the share of an axis population, and of a diagonal one in two roundings that
  // add up to it; one unit each for what the products below lose on average by
  // rounding down
  const int64_t P4 = to_fixed(even * (1.0 / 9.0), top) + 4;
  const int64_t P2 = (P4 - 1) >> 1, P = P4 >> 2, Q = (P4 + 2) >> 2;
  // b = w (3 omega m + 3 (1 - omega/2) F) = omega/12 j + F/12 with j in whole units:
  // a factor omega/12 of 53 bits gave or took the same 1e-16 of the momentum in
  // every step, and the velocities drifted: a quarter of the set-ups of
  // tests/lattice_error_check.cpp were up to 1.3 times as far off as FP64, of
  // which none is half as far now.  a = w (4.5 omega m + 9 (1 - omega/2) F) is 3/2
  // of it and F (1 - omega/2) / 8.
  auto share = [&](int64_t J, double F) { return momentum_share(J, k) + to_fixed(F * (1.0 / 12.0), top); };
  auto forced = [&](int64_t b, double F) { return b + (b >> 1) + to_fixed(k.aF * F, top); };
  const int64_t bx = share(M.Jx, Fx), by = share(M.Jy, Fy), bz = share(M.Jz, Fz);
  const int64_t ax = forced(bx, Fx), ay = forced(by, Fy), az = forced(bz, Fz);
  const int64_t vx = to_fixed(ux, kVelocityTop), vy = to_fixed(uy, kVelocityTop), vz = to_fixed(uz, kVelocityTop);
  // c = c_j of the pair (i, j = i + 9): (c.u) (c.a) + P and c.b.  The products
  // round down, alike for i and j, so their momentum cancels; the rest population
  // is what is left of the node's mass.  The 19 integers keep that mass exactly,
  // the doubles they become to their own rounding.
  int64_t left = M.mass;
  auto pair = [&](int i, int64_t cu, int64_t ca, int64_t cb, int64_t p) {
    const int64_t e = p + mul_high(cu, ca);
    const int64_t plus = mul_high(4 * x[i + 9], k.om1) + e + cb, minus = mul_high(4 * x[i], k.om1) + e - cb;
    left -= plus + minus;
    store(i + 9, from_fixed(plus, top));
    store(i, from_fixed(minus, top));
  };
  pair(1, vx, 2 * ax, 2 * bx, P2);
  pair(2, vy, 2 * ay, 2 * by, P2);
  pair(3, vz, 2 * az, 2 * bz, P2);
  pair(4, vx + vy, ax + ay, bx + by, P);
  pair(5, vx - vy, ax - ay, bx - by, Q);
  pair(6, vx + vz, ax + az, bx + bz, P);
  pair(7, vx - vz, ax - az, bx - bz, Q);
  pair(8, vy + vz, ay + az, by + bz, P);
  pair(9, vy - vz, ay - az, by - bz, Q);
  store(0, from_fixed(left, top));
  return true;
}

// u = (j + F/2) / rho; false where the block's values are not finite
HC_POS_HD bool velocity(const double f[19], double Fx, double Fy, double Fz, double& ux, double& uy, double& uz) {
  const int top = block_top(f, Fx, Fy, Fz);
  if (top >= 2047) return false;
  int64_t x[19];
#ifdef __CUDACC__
#pragma unroll
#endif
  for (int i = 0; i < 19; ++i) x[i] = to_fixed(f[i], top);
  const Moments M = fixed_moments(x, top);
  const double rho = 1.0 + M.rhoBar;
  if (magnitude_word(rho) - 0x3fe00000u >= 0x00200000u || rho < 0.0) return false;
  const double inv = reciprocal(rho);
  const double mx = fma(0.5, Fx, M.jx), my = fma(0.5, Fy, M.jy), mz = fma(0.5, Fz, M.jz);
  // quotients, rounded as divisions are (to one residual)
  ux = mx * inv;
  uy = my * inv;
  uz = mz * inv;
  ux = fma(fma(-ux, rho, mx), inv, ux);
  uy = fma(fma(-uy, rho, my), inv, uy);
  uz = fma(fma(-uz, rho, mz), inv, uz);
  return true;
}

}  // namespace hcfix
