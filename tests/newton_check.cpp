// Host check of hc_newton.h (reciprocal and reciprocal square root from a seed)
// against long double, and of hcpos::floor_bits against floor().
#include <cmath>
#include <cstdio>
#include <cstring>

#include "hc_newton.h"
#include "hc_posbits.h"

static uint64_t state = 0x853c49e6748fea9bull;
static uint64_t next_u64() {
  state ^= state << 13;
  state ^= state >> 7;
  state ^= state << 17;
  return state;
}
static double uniform() { return (double)(next_u64() >> 11) * 0x1p-53; }

int main() {
  const double bound = 0x1p-52;
  long long cases = 0;
  for (int k = 0; k < 2000000; ++k) {
    // arguments over sixty binades either way, seeds off by up to 2^-19
    const double x = (1.0 + uniform()) * std::ldexp(1.0, (int)(next_u64() % 121) - 60);
    const double off = 1.0 + (2.0 * uniform() - 1.0) * 0x1p-19;
    const double r = hcnewton::recip_from(x, off / x);
    if (!(fabsl((long double)r * x - 1.0L) <= bound)) {
      printf("recip(%.17g) = %.17g\n", x, r);
      return 1;
    }
    double inv, root;
    hcnewton::rsqrt_from(x, off / std::sqrt(x), inv, root);
    const long double s = sqrtl((long double)x);
    if (!(fabsl(inv * s - 1.0L) <= bound) || !(fabsl(root / s - 1.0L) <= bound)) {
      printf("rsqrt(%.17g) = %.17g, sqrt %.17g\n", x, inv, root);
      return 1;
    }
    cases += 2;
  }
  for (int k = 0; k < 1000000; ++k) {
    // coordinates in [1, 2^20), a fifth of them on or next to an integer, and some outside
    double P = (1.0 + uniform()) * std::ldexp(1.0, (int)(next_u64() % 20));
    if (k % 5 == 0) P = std::floor(P);
    if (k % 10 == 0) P = std::nextafter(P, k % 20 ? 0.0 : 1e9);
    if (k % 97 == 0) P = (k % 2 ? -1.0 : 1.0) * uniform() * (k % 3 ? 1.0 : 1e9);
    int q;
    double q0;
    if (hcpos::floor_bits(P, q, q0) != (P >= 1.0 && P < 1048576.0) ||
        (P >= 1.0 && P < 1048576.0 && (q0 != std::floor(P) || q != (int)q0))) {
      printf("floor_bits(%.17g)\n", P);
      return 1;
    }
    cases++;
  }
  printf("ok %lld\n", cases);
  return 0;
}
