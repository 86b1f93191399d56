// Device check of hc_newton.h: recip and inv_length, with the hardware's seeds,
// against long double over dense mantissas and many binades, and at the ends of
// their ranges; CUDA's own quotient and root beside them.
#include <cmath>
#include <cstdio>
#include <limits>
#include <vector>

#include <cuda_runtime.h>

#include "hc_newton.h"

__global__ void evaluate(const double* x, int n, double* recip, double* inv, double* len, double* cuda) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  recip[i] = hcnewton::recip(x[i]);
  hcnewton::inv_length(x[i], inv[i], len[i]);
  cuda[2 * i] = 1.0 / x[i];
  cuda[2 * i + 1] = sqrt(x[i]);
}

#define CHECK(call)                                                   \
  do {                                                                \
    const cudaError_t e_ = (call);                                    \
    if (e_ != cudaSuccess) {                                          \
      printf("%s: %s\n", #call, cudaGetErrorString(e_));              \
      return 2;                                                       \
    }                                                                 \
  } while (0)

int main() {
  std::vector<double> x;
  // every 2^-18 of the two binades a square root's seed tells apart
  for (int k = 0; k < 1 << 19; ++k) x.push_back(1.0 + 3.0 * k / (1 << 19));
  // mantissas of all widths, over the binades where 1/x and sqrt(x) are normal
  uint64_t s = 0x853c49e6748fea9bull;
  for (int k = 0; k < 1 << 19; ++k) {
    s ^= s << 13;
    s ^= s >> 7;
    s ^= s << 17;
    const int e = (int)(s % 2043) - 1021;
    x.push_back(std::ldexp(1.0 + (double)((s >> 12) >> (k % 52)) * std::ldexp(1.0, k % 52 - 52), e));
  }
  for (int e = -1021; e <= 1021; ++e)
    for (double m : {1.0, std::nextafter(1.0, 2.0), std::nextafter(2.0, 1.0)}) x.push_back(std::ldexp(m, e));
  const int regular = (int)x.size();
  for (double v : {0.0, 5e-324, 1e-310, 2.2250738585072009e-308, 2.2250738585072014e-308}) x.push_back(v);
  const int n = (int)x.size();
  double* d;
  CHECK(cudaMalloc(&d, 6 * sizeof(double) * n));
  CHECK(cudaMemcpy(d, x.data(), sizeof(double) * n, cudaMemcpyHostToDevice));
  evaluate<<<(n + 255) / 256, 256>>>(d, n, d + n, d + 2 * n, d + 3 * n, d + 4 * n);
  CHECK(cudaGetLastError());
  std::vector<double> r(5 * (size_t)n);
  CHECK(cudaMemcpy(r.data(), d + n, 5 * sizeof(double) * n, cudaMemcpyDeviceToHost));
  CHECK(cudaFree(d));
  const double *recip = r.data(), *inv = recip + n, *len = inv + n, *cuda = len + n;
  // relative errors in units of 2^-53
  long double worst[5] = {}, square[5] = {};
  for (int i = 0; i < regular; ++i) {
    const long double X = x[i], S = sqrtl(X);
    const long double e[5] = {fabsl(recip[i] * X - 1.0L), fabsl(inv[i] * S - 1.0L), fabsl(len[i] / S - 1.0L),
                              fabsl(cuda[2 * i] * X - 1.0L), fabsl(cuda[2 * i + 1] / S - 1.0L)};
    for (int k = 0; k < 5; ++k) {
      if (!(e[k] <= 0x1p-52L)) {
        printf("x = %.17g: result %d off by %.3Lg of 2^-53\n", x[i], k, e[k] * 0x1p53L);
        return 1;
      }
      worst[k] = fmaxl(worst[k], e[k] * 0x1p53L);
      square[k] += e[k] * e[k] * 0x1p106L;
    }
  }
  const char* name[5] = {"recip", "inverse length", "length", "CUDA 1/x", "CUDA sqrt"};
  for (int k = 0; k < 5; ++k) printf("%s: rms %.4Lf worst %.4Lf of 2^-53\n", name[k], sqrtl(square[k] / regular), worst[k]);
  // no length for zero and subnormals; the smallest normal number has one
  for (int i = regular; i < n - 1; ++i)
    if (inv[i] != 0.0 || len[i] != 0.0) {
      printf("length of %.17g: %.17g %.17g\n", x[i], inv[i], len[i]);
      return 1;
    }
  if (!(fabsl(len[n - 1] / sqrtl((long double)x[n - 1]) - 1.0L) <= 0x1p-52L)) {
    printf("length of %.17g: %.17g\n", x[n - 1], len[n - 1]);
    return 1;
  }
  printf("ok %d\n", n);
  return 0;
}
