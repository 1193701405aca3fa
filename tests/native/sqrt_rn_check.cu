// sqrt_rn (rt_exact.cuh) against the correctly rounded square root: the same
// bits for squares and their neighbours, roots next to half-way values, every
// exponent, zeros, infinities, negative numbers and NaN.  Host form by
// default, "--device" on a GPU.
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <vector>

#include "rt_exact.cuh"

using namespace rt;

static uint64_t rng_state = 88172645463325252ull;
static uint64_t rnd() {
  rng_state ^= rng_state << 13;
  rng_state ^= rng_state >> 7;
  rng_state ^= rng_state << 17;
  return rng_state * 2685821657736338717ull;
}
__global__ void run(const double* x, double* a, double* b, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    a[i] = sqrt_rn(x[i]);
    b[i] = __dsqrt_rn(x[i]);
  }
}

int main(int argc, char** argv) {
  const bool device = argc > 1 && std::strcmp(argv[1], "--device") == 0;
  std::vector<double> X;
  const uint64_t frac = 0xfffffffffffffull;
  for (int e = 0; e < 2048; e++)
    for (int i = 0; i < 2000; i++) {
      uint64_t f = rnd() & frac;
      if (i % 8 == 0) f = rnd() & 7;
      if (i % 8 == 1) f = frac - (rnd() & 7);
      if (i % 8 == 2) f &= ~0xffffffffull;
      if (i % 8 >= 3 && i % 8 < 6) {   // the square of a short or half-way root, and beside it
        const int k = i % 8 == 3 ? 27 : (i % 8 == 4 ? 1 : 0);
        const double r = 1.0 + (double)((rnd() & frac) >> k << k) * 0x1p-52 + (k == 1 ? 0x1p-53 : 0.0);
        double q = r * r;
        uint64_t u;
        std::memcpy(&u, &q, 8);
        f = (u + (rnd() % 5) - 2) & frac;
      }
      const uint64_t u = ((uint64_t)(i % 500 == 499) << 63) | ((uint64_t)e << 52) | f;
      double x;
      std::memcpy(&x, &u, 8);
      X.push_back(x);
    }
  X.push_back(0.0);
  X.push_back(-0.0);
  const long long n = (long long)X.size();
  std::vector<double> A(n), B(n);
  if (device) {
    double* x;
    double *a, *b;
    if (cudaMalloc(&x, n * 8) != cudaSuccess || cudaMalloc(&a, n * 8) != cudaSuccess || cudaMalloc(&b, n * 8) != cudaSuccess)
      return 2;
    cudaMemcpy(x, X.data(), n * 8, cudaMemcpyHostToDevice);
    run<<<152, 256>>>(x, a, b, n);
    if (cudaDeviceSynchronize() != cudaSuccess) return 2;
    cudaMemcpy(A.data(), a, n * 8, cudaMemcpyDeviceToHost);
    cudaMemcpy(B.data(), b, n * 8, cudaMemcpyDeviceToHost);
  } else {
    for (long long i = 0; i < n; i++) {
      A[i] = sqrt_rn(X[i]);
      B[i] = __builtin_sqrt(X[i]);
    }
  }
  long long bad = 0;
  for (long long i = 0; i < n; i++)
    if (std::memcmp(&A[i], &B[i], 8) && !(A[i] != A[i] && B[i] != B[i]) && bad++ < 10)
      std::printf("%a: %a, want %a\n", X[i], A[i], B[i]);
  std::printf("%lld values, %lld wrong\n", n, bad);
  return bad ? 1 : 0;
}
