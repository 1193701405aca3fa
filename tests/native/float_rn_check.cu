// float_rn (rt_exact.cuh) against the conversion itself: the same bits for
// ties, carries into the next exponent, both ends of the normal range,
// denormals, zeros, infinities and NaN.  Host form by default, "--device" on a
// GPU.
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
__global__ void run(const double* x, float* a, float* b, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    a[i] = float_rn(x[i]);
    b[i] = __double2float_rn(x[i]);
  }
}

int main(int argc, char** argv) {
  const bool device = argc > 1 && std::strcmp(argv[1], "--device") == 0;
  std::vector<double> X;
  for (int e = 0; e < 2048; e++)
    for (int i = 0; i < 600; i++) {
      uint64_t f = rnd() & 0xfffffffffffffull;
      switch (i % 6) {
        case 0: f = (f & ~0x1fffffffull) | 0x10000000ull; break;                  // a tie
        case 1: f = (f & ~0x1fffffffull) | (0x10000000ull + (rnd() % 3) - 1); break;
        case 2: f = 0xfffffffffffffull - (rnd() & 0x3fffffffull); break;          // carries
        case 3: f = rnd() & 3; break;
      }
      const uint64_t u = ((uint64_t)(rnd() & 1) << 63) | ((uint64_t)e << 52) | f;
      double x;
      std::memcpy(&x, &u, 8);
      X.push_back(x);
    }
  X.push_back(0.0);
  X.push_back(-0.0);
  const long long n = (long long)X.size();
  std::vector<float> A(n), B(n);
  if (device) {
    double* x;
    float *a, *b;
    if (cudaMalloc(&x, n * 8) != cudaSuccess || cudaMalloc(&a, n * 4) != cudaSuccess || cudaMalloc(&b, n * 4) != cudaSuccess)
      return 2;
    cudaMemcpy(x, X.data(), n * 8, cudaMemcpyHostToDevice);
    run<<<152, 256>>>(x, a, b, n);
    if (cudaDeviceSynchronize() != cudaSuccess) return 2;
    cudaMemcpy(A.data(), a, n * 4, cudaMemcpyDeviceToHost);
    cudaMemcpy(B.data(), b, n * 4, cudaMemcpyDeviceToHost);
  } else {
    for (long long i = 0; i < n; i++) {
      A[i] = float_rn(X[i]);
      B[i] = (float)X[i];
    }
  }
  long long bad = 0;
  for (long long i = 0; i < n; i++)
    if (std::memcmp(&A[i], &B[i], 4) && !(A[i] != A[i] && B[i] != B[i]) && bad++ < 10)
      std::printf("%a: %a, want %a\n", X[i], A[i], B[i]);
  std::printf("%lld values, %lld wrong\n", n, bad);
  return bad ? 1 : 0;
}
