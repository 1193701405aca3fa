// superbee_near64 (rt_fast.cuh), the limited slope as exact integers rounded
// once, against superbee_slope64 on the rounded differences: the same bits
// for every triple that slope_near accepts, and none accepted outside the
// range it states.  Host form by default; "--device" on a GPU.
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <vector>

#include "rt_fast.cuh"

using namespace rt;

static uint64_t rng_state = 88172645463325252ull;
static uint64_t rnd() {
  rng_state ^= rng_state << 13;
  rng_state ^= rng_state >> 7;
  rng_state ^= rng_state << 17;
  return rng_state * 2685821657736338717ull;
}
static double value(int e) {
  uint64_t f = rnd() & 0xfffffffffffffull;
  if ((rnd() & 3) == 0) f &= 7;
  if ((rnd() & 7) == 0) f = 0xfffffffffffffull - (rnd() & 7);
  return f64_from_bits(((uint64_t)e << 52) | f);
}

__host__ __device__ inline double direct(double b, double c, double w, bool pos) {
  return superbee_slope64(c - b, (pos ? b : w) - (pos ? w : c));
}
__global__ void run(const double* b, const double* c, const double* w, const int* pos, double* x, double* y, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    x[i] = superbee_near64(b[i], c[i], w[i], pos[i]);
    y[i] = direct(b[i], c[i], w[i], pos[i]);
  }
}

int main(int argc, char** argv) {
  const bool device = argc > 1 && std::strcmp(argv[1], "--device") == 0;
  std::vector<double> B, C, W;
  std::vector<int> P;
  long long refused = 0, bad = 0;
  for (long long i = 0; i < 4000000; i++) {
    const int e = i % 9 == 0 ? 90 + (int)(rnd() % 30) : (i % 9 == 1 ? 1880 + (int)(rnd() % 40) : 900 + (int)(rnd() % 200));
    double b = value(e + (int)(rnd() % 10)), c = value(e + (int)(rnd() % 10)), w = value(e + (int)(rnd() % 10));
    if (i % 5 == 0) c = b;
    if (i % 7 == 0) w = c;
    if (i % 11 == 0) c = b * (1 + 1e-15);
    if (i % 13 == 0) w = 2 * b - c > 0 ? 2 * b - c : w;
    if (i % 1001 == 0) b = -b;
    if (i % 1003 == 0) c = 0.0;
    if (!slope_near(b, c, w)) {
      refused++;
      continue;
    }
    const double hi = b > c ? (b > w ? b : w) : (c > w ? c : w), lo = b < c ? (b < w ? b : w) : (c < w ? c : w);
    if (!(lo > 0x1p-930) || !(hi < 0x1p890) || !(hi < lo * 512)) bad++;
    B.push_back(b);
    C.push_back(c);
    W.push_back(w);
    P.push_back((int)(rnd() & 1));
  }
  const long long n = (long long)B.size();
  std::vector<double> X(n), Y(n);
  if (device) {
    double* d[5];
    int* p;
    for (auto& q : d)
      if (cudaMalloc(&q, n * 8) != cudaSuccess) return 2;
    if (cudaMalloc(&p, n * 4) != cudaSuccess) return 2;
    cudaMemcpy(d[0], B.data(), n * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(d[1], C.data(), n * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(d[2], W.data(), n * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(p, P.data(), n * 4, cudaMemcpyHostToDevice);
    run<<<152 * 4, 256>>>(d[0], d[1], d[2], p, d[3], d[4], n);
    if (cudaDeviceSynchronize() != cudaSuccess) return 2;
    cudaMemcpy(X.data(), d[3], n * 8, cudaMemcpyDeviceToHost);
    cudaMemcpy(Y.data(), d[4], n * 8, cudaMemcpyDeviceToHost);
  } else {
    for (long long i = 0; i < n; i++) {
      X[i] = superbee_near64(B[i], C[i], W[i], P[i]);
      Y[i] = direct(B[i], C[i], W[i], P[i]);
    }
  }
  for (long long i = 0; i < n; i++)
    if (f64_bits(X[i]) != f64_bits(Y[i]) && !(X[i] == 0.0 && Y[i] == 0.0) && bad++ < 10)
      std::printf("b %a c %a w %a pos %d: %a, want %a\n", B[i], C[i], W[i], P[i], X[i], Y[i]);
  std::printf("%lld triples, %lld refused, %lld wrong\n", n, refused, bad);
  return bad || n < 1000000 ? 1 : 0;
}
