// flux_near (rt_exact.cuh), the bit-exact flux with its differences on the
// integer pipes, against the reference's sequence in binary64 instructions
// (flux_slow) on a GPU: the same bits (zeros of either sign alike) for every
// operand flux_is_near accepts.
// Values next to powers of two (the rounded differences carry), equal ones,
// gaps of 2^7 to 2^9, and both ends of the accepted range.
#include <cstdint>
#include <cstdio>
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
static double value(int e) {
  uint64_t f = rnd() & 0xfffffffffffffull;
  if ((rnd() & 3) == 0) f &= 7;
  if ((rnd() & 7) == 0) f = 0xfffffffffffffull - (rnd() & 7);
  return f64_from_bits(((uint64_t)e << 52) | f);
}

__global__ void run(const double* v, const double* u, const double* b, const double* c, const double* w, long long n,
                    unsigned long long* taken, unsigned long long* wrong) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    if (!flux_is_near(v[i], u[i], b[i], c[i], w[i])) continue;
    atomicAdd(taken, 1ull);
    const bool pos = f64_pos(v[i]);
    const double got = flux_near(v[i], u[i], b[i], c[i], w[i], pos);
    const double up = pos ? rt::dsub(b[i], w[i]) : rt::dsub(w[i], c[i]);
    const double want = flux_slow(v[i], u[i], rt::dadd(c[i], b[i]), rt::dsub(c[i], b[i]), up);
    // a zero flux (v = 0) may have the other sign: the sum of differences it enters starts at +0 and keeps no -0
    if (f64_bits(got) != f64_bits(want) && !(got == 0.0 && want == 0.0) && atomicAdd(wrong, 1ull) < 10)
      printf("v %.17g u %.17g b %.17g c %.17g w %.17g: %.17g, want %.17g\n", v[i], u[i], b[i], c[i], w[i], got, want);
  }
}

int main() {
  const long long n = 4000000;
  std::vector<double> h[5];
  for (long long i = 0; i < n; i++) {
    const int e = i % 9 == 0 ? 756 + (int)(rnd() % 10) : (i % 9 == 1 ? 1270 + (int)(rnd() % 12) : 900 + (int)(rnd() % 200));
    double b = value(e + (int)(rnd() % 10)), c = value(e + (int)(rnd() % 10)), w = value(e + (int)(rnd() % 10));
    if (i % 5 == 0) c = b;
    if (i % 7 == 0) w = c;
    if (i % 11 == 0) c = b * (1 + 1e-15);
    if (i % 13 == 0 && 2 * b - c > 0) w = 2 * b - c;
    double v = value(1000 + (int)(rnd() % 30)), u = value(990 + (int)(rnd() % 34));
    if (i % 17 == 0) v = value(700 + (int)(rnd() % 4));
    if (i % 19 == 0) u = value(700 + (int)(rnd() % 4));
    if (i % 23 == 0) v = u = 0.0;
    if (rnd() & 1) v = -v;
    const double all[5] = {v, u, b, c, w};
    for (int k = 0; k < 5; k++) h[k].push_back(all[k]);
  }
  double* d[5];
  unsigned long long *count, got[2] = {0, 0};
  for (int k = 0; k < 5; k++) {
    if (cudaMalloc(&d[k], n * 8) != cudaSuccess) return 2;
    cudaMemcpy(d[k], h[k].data(), n * 8, cudaMemcpyHostToDevice);
  }
  if (cudaMalloc(&count, 16) != cudaSuccess) return 2;
  cudaMemset(count, 0, 16);
  run<<<152 * 4, 256>>>(d[0], d[1], d[2], d[3], d[4], n, count, count + 1);
  if (cudaDeviceSynchronize() != cudaSuccess) return 2;
  cudaMemcpy(got, count, 16, cudaMemcpyDeviceToHost);
  std::printf("%llu fluxes, %llu wrong\n", got[0], got[1]);
  return got[1] || got[0] < 1000000 ? 1 : 0;
}
