// The integer quotient of rt_exact.cuh against the division instruction:
// div_rn(a, b) must give the bits of a / b, and limited_ratio(up, Rj) the
// bits of the reference's limiter of the rounded ratio.  Operands: random
// significands over random exponent gaps, neighbours of powers of two,
// quotients next to rounding ties, special values.  Host form by default;
// "--device" runs the device form on the same pairs on a GPU.
#include <cmath>
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
static uint64_t bits(double x) {
  uint64_t u;
  std::memcpy(&u, &x, 8);
  return u;
}
static double from(uint64_t u) {
  double x;
  std::memcpy(&x, &u, 8);
  return x;
}
static double limiter(double up, double Rj) {
  double Cr = Rj != 0.0 ? up / Rj : 0.0;
  const double a = 1.0 < 2.0 * Cr ? 1.0 : 2.0 * Cr, b = 2.0 < Cr ? 2.0 : Cr;
  const double m = a > b ? a : b;
  return 0.0 > m ? 0.0 : m;
}
static bool same(double a, double b) { return bits(a) == bits(b) || (a != a && b != b) || (a == 0.0 && b == 0.0); }

__global__ void check_kernel(const double* a, const double* b, double* q, double* c, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    q[i] = div_rn(a[i], b[i]);
    c[i] = isfinite(a[i]) && isfinite(b[i]) ? limited_ratio(a[i], b[i]) : 0.0;
  }
}

int main(int argc, char** argv) {
  const bool device = argc > 1 && std::strcmp(argv[1], "--device") == 0;
  std::vector<double> A, B;
  const double special[] = {0.0, -0.0, 1.0, -1.0, 2.0, 0.5, 3.0, 1e-3, 4.9406564584124654e-324, 2.2250738585072014e-308,
                            1e-310, 1.7976931348623157e308, INFINITY, -INFINITY, NAN, 1e-200, 1e200, 1.0 + 0x1p-52,
                            1.0 - 0x1p-53, 2.0 - 0x1p-52};
  for (double a : special)
    for (double b : special) {
      A.push_back(a);
      B.push_back(b);
    }
  const uint64_t frac = 0xfffffffffffffull;
  for (long long i = 0; i < 4000000; i++) {
    uint64_t fa = rnd() & frac, fb = rnd() & frac;
    switch (i & 15) {
      case 0: fa = rnd() & 15; break;
      case 1: fb = rnd() & 15; break;
      case 2: fa = frac - (rnd() & 15); break;
      case 3: fb = frac - (rnd() & 15); break;
      case 4: fa = (fb + (rnd() & 7)) & frac; break;
      case 5: fa = frac - (rnd() & 3); fb = rnd() & 3; break;
      case 6: fb = frac - (rnd() & 3); fa = rnd() & 3; break;
      case 7: fa &= ~0xffffffffull; fb &= ~0xffffffffull; break;
      default: break;
    }
    const int eb = 1023 + (int)(rnd() % 120) - 60;
    const int gap = (i & 31) == 31 ? (int)(rnd() % 1800) - 900 : (int)(rnd() % 9) - 5;
    int ea = eb + gap;
    ea = ea < 0 ? 0 : (ea > 2046 ? 2046 : ea);
    double a = from(((uint64_t)ea << 52) | fa), b = from(((uint64_t)eb << 52) | fb);
    if ((i & 15) == 8) {   // a just beside a multiple of b's half-way quotients
      const double q = from((1023ull << 52) | fa) + 0x1p-53;
      a = std::ldexp(q * from((1023ull << 52) | fb), ea - 1023);
      b = std::ldexp(from((1023ull << 52) | fb), eb - 1023);
    }
    if (rnd() & 1) a = -a;
    if (rnd() & 1) b = -b;
    A.push_back(a);
    B.push_back(b);
  }
  const long long n = (long long)A.size();
  std::vector<double> Q(n), C(n);
  if (device) {
    double* d[4];
    for (auto& p : d)
      if (cudaMalloc(&p, n * 8) != cudaSuccess) return 2;
    cudaMemcpy(d[0], A.data(), n * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(d[1], B.data(), n * 8, cudaMemcpyHostToDevice);
    check_kernel<<<152 * 4, 256>>>(d[0], d[1], d[2], d[3], n);
    if (cudaDeviceSynchronize() != cudaSuccess) return 2;
    cudaMemcpy(Q.data(), d[2], n * 8, cudaMemcpyDeviceToHost);
    cudaMemcpy(C.data(), d[3], n * 8, cudaMemcpyDeviceToHost);
  } else {
    for (long long i = 0; i < n; i++) {
      Q[i] = div_rn(A[i], B[i]);
      C[i] = std::isfinite(A[i]) && std::isfinite(B[i]) ? limited_ratio(A[i], B[i]) : 0.0;
    }
  }
  long long bad = 0;
  for (long long i = 0; i < n; i++) {
    const double ref = A[i] / B[i];
    const double lim = std::isfinite(A[i]) && std::isfinite(B[i]) ? limiter(A[i], B[i]) : 0.0;
    if (!same(Q[i], ref) || !same(C[i], lim)) {
      if (bad++ < 10) std::printf("%a / %a: %a, want %a; limiter %a, want %a\n", A[i], B[i], Q[i], ref, C[i], lim);
    }
  }
  std::printf("%lld pairs, %lld wrong\n", n, bad);
  return bad ? 1 : 0;
}
