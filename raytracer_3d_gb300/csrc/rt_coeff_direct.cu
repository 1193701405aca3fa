// rt_coeff_direct.cu -- coefficients of a binary64 field without scratch:
// every value straight from the dispersion relation at the points it depends
// on (some 25 evaluations per cell; calc_parameter.f90:13-261, the same bits as
// rt_coeff.cu).  For fields that leave no room for three m planes of the
// relation: with nm = 2 those take up to 27 bytes per cell beside the 144 of
// the handle.  The binary64 pipe bounds it: rt_calc_parameter of 24^3x12x12x16
// takes 65.4 ms this way and 11.5 with the scratch (uCFL included in both),
// 32^3x12x12x2 20.6 and 4.4.
#include "rt_coeff.cuh"
#include "rt_kernels.h"
#include "rt_step.cuh"

namespace rt {

namespace {

// omega_e, calc_parameter.f90:21 (Fortran indices, ghosts allowed)
__device__ __forceinline__ double omega_e_at(const Background& bg, const Grid& g, const Phys& ph, const int c[6]) {
  const long long q = bg_idx(bg, c[0], c[1], c[2]);
  const double oi = omega_i_at(bg, g, ph, c[0], c[1], c[2], c[3], c[4], c[5]);
  return dadd(dadd(oi, dmul(g.kt[pidx(c[3])], bg.U[q])), dmul(g.lt[pidx(c[4])], bg.V[q]));
}

// the reference's aloc: the average of omega_e over index q and q + 1 along
// the wavenumber axis w (calc_parameter.f90:38-40, :116-118, :192-194)
__device__ __forceinline__ double aloc_at(const Background& bg, const Grid& g, const Phys& ph, const int c[6], int w) {
  int u[6];
#pragma unroll
  for (int b = 0; b < 6; b++) u[b] = c[b] + (b == w ? 1 : 0);
  return dmul(0.5, dadd(omega_e_at(bg, g, ph, c), omega_e_at(bg, g, ph, u)));
}

// velocity of axis a at its face c[a] (0..n_a), the other indices interior
__device__ __noinline__ double face_velocity(const Dims& d, const Background& bg, const Grid& g, const Phys& ph, int a,
                                             const int c[6]) {
  const int s = a < 3 ? a : a - 3, w = s + 3;   // the pair x/k, y/l or z/m
  const int f = c[a], n = d.n[a];
  if (s < 2 && !(d.n[s] > 1 && d.n[w] > 1))     // analytic on interior cells, 0 elsewhere
    return a < 3 && f >= 1 ? analytic_vel(bg, g, ph, c, s) : 0.0;
  const int other = a < 3 ? w : s;              // the difference runs along the partner axis
  int lo[6];
#pragma unroll
  for (int b = 0; b < 6; b++) lo[b] = c[b] - (b == other ? 1 : 0);
  double v = ddiv(dsub(aloc_at(bg, g, ph, c, w), aloc_at(bg, g, ph, lo, w)), g.d[other][pidx(c[other])]);
  if (a >= 3) v = -v;
  // outflow-only ends; the z walls may reflect
  if (f == n && !(a == 2 && d.upper_refl)) v = fmax2(0.0, v);
  if (f == 0 && !(a == 2 && d.lower_refl)) v = -fmax2(0.0, -v);
  return v;
}

__global__ void __launch_bounds__(128) direct_cells_kernel(Dims d, Background bg, Grid g, Phys ph,
                                                           CoeffOut<double> out) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < d.ncell; p += stride) {
    int c[6];
    long long r = p;
    for (int b = 0; b < 6; b++) {
      c[b] = (int)(r % d.n[b]) + 1;
      r /= d.n[b];
    }
    double v[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
    for (int a = 0; a < 6; a++) {
      const double x = face_velocity(d, bg, g, ph, a, c);
      out.vel[a][p] = x;
#pragma unroll
      for (int s = 0; s < 3; s++) v[s] = s == a ? x : v[s];
    }
    // growth rates, calc_parameter.f90:246-254
    const long long q = bg_idx(bg, c[0], c[1], c[2]);
    const long long st[3] = {1, bg.px, (long long)bg.px * bg.py};
    const double ktv = g.kt[pidx(c[3])], ltv = g.lt[pidx(c[4])];
    const double inv = ddiv(1.0, omega_i_at(bg, g, ph, c[0], c[1], c[2], c[3], c[4], c[5]));
    const double xu = dsub(v[0], bg.U[q]), yv = dsub(v[1], bg.V[q]);
#pragma unroll
    for (int s = 0; s < 3; s++) {
      const double d2 = dmul(2.0, g.d[s][pidx(c[s])]);
      const double dU = dsub(bg.U[q + st[s]], bg.U[q - st[s]]), dV = dsub(bg.V[q + st[s]], bg.V[q - st[s]]);
      const double head = dmul(inv, s == 0 ? ktv : (s == 1 ? ltv : v[2]));
      out.lam[s][p] = dmul(head, dadd(ddiv(dmul(s < 2 ? xu : ktv, dU), d2), ddiv(dmul(s < 2 ? yv : ltv, dV), d2)));
    }
  }
}

// the face-0 plane of axis a
__global__ void __launch_bounds__(128) direct_plane_kernel(Dims d, Background bg, Grid g, Phys ph, int a, double* out) {
  const long long n = d.ncell / d.n[a], stride = (long long)gridDim.x * blockDim.x;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += stride) {
    int c[6];
    long long r = q;
    for (int b = 0; b < 6; b++) {
      c[b] = b == a ? 0 : (int)(r % d.n[b]) + 1;
      r /= b == a ? 1 : d.n[b];
    }
    out[q] = face_velocity(d, bg, g, ph, a, c);
  }
}

// the CFL rate of the finished velocities: rates are >= 0, so their bit
// patterns order as unsigned integers
__global__ void __launch_bounds__(256) direct_rate_kernel(Dims d, Grid g, CoeffOut<double> cf, unsigned long long* rate) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  unsigned long long best = 0;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < d.ncell; p += stride) {
    int c[6];
    long long r = p;
    for (int b = 0; b < 6; b++) {
      c[b] = (int)(r % d.n[b]);
      r /= d.n[b];
    }
    double sum = 0.0;
    for (int a = 0; a < 6; a++) {
      if (d.n[a] <= 1) continue;
      const double vr = cf.vel[a][p], vl = c[a] > 0 ? cf.vel[a][p - d.s[a]] : cf.vlo[a][plane_index(d, a, c)];
      sum = dadd(sum, ddiv(fmax2(fabs(vl), fabs(vr)), g.d[a][pidx(c[a] + 1)]));
    }
    const unsigned long long b = (unsigned long long)__double_as_longlong(sum) & 0x7fffffffffffffffull;
    best = b > best ? b : best;
  }
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) {
    const unsigned long long o = __shfl_xor_sync(0xffffffffu, best, w);
    best = o > best ? o : best;
  }
  if ((threadIdx.x & 31) == 0) atomicMax(rate, best);
}

}  // namespace

cudaError_t launch_coeff_direct(const Dims& d, const Background& bg, const Grid& g, const Phys& ph,
                                const CoeffOut<double>& out, double* rate, int* nlaunch, cudaStream_t st) {
  *nlaunch = 8;
  cudaError_t e = cudaMemsetAsync(rate, 0, sizeof(double), st);
  if (e != cudaSuccess) return e;
  direct_cells_kernel<<<8 * 152, 128, 0, st>>>(d, bg, g, ph, out);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  for (int a = 0; a < 6; a++) {
    direct_plane_kernel<<<4 * 152, 128, 0, st>>>(d, bg, g, ph, a, out.vlo[a]);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  direct_rate_kernel<<<8 * 152, 256, 0, st>>>(d, g, out, reinterpret_cast<unsigned long long*>(rate));
  return cudaGetLastError();
}

}  // namespace rt
