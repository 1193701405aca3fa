// rt_coeff.cuh -- the dispersion relation and the analytic velocities of
// calc_parameter.f90, in the reference's binary64 sequence.
//
// The reference builds omega_i/omega_e on every padded cell
// (calc_parameter.f90:13-27), averages omega_e along one axis of a pair and
// then OVERWRITES that average with the average along the partner axis
// (:34-40, :112-118, :188-194), and differences the result (:44-46, :69-71,
// ...): pairs x<->k, y<->l, z<->m, the average aloc along the wavenumber;
//   spatial velocity at face f    (aloc(f, q) - aloc(f, q-1)) / d_partner(q)
//                                 over the wavenumber (:44-46, :122-124, :198-200)
//   spectral velocity at face f   -(aloc(q, f) - aloc(q-1, f)) / d_partner(q)
//                                 over the spatial partner (:69-71, :147-149, :219-221)
// then the outflow-only clamps at faces 0 and n (:55-66, :76-87, :133-144,
// :154-165, :204-216, :226-237).  A collapsed x/k or y/l pair has the
// analytic spatial velocity on interior cells, 0 elsewhere.  rt_coeff.cu
// evaluates them.
#pragma once
#include "rt_common.cuh"

namespace rt {

struct Phys {
  double f0;     // Coriolis parameter (main_module.f90:24)
  double sgn;    // sign_of_omega_i (main_module.f90:26)
  double dt;     // time step (main_module.f90:20)
};

__device__ __forceinline__ long long bg_idx(const Background& bg, int i, int j, int k) {
  return (long long)pidx(i) + (long long)bg.px * (pidx(j) + (long long)bg.py * pidx(k));
}

// omega_i, calc_parameter.f90:19-20 (Fortran indices, ghosts allowed)
__device__ __forceinline__ double omega_i_at(const Background& bg, const Grid& g, const Phys& ph,
                                             int i, int j, int k, int l, int n, int m) {
  const double ktv = g.kt[pidx(l)], ltv = g.lt[pidx(n)], mtv = g.mt[pidx(m)];
  const double kh2 = dadd(dmul(ltv, ltv), dmul(ktv, ktv));
  const double m2 = dmul(mtv, mtv);
  const double Nq = bg.Nsqr[bg_idx(bg, i, j, k)];
  const double num = dadd(dmul(Nq, kh2), dmul(dmul(ph.f0, ph.f0), m2));
  const double den = dadd(m2, kh2);
  return dmul(ph.sgn, __dsqrt_rn(ddiv(num, den)));
}

// analytic velocity of a collapsed pair, calc_parameter.f90:98 (x) / :176 (y)
__device__ __forceinline__ double analytic_vel(const Background& bg, const Grid& g, const Phys& ph,
                                               const int c[6], int which) {
  const long long q = bg_idx(bg, c[0], c[1], c[2]);
  const double ktv = g.kt[pidx(c[3])], ltv = g.lt[pidx(c[4])], mtv = g.mt[pidx(c[5])];
  const double kh2 = dadd(dmul(ltv, ltv), dmul(ktv, ktv));
  const double oi = omega_i_at(bg, g, ph, c[0], c[1], c[2], c[3], c[4], c[5]);
  const double m2 = dmul(mtv, mtv);
  const double den = dadd(m2, kh2);
  double t = ddiv(dsub(bg.Nsqr[q], dmul(ph.f0, ph.f0)), oi);
  t = dmul(t, m2);
  t = ddiv(t, dmul(den, den));
  if (which == 0) return dadd(bg.U[q], dmul(t, ktv));
  return dadd(bg.V[q], dmul(t, ltv));
}

}  // namespace rt
