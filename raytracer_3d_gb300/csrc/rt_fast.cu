// rt_fast.cu -- fast binary64 step (variant RT_VARIANT_FAST): no division, no
// binary64 comparison, and the limited slopes on the integer pipes.
//
// GB300's binary64 pipe takes 19 cycles of an SM for an instruction of a warp
// (about 0.5 T operations/s in all), so the step is arranged to need few of
// them.  With the flux of a face F = v*E_up + h*psi (rt_fast.cuh) a cell's
// outgoing upwind fluxes are multiples of its own E; together with the
// mean-flow term they are one factor per cell,
//   nu = -dt*lambda - sum_a (dt/d_a)*(max(v_r, 0) - min(v_l, 0)),
// and the update (integrate.f90:105-262, regrouped) is
//   E_new = E + (nu*E + sum_a [V_in*E_in + H_l*psi_l - H_r*psi_r])
// with E_in the neighbour the axis lets in (at most one, but where two faces
// converge on the cell), V = (dt/d)*v and H = (dt/d)*h cached per face:
// three binary64 instructions per axis and two more, 20 per cell.  Fields of
// varying spacings keep V = dt*v and H = dt*h and multiply by 1/d per axis
// (one instruction more).  Results agree with the reference to a few
// units in the last place per step; the parity tests hold them to 1e-12
// relative L-infinity.
//
//   role A  psi of every right face into rings, all integer work where the
//           values of a warp lie within 2^8 of each other (superbee_near64),
//           one or two binary64 subtractions per face otherwise;
//   role B  the update.
// One launch has CTAs of role A on one slab of the field and of role B on the
// slab before in turns, so that the integer and the binary64 pipes work side
// by side, and starts while the launch ahead drains.  32x32x32x12^3 has the
// binary64 pipe 56% busy, the issue slots 60% and DRAM 67% (78% of the
// measured copy rate: the slopes leave L2 before they are read), 58 warps per
// SM; with 6, 5 and 4 CTAs per SM of more registers a step takes
// 3.4, 3.8 and 3.8 ms.  Measured per step, against two launches of fluxes (37
// binary64 instructions per cell) and update: 32x32x32x12^3 4.30 -> 3.15 ms
// (3.48 with varying spacings), 32^6 81.3 -> 61.3 ms, 18x14x20x10x12x14 677 ->
// 517 us (572).  (One launch for the whole step, its CTAs ordered by counters
// of finished chunks, measured 5.8 ms against 3.2 at 32x32x32x12^3: CTAs wait
// for one another and the slopes still go to memory.)
//
// Cached fields: H of the right faces and the face-0 planes in the handle's
// uCFL fields (recomputed when a bit-exact kernel runs next), V beside them,
// nu, and per cell the signs of its faces' velocities (16 bits).
#include <algorithm>

#include "rt_cells.cuh"
#include "rt_exact.cuh"
#include "rt_kernels.h"

namespace rt {

namespace {

// running sum with its rounding error (Knuth's two-sum)
__device__ __forceinline__ void add2(double& s, double& e, double x) {
  const double t = dadd(s, x), b = dsub(t, s);
  e = dadd(e, dadd(dsub(s, dsub(t, b)), dsub(x, b)));
  s = t;
}

// V, H, nu and the signs of every cell (bit a: V_l > 0, bit 6 + a: V_r < 0); the face-0 planes of V and H
// come from the cells at coordinate 0
__global__ void __launch_bounds__(256) fast_prepare_kernel(Dims d, Grid g, double dt, FastFields C, CellGeom G) {
  for (unsigned pu = blockIdx.x * blockDim.x + threadIdx.x; pu < G.ncell; pu += gridDim.x * blockDim.x) {
    const int p = (int)pu;
    int c[6];
    cell_coords(G, pu, c);
    double lam = 0.0;
    if (d.n[0] > 1) lam += C.lam[0][p];
    if (d.n[1] > 1) lam += C.lam[1][p];
    if (d.n[2] > 1) lam += C.lam[2][p];
    double s = -dmul(dt, lam), e = 0.0;
    unsigned signs = 0;
#pragma unroll
    for (int a = 0; a < 6; a++) {
      if (d.n[a] <= 1) continue;
      const double dr = g.d[a][pidx(c[a] + 1)];
      const double vr = C.vel[a][p];
      const double cr = div_rn(dmul(vr, dt), dr);
      const double V = C.uniform ? cr : dmul(vr, dt);
      C.V[a][p] = V;
      C.H[a][p] = 0.5 * fabs(V) * (1.0 - fabs(cr));
      if ((long long)f64_bits(vr) < 0) signs |= 64u << a;
      double vl, cl;
      if (c[a] > 0) {
        vl = C.vel[a][p - G.s[a]];
      } else {
        const int q = plane32(G, a, c);
        vl = C.vlo[a][q];
        const double c0 = div_rn(dmul(vl, dt), g.d[a][pidx(0)]);
        const double V0 = C.uniform ? c0 : dmul(vl, dt);
        C.V0[a][q] = V0;
        C.H0[a][q] = 0.5 * fabs(V0) * (1.0 - fabs(c0));
      }
      cl = div_rn(dmul(vl, dt), dr);
      if (f64_pos(vl)) signs |= 1u << a;
      if (f64_pos(vr)) add2(s, e, -cr);
      if (f64_pos(-vl)) add2(s, e, cl);
    }
    C.nu[p] = dadd(s, e);
    C.signs[p] = (unsigned short)signs;
  }
}

// 1/d of every axis on the padded index range
__global__ void fast_table_kernel(Dims d, Grid g, double* tab, long long o1, long long o2, long long o3, long long o4,
                                  long long o5) {
  const long long off[7] = {0, o1, o2, o3, o4, o5, o5 + d.n[5] + 2 * RT_ONX};
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < off[6]; i += (long long)gridDim.x * blockDim.x) {
    int a = 0;
    while (i >= off[a + 1]) a++;
    tab[i] = ddiv(1.0, g.d[a][i - off[a]]);
  }
}

// limited slope of the face between b and c, w behind the upwind side
__device__ __forceinline__ double slope(double b, double c, double w, bool pos) {
  if (__all_sync(0xffffffffu, slope_near(b, c, w))) return superbee_near64(b, c, w, pos);
  return superbee_slope64(__dsub_rn(c, b), __dsub_rn(pos ? b : w, pos ? w : c));
}

// role A, a warp's 32 consecutive cells [.., end) (the last ones repeat cell
// end - 1 and store nothing).  XW: x rows are whole segments of a warp (nx
// divides 32); the x faces then share their differences: lane x forms
// D(x) = E(x+1) - E(x) once, the upwind difference of face x+1/2 is D(x-1) or
// D(x+1) from the neighbouring lane and E(x+1) comes from the next lane too;
// beyond the row's ends the ghosts copy the edge, so D = 0 there.
template <bool XW>
__device__ __forceinline__ void fast_slopes(const Dims& d, const FastFields& C, const CellGeom& G,
                                            const double* __restrict__ E, unsigned pu, unsigned end) {
  const bool valid = pu < end;
  if (!valid) pu = end - 1;
  const int p = (int)pu;
  int c[6];
  cell_coords(G, pu, c);
  const double e0 = E[p];
  const unsigned signs = C.signs[p];
#pragma unroll
  for (int a = 0; a < 6; a++) {
    if (d.n[a] <= 1) continue;
    const int ca = c[a];
    const bool pos = !(signs >> (6 + a) & 1u);   // (a face of zero velocity has H = 0: either way)
    double psi;
    if (XW && a == 0) {
      const int nx = d.n[0];
      const double Ep1 = __shfl_down_sync(0xffffffffu, e0, 1, nx);   // the row's last lane: its own E
      const double Rj = __dsub_rn(Ep1, e0);
      const double Dm = __shfl_up_sync(0xffffffffu, Rj, 1, nx);
      const double Dp = __shfl_down_sync(0xffffffffu, Rj, 1, nx);
      psi = superbee_slope64(Rj, pos ? (ca > 0 ? Dm : 0.0) : (ca < nx - 1 ? Dp : 0.0));
    } else {
      const double Ep1 = E[nb32(d, G, p, a, ca, +1, c[5])];
      const double w = E[nb32(d, G, p, a, ca, pos ? -1 : +2, c[5])];
      psi = slope(e0, Ep1, w, pos);
    }
    if (valid) C.psi[a][pu & C.mask[a]] = psi;
    if (a == 2 && d.lower_refl && __any_sync(0xffffffffu, ca == 0)) {   // the reflected z face 0
      if (ca == 0 && valid) {
        const bool pos0 = f64_pos(C.V0[2][plane32(G, 2, c)]);
        const double b = E[nb32(d, G, p, 2, 0, -1, c[5])];
        const double w = E[nb32(d, G, p, 2, 0, pos0 ? -2 : +1, c[5])];
        C.psi0[pu & C.mask[2]] = superbee_slope64(__dsub_rn(e0, b), __dsub_rn(pos0 ? b : w, pos0 ? w : e0));
      }
    }
  }
}

// V_in: V_l, else -V_r, else 0.  As integer PTX: the sign change of a value
// that is then selected would become a binary64 instruction.
__device__ __forceinline__ double inflow(double Vl, double Vr, bool inl, bool inr) {
  double r;
  asm("{\n\t.reg .b64 l, n;\n\t.reg .pred pl, pr;\n\t"
      "setp.ne.s32 pl, %3, 0;\n\tsetp.ne.s32 pr, %4, 0;\n\t"
      "mov.b64 l, %1;\n\tmov.b64 n, %2;\n\t"
      "xor.b64 n, n, 0x8000000000000000;\n\t"
      "selp.b64 n, n, 0, pr;\n\tselp.b64 n, l, n, pl;\n\t"
      "mov.b64 %0, n;\n\t}"
      : "=d"(r)
      : "d"(Vl), "d"(Vr), "r"((int)inl), "r"((int)inr));
  return r;
}

// role B, cells as in role A.  UNI: every axis has one spacing.
template <bool UNI>
__device__ __forceinline__ void fast_update(const Dims& d, const FastFields& C, const CellGeom& G,
                                            const double* __restrict__ E, double* __restrict__ Enew, unsigned pu,
                                            unsigned end) {
  const bool valid = pu < end;
  if (!valid) pu = end - 1;
  const int p = (int)pu;
  int c[6];
  cell_coords(G, pu, c);
  const unsigned signs = C.signs[p];
  const double e0 = E[p];
  double acc = __dmul_rn(e0, __ldcs(C.nu + p));
#pragma unroll
  for (int a = 0; a < 6; a++) {
    if (d.n[a] <= 1) continue;
    const int ca = c[a];
    const bool inl = signs >> a & 1u, inr = signs >> (6 + a) & 1u;
    const double Ein = E[inl || inr ? nb32(d, G, p, a, ca, inl ? -1 : +1, c[5]) : p];
    const double Vr = a < 4 ? C.V[a][p] : __ldcs(C.V[a] + p), Hr = a < 4 ? C.H[a][p] : __ldcs(C.H[a] + p);
    const double sr = C.psi[a][pu & C.mask[a]];
    // the left face: only addresses depend on where the cell is, so that no
    // arithmetic stands in a branch (a warp would issue it for both sides).
    // What nobody reads after this, or only a long way on (l, m), goes from
    // L2 first: 3.20 -> 3.15 ms per step at 32x32x32x12^3.
    const bool in = ca > 0;
    const int q = in ? p - G.s[a] : plane32(G, a, c);
    const double Vl = __ldcs((in ? C.V[a] : C.V0[a]) + q), Hl = __ldcs((in ? C.H[a] : C.H0[a]) + q);
    const bool mirror = a == 2 && d.lower_refl;
    const double ps = __ldcs((in || !mirror ? C.psi[a] : C.psi0) + ((in ? (unsigned)q : pu) & C.mask[a]));
    const double sl = in || mirror ? ps : 0.0;
    const double Vin = inflow(Vl, Vr, inl, inr);
    double t = UNI ? __fma_rn(Vin, Ein, acc) : __dmul_rn(Vin, Ein);
    t = __fma_rn(Hl, sl, t);
    t = __fma_rn(-Hr, sr, t);
    acc = UNI ? t : __fma_rn(C.inv_d[a][pidx(ca + 1)], t, acc);
  }
  // faces that converge on the cell: its right face lets E in too
  const unsigned both = signs & (signs >> 6) & 63u;
  if (__any_sync(0xffffffffu, both != 0)) {
#pragma unroll 1
    for (int a = 0; a < 6; a++) {
      if (!(both >> a & 1u)) continue;
      int ca = 0;
#pragma unroll
      for (int b = 0; b < 6; b++) ca = b == a ? c[b] : ca;
      const double Eo = E[nb32(d, G, p, a, ca, +1, c[5])], Vr = C.V[a][p];
      acc = __fma_rn(UNI ? -Vr : __dmul_rn(-Vr, C.inv_d[a][pidx(ca + 1)]), Eo, acc);
    }
  }
  if (valid) __stcs(Enew + p, __dadd_rn(e0, acc));
}

// slab A [a0, a1): slopes, slab B [b0, b1): update; `lead` blocks of the one
// role, then the two in turns, then what is left.  The launch may start
// before the one ahead of it has ended: slopes depend on E alone, the update
// waits until that launch is complete (and with it all before it, whose
// completion its own update blocks waited for before they let this launch
// start).  Rings hold the three slabs that are then in use.
template <bool XW, bool UNI>
__global__ void __launch_bounds__(256, 7)
    fast_step_kernel(const __grid_constant__ Dims d, const __grid_constant__ FastFields C,
                     const __grid_constant__ CellGeom G, const double* __restrict__ E, double* __restrict__ Enew,
                     unsigned a0, unsigned a1, unsigned b0, unsigned b1, unsigned lead, unsigned na, unsigned nb) {
  bool slopes = true;
  unsigned blk = blockIdx.x;
  if (blk >= lead) {
    const unsigned t = blk - lead;               // update, slopes, update, ... while both last
    const unsigned turns = min(na - lead, nb);
    slopes = t < 2 * turns ? (t & 1u) != 0 : na - lead > nb;
    blk = t < 2 * turns ? t >> 1 : t - turns;
    if (slopes) blk += lead;
  }
  if (slopes) {
    asm volatile("griddepcontrol.launch_dependents;");
    fast_slopes<XW>(d, C, G, E, a0 + blk * 256 + threadIdx.x, a1);
  } else {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
    fast_update<UNI>(d, C, G, E, Enew, b0 + blk * 256 + threadIdx.x, b1);
  }
}

// Cells of a slab: whole (x,y,z) volumes, a quarter of the field within 2^19
// and 2^22, all slabs alike.  At 2^19, 2^20, 2^21 and 2^22 cells
// 32x32x32x12^3 (57 M) measured 3.43, 3.31, 3.24 and 3.20 ms per step,
// 18x14x20x10x12x14 (8.5 M) 527, 516, 512 and 520 us (the first and the last
// launch have one role only), 10x10x12x10x10x12 (1.4 M) 101, 103, 108, 108.
long long slab_cells(const Dims& d) {
  const long long want = std::min(1ll << 22, std::max(1ll << 19, d.ncell / 4));
  const long long planes = std::min((long long)d.nspec, std::max(1ll, want / d.nvol3));
  const long long slabs = (d.nspec + planes - 1) / planes;
  return (d.nspec + slabs - 1) / slabs * d.nvol3;
}
// blocks of slopes at the front of a launch: half of those the GPU holds, so
// that the blocks which wait for the launch ahead do not fill it (0, 532 and
// 1064 measured 3.40, 3.31 and 3.32 ms per step with slabs of 2^20 cells)
constexpr unsigned kLead = 152 * 7 / 2;

}  // namespace

// ring of axis a: three slabs and the stride, a power of two
long long fast_ring(const Dims& d, int a) {
  if (d.n[a] <= 1) return 0;
  const long long need = std::min(3 * slab_cells(d) + d.s[a], d.ncell);
  long long r = 1;
  while (r < need) r *= 2;
  return r;
}

// the kernels index cells with 32 bits
bool fast_ok(const Dims& d) { return d.ncell < (1ll << 31); }

cudaError_t launch_fast_prepare(const Dims& d, const Grid& g, double dt, const FastFields& C, double* tab,
                                const long long* toff, int* nlaunch, cudaStream_t st) {
  *nlaunch = 0;
  if (!fast_ok(d)) return cudaErrorInvalidValue;
  *nlaunch = 2;
  fast_prepare_kernel<<<8 * 152, 256, 0, st>>>(d, g, dt, C, make_cells(d));
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  fast_table_kernel<<<4, 256, 0, st>>>(d, g, tab, toff[1], toff[2], toff[3], toff[4], toff[5]);
  return cudaGetLastError();
}

cudaError_t launch_step_fast(const Dims& d, const FastFields& C, const double* E, double* Enew, int* nlaunch,
                             cudaStream_t st) {
  *nlaunch = 0;
  if (!fast_ok(d)) return cudaErrorInvalidValue;
  const CellGeom G = make_cells(d);
  const long long slab = slab_cells(d);
  const bool xw = d.n[0] >= 2 && 32 % d.n[0] == 0;
  auto kernel = xw ? (C.uniform ? fast_step_kernel<true, true> : fast_step_kernel<true, false>)
                   : (C.uniform ? fast_step_kernel<false, true> : fast_step_kernel<false, false>);
  // slab j takes role A beside role B of slab j - 1
  for (long long at = 0; at < d.ncell + slab; at += slab) {
    const long long a0 = std::min(at, d.ncell), a1 = std::min(at + slab, d.ncell);
    const long long b0 = std::max(0ll, at - slab), b1 = std::min(at, d.ncell);
    const unsigned na = (unsigned)((a1 - a0 + 255) / 256), nb = (unsigned)((b1 - b0 + 255) / 256);
    const unsigned lead = nb ? std::min(na, kLead) : na;
    cudaLaunchAttribute early;
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(na + nb);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cfg.attrs = &early;
    cfg.numAttrs = at > 0 ? 1 : 0;   // the first launch reads what the step before wrote
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, d, C, G, E, Enew, (unsigned)a0, (unsigned)a1, (unsigned)b0,
                                             (unsigned)b1, lead, na, nb);
    if (e != cudaSuccess) return e;
    *nlaunch += 1;
  }
  return cudaSuccess;
}

}  // namespace rt
