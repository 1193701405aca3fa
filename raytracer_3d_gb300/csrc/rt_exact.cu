// rt_exact.cu -- bit-exact binary64 step without binary64 divisions
// (arithmetic in rt_exact.cuh), in two forms:
//
//   exact_cell_kernel    one launch, one thread per cell, both faces of every
//                        axis: small fields, where the launch and the latency
//                        of one pass are the cost;
//   exact_flux_kernel,   two passes that evaluate every face flux once, as the
//   exact_update_kernel  reference does, over slabs of the slowest axis: the
//                        flux fields of one slab stay in L2 between the passes
//                        and the scratch is one slab, not the field.
//
// Both give the bits of the other binary64 kernels and of the oracle.
//
// The bound is the binary64 pipe: 10 instructions per face flux, two per
// axis in the divergence and eight in the update, 80 per cell with six axes
// in the two passes (290 with the divisions on that pipe).  32x32x32x12^3
// measured 9.46 ms per step, 5.98 G cells/s and 478 G binary64
// instructions/s, 90% of the measured rate; the TMA plane kernel took 39.9
// ms, and a CTA of 512 threads per x-y plane 280 us for a 40x120 column
// (one launch here: 8.2 us), 6.3 ms for a 10x20x60x60 section (97 us) and
// 8.7 ms for 8x8x16x16^3 (0.74 ms).
#include "rt_exact.cuh"
#include "rt_fast.cuh"
#include "rt_kernels.h"
#include "rt_step.cuh"

namespace rt {

namespace {

// 32-bit index geometry (fields of 2^31 cells and more keep the other kernels)
struct CellGeom {
  unsigned ncell;
  int s[6];
  int ps[6][6];
  DivU32 n[5];     // divisors of the coordinates, x..l
};

CellGeom make_cells(const Dims& d) {
  CellGeom G;
  G.ncell = (unsigned)d.ncell;
  for (int a = 0; a < 6; a++) {
    G.s[a] = (int)d.s[a];
    for (int b = 0; b < 6; b++) G.ps[a][b] = (int)d.ps[a][b];
    if (a < 5) G.n[a] = make_div((unsigned)d.n[a]);
  }
  return G;
}

__device__ __forceinline__ void cell_coords(const CellGeom& G, unsigned p, int c[6]) {
  unsigned r = p;
#pragma unroll
  for (int a = 0; a < 5; a++) {
    const unsigned q = G.n[a].div(r);
    c[a] = (int)(r - q * G.n[a].d);
    r = q;
  }
  c[5] = (int)r;
}

// nb_index and plane_index in 32-bit arithmetic
__device__ __forceinline__ int nb32(const Dims& d, const CellGeom& G, int p, int a, int c, int off, int cm) {
  int flip = 0;
  const int c2 = map_coord(d, a, c + off, flip);
  int q = p + (c2 - c) * G.s[a];
  if (flip) q += ((d.n[5] - 1 - cm) - cm) * G.s[5];
  return q;
}
__device__ __forceinline__ int plane32(const CellGeom& G, int a, const int c[6]) {
  int q = 0;
#pragma unroll
  for (int b = 0; b < 6; b++) q += c[b] * G.ps[a][b];
  return q;
}

// face 0 of an axis whose lower ghosts copy the edge cell: Rj = 0 and the
// flux is v*(E0+E0)*0.5 = v*E0 exactly
__device__ __forceinline__ bool face0_is_copy(const Dims& d, int a) { return a != 2 || !d.lower_refl; }

// dE - meanfl and the update, integrate.f90:202-262
__device__ __forceinline__ double exact_update(const StepArgs<double>& A, int p, double e0, double dE) {
  const Dims& d = A.d;
  double mf = 0.;
  if (d.n[0] > 1) mf = dmul(e0, __ldcs(A.lam[0] + p));
  if (d.n[1] > 1) mf = dadd(mf, dmul(e0, __ldcs(A.lam[1] + p)));
  if (d.n[2] > 1) mf = dadd(mf, dmul(e0, __ldcs(A.lam[2] + p)));
  return dadd(e0, dmul(A.dt, dsub(dE, mf)));
}

__global__ void __launch_bounds__(128) exact_cell_kernel(StepArgs<double> A, CellGeom G) {
  const Dims& d = A.d;
  const unsigned pu = blockIdx.x * blockDim.x + threadIdx.x;
  if (pu >= G.ncell) return;
  const int p = (int)pu;
  int c[6];
  cell_coords(G, pu, c);
  const double e0 = A.E[p];
  double dE = 0.;
#pragma unroll
  for (int a = 0; a < 6; a++) {
    if (d.n[a] <= 1) continue;
    const int ca = c[a];
    const double Em1 = A.E[nb32(d, G, p, a, ca, -1, c[5])];
    const double Ep1 = A.E[nb32(d, G, p, a, ca, +1, c[5])];
    const double Ep2 = A.E[nb32(d, G, p, a, ca, +2, c[5])];
    const double fr = flux_exact(A.vel[a][p], A.uc[a][p], Em1, e0, Ep1, Ep2);
    double fl;
    if (ca > 0 || !face0_is_copy(d, a)) {
      const int q = ca > 0 ? p - G.s[a] : plane32(G, a, c);
      const double vl = ca > 0 ? A.vel[a][q] : A.vlo[a][q], ul = ca > 0 ? A.uc[a][q] : A.ucl[a][q];
      fl = flux_exact(vl, ul, A.E[nb32(d, G, p, a, ca, -2, c[5])], Em1, e0, Ep1);
    } else {
      fl = dmul(A.vlo[a][plane32(G, a, c)], e0);
    }
    dE = dsub(dE, div_rn(dsub(fr, fl), A.g.d[a][pidx(ca + 1)]));
  }
  A.Enew[p] = exact_update(A, p, e0, dE);
}

// ---- the two passes over a slab: values [c0, c0 + count) of the slowest
// axis with n > 1 (axis `ax`), which are contiguous cells [base, end) ----
struct Slab {
  unsigned base, end;   // cells
  int ax, s_ax;         // slab axis and its stride
  int ring;             // planes of the flux ring along the slab axis
  int q0;               // first entry of the slab in the face-0 plane of z
};

__device__ __forceinline__ int ring_at(const Slab& L, int p, int c) {
  return p - c * L.s_ax + (c % L.ring) * L.s_ax;
}

__global__ void __launch_bounds__(256, 4) exact_flux_kernel(StepArgs<double> A, SplitFluxes F, CellGeom G, Slab L) {
  const Dims& d = A.d;
  const unsigned pu = L.base + blockIdx.x * blockDim.x + threadIdx.x;
  if (pu >= L.end) return;
  const int p = (int)pu;
  int c[6];
  cell_coords(G, pu, c);
  const double e0 = A.E[p];
#pragma unroll
  for (int a = 0; a < 6; a++) {
    if (d.n[a] <= 1) continue;
    const int ca = c[a];
    const double Em1 = A.E[nb32(d, G, p, a, ca, -1, c[5])];
    const double Ep1 = A.E[nb32(d, G, p, a, ca, +1, c[5])];
    const double Ep2 = A.E[nb32(d, G, p, a, ca, +2, c[5])];
    const double f = flux_exact(__ldcs(A.vel[a] + p), __ldcs(A.uc[a] + p), Em1, e0, Ep1, Ep2);
    F.f[a][a == L.ax ? ring_at(L, p, ca) : p - (int)L.base] = f;
    if (ca == 0 && !face0_is_copy(d, a)) {
      const int q = plane32(G, a, c);
      F.f0[a][q - L.q0] = flux_exact(A.vlo[a][q], A.ucl[a][q], A.E[nb32(d, G, p, a, ca, -2, c[5])], Em1, e0, Ep1);
    }
  }
}

__global__ void __launch_bounds__(256, 4) exact_update_kernel(StepArgs<double> A, SplitFluxes F, CellGeom G, Slab L) {
  const Dims& d = A.d;
  const unsigned pu = L.base + blockIdx.x * blockDim.x + threadIdx.x;
  if (pu >= L.end) return;
  const int p = (int)pu;
  int c[6];
  cell_coords(G, pu, c);
  const double e0 = A.E[p];
  double dE = 0.;
#pragma unroll
  for (int a = 0; a < 6; a++) {
    if (d.n[a] <= 1) continue;
    const int ca = c[a], q = p - (int)L.base;
    const double fr = F.f[a][a == L.ax ? ring_at(L, p, ca) : q];
    double fl;
    if (ca > 0) {
      fl = F.f[a][a == L.ax ? ring_at(L, p - L.s_ax, ca - 1) : q - G.s[a]];
    } else {
      const int q0 = plane32(G, a, c);
      fl = face0_is_copy(d, a) ? dmul(A.vlo[a][q0], e0) : F.f0[a][q0 - L.q0];
    }
    dE = dsub(dE, div_rn(dsub(fr, fl), A.g.d[a][pidx(ca + 1)]));
  }
  __stcs(A.Enew + p, exact_update(A, p, e0, dE));
}

// Cells of a slab (at least one plane of the slab axis).  The flux fields of
// a slab are 48 bytes per cell: 100 MB here, 15% of a 4 M-cell field and
// nothing beside a large one.  Smaller slabs pay more launches and last
// waves: a step of 8x8x16x16^3 measured 809 us at 2^19 cells, 739 at 2^20,
// 703 at 2^22; 18x14x20x10x12x14 1587, 1587 and 1439 us.
constexpr long long kSlabCells = 1ll << 21;
// Largest field stepped in one launch, both faces of every axis per cell
// (twice the flux work, one launch less): 160x300 took 10.3 us against 14.4
// in two passes, 6x6x8x6^3 (62,208 cells) 24.8 against 24.5, 10x20x24x24
// (115,200) 26.7 against 22.6.
constexpr long long kOneLaunchCells = 1ll << 16;

int slab_axis(const Dims& d) {
  int ax = 5;
  while (ax > 0 && d.n[ax] <= 1) ax--;
  return ax;
}
}  // namespace

bool exact_in_slabs(const Dims& d) { return d.ncell > kOneLaunchCells; }

// planes of the slab axis per slab
int exact_slab_planes(const Dims& d) {
  const int ax = slab_axis(d);
  const long long plane = d.s[ax];
  long long m = kSlabCells / plane;
  if (m < 1) m = 1;
  if (m >= d.n[ax]) return d.n[ax];
  const long long slabs = (d.n[ax] + m - 1) / m;
  return (int)((d.n[ax] + slabs - 1) / slabs);
}

// doubles of flux field a (right faces), and of the face-0 plane of z
long long exact_scratch(const Dims& d, int a) {
  if (d.n[a] <= 1) return 0;
  const int ax = slab_axis(d), m = exact_slab_planes(d);
  if (a == ax) return (m == d.n[ax] ? m : m + 1LL) * d.s[ax];
  return m * d.s[ax];
}
long long exact_scratch_z0(const Dims& d) {
  if (d.n[2] <= 1 || !d.lower_refl) return 0;
  const int ax = slab_axis(d);
  return ax == 2 ? d.s[2] : exact_slab_planes(d) * (d.s[ax] / d.n[2]);
}

cudaError_t launch_step_exact_cells(const StepArgs<double>& A, cudaStream_t st) {
  exact_cell_kernel<<<(unsigned)((A.d.ncell + 127) / 128), 128, 0, st>>>(A, make_cells(A.d));
  return cudaGetLastError();
}

cudaError_t launch_step_exact_slabs(const StepArgs<double>& A, const SplitFluxes& F, cudaStream_t st, int* nlaunch) {
  const Dims& d = A.d;
  const CellGeom G = make_cells(d);
  const int ax = slab_axis(d), m = exact_slab_planes(d);
  *nlaunch = 0;
  for (int c0 = 0; c0 < d.n[ax]; c0 += m) {
    const int count = c0 + m <= d.n[ax] ? m : d.n[ax] - c0;
    Slab L;
    L.base = (unsigned)(c0 * d.s[ax]);
    L.end = (unsigned)((c0 + count) * d.s[ax]);
    L.ax = ax;
    L.s_ax = (int)d.s[ax];
    L.ring = m == d.n[ax] ? m : m + 1;
    L.q0 = ax == 2 ? 0 : (int)(c0 * (d.s[ax] / d.n[2]));
    const unsigned blocks = (L.end - L.base + 255) / 256;
    exact_flux_kernel<<<blocks, 256, 0, st>>>(A, F, G, L);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    exact_update_kernel<<<blocks, 256, 0, st>>>(A, F, G, L);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    *nlaunch += 2;
  }
  return cudaSuccess;
}

}  // namespace rt
