// rt_exact.cu -- bit-exact binary64 step without binary64 divisions
// (arithmetic in rt_exact.cuh), in two forms:
//
//   exact_small_kernel   small fields: one CTA per SM over a range of cells,
//                        fluxes through shared memory, one step or many in one
//                        launch (a grid-wide wait between them);
//   exact_flux_kernel,   two passes that evaluate every face flux once, as the
//   exact_update_kernel  reference does, over slabs of the slowest axis: the
//                        flux fields of one slab stay in L2 between the passes
//                        and the scratch is one slab, not the field.
//
// Both give the bits of the other binary64 kernels and of the oracle.
//
// The bound is the binary64 pipe: 7 instructions per face flux (10 where
// values next to each other differ by more than 2^8), two per axis in the
// divergence and seven in the update, 61 per cell with six axes in the two
// passes (290 with the divisions on that pipe).  32x32x32x12^3 measures 7.22
// ms per step, 7.8 G cells/s and 484 G binary64 instructions/s, 91% of the
// measured rate (7.57 ms with the edge fluxes as bare multiplications in a
// branch; 9.45 ms with 10 per flux); the TMA plane kernel took
// 39.9 ms, and a CTA of 512 threads per x-y plane 280 us for a 40x120 column
// (one launch here: 8.2 us), 6.3 ms for a 10x20x60x60 section (76 us) and
// 8.7 ms for 8x8x16x16^3 (0.56 ms).  The integer work (340 instructions per
// flux) wants many warps to hide behind: 32 registers and 8 resident CTAs
// with some spilling measured 7.65 ms then, 40 and 6 CTAs 7.90, 48 and 5 CTAs
// 8.15, 52 and 4 CTAs 8.40.
#include <algorithm>

#include "../../include/rt_gb300.h"
#include "rt_cells.cuh"
#include "rt_exact.cuh"
#include "rt_kernels.h"
#include "rt_step.cuh"

namespace rt {

namespace {

// dE - meanfl and the update, integrate.f90:202-262
__device__ __forceinline__ double exact_update(const StepArgs<double>& A, int p, double e0, double dE) {
  const Dims& d = A.d;
  double mf = 0.;
  if (d.n[0] > 1) mf = dmul(e0, A.lam[0][p]);
  if (d.n[1] > 1) mf = dadd(mf, dmul(e0, A.lam[1][p]));
  if (d.n[2] > 1) mf = dadd(mf, dmul(e0, A.lam[2][p]));
  return dadd(e0, dmul(A.dt, dsub(dE, mf)));
}

// ---- small fields: CTA b owns the cells [b*C, (b+1)*C) ----
// Its face fluxes go through shared memory, evaluated once: list a holds the
// left-face fluxes of the first sh = min(stride, C) cells (right-face fluxes
// of cells before the CTA's) and then the right-face fluxes of all C, so
// cell i has its left flux at i and its right flux at i + sh.  One more list
// holds the reflected z face 0 of the cells that have it.
struct SmallGeom {
  CellGeom G;
  int C;
  int axes, axis[6];             // axes with n > 1
  int sh[6], start[8];           // by position in axis[]; start[axes]: the z face-0 list, start[axes + 1]: the end
  DivU32 sdiv[6], ndiv[6];       // stride and extent of every axis
};

struct Forcing {
  int kind;                      // RT_FORCING_NONE: none between the steps
  const double* F;
  double dz;
  DivU32 s3;                     // cells of a (k,l,m) volume
};

__device__ __forceinline__ int coord(const SmallGeom& S, int a, unsigned p) {
  const unsigned q = S.sdiv[a].div(p);
  return (int)(q - S.ndiv[a].div(q) * S.ndiv[a].d);
}

// set_forcing on one cell of the bottom plane, as forcing_kernel does
__device__ __forceinline__ double forced(const StepArgs<double>& A, const Forcing& W, int p, double e) {
  const unsigned sp = W.s3.div((unsigned)p);
  const int nxy = A.d.n[0] * A.d.n[1];
  const double f = W.F[(p - (int)(sp * W.s3.d)) + (int)sp * nxy];
  if (W.kind == RT_FORCING_FLUX) return dadd(e, div_rn(dmul(A.dt, f), W.dz));
  const double w = fmax2(0.0, A.vel[2][p]);
  return dsub(e, div_rn(dmul(dmul(A.dt, w), dsub(e, f)), W.dz));
}

// all CTAs of the launch (a cooperative one) have passed their `round`-th
// call; false when the wait ran out (status raised, every CTA leaves)
__device__ __forceinline__ bool grid_wait(unsigned* counter, unsigned round, int* status, int* ok) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(counter, 1u);
    const unsigned target = round * gridDim.x;
    bool there = false;
    for (unsigned it = 0; it < (1u << 22) && !there; it++) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
      there = v >= target;
    }
    if (!there) atomicOr(status, 1);
    *ok = there ? 1 : 0;
  }
  __syncthreads();
  return *ok != 0;
}

// what a thread knows of one face flux for the whole launch
struct FaceJob {
  bool live;
  int at, q, m1, p1, p2;   // slot; cell left of the face and its neighbours
  double v, u;
};
__device__ __forceinline__ FaceJob face_job(const StepArgs<double>& A, const SmallGeom& S, int p0, int count, int j) {
  const Dims& d = A.d;
  const CellGeom& G = S.G;
  FaceJob J;
  J.live = false;
  if (j >= S.start[S.axes + 1]) return J;
  int f = 0;
  while (j >= S.start[f + 1]) f++;
  const int i = j - S.start[f];
  J.at = j;
  if (f < S.axes) {
    const int a = S.axis[f], s = G.s[a], sh = S.sh[f];
    const int owner = i < sh ? i : i - sh;               // the CTA's cell this flux is for
    const int q = i < sh ? p0 + i - s : p0 + i - sh;     // its right face
    if (owner >= count || q < 0) return J;
    const int ca = coord(S, a, (unsigned)q);
    if (i < sh && ca == d.n[a] - 1) return J;            // the owner has face 0 on its left
    const int cm = a == 2 ? coord(S, 5, (unsigned)q) : 0;
    J.q = q;
    J.m1 = nb32(d, G, q, a, ca, -1, cm);
    J.p1 = nb32(d, G, q, a, ca, +1, cm);
    J.p2 = nb32(d, G, q, a, ca, +2, cm);
    J.v = A.vel[a][q];
    J.u = A.uc[a][q];
  } else {                                               // reflected z face 0
    const int p = p0 + i;
    if (i >= count || coord(S, 2, (unsigned)p) != 0) return J;
    int c[6];
    cell_coords(G, (unsigned)p, c);
    const int r = plane32(G, 2, c);
    J.q = nb32(d, G, p, 2, 0, -1, c[5]);
    J.m1 = nb32(d, G, p, 2, 0, -2, c[5]);
    J.p1 = p;
    J.p2 = nb32(d, G, p, 2, 0, +1, c[5]);
    J.v = A.vlo[2][r];
    J.u = A.ucl[2][r];
  }
  J.live = true;
  return J;
}
__device__ __forceinline__ void face_run(const FaceJob& J, const double* E, double* sF) {
  if (!J.live) return;
  sF[J.at] = flux_exact(J.v, J.u, __ldcg(E + J.m1), __ldcg(E + J.q), __ldcg(E + J.p1), __ldcg(E + J.p2));
}

// and of one cell: its axes' spacing, and the slots of its two fluxes (left
// -1: v*E with the face-0 velocity)
template <int AX>
struct CellJob {
  bool live, bottom;
  int p;
  int right[AX], left[AX];
  double dd[AX], v0[AX], lam[3];
};
template <int AX>
__device__ __forceinline__ CellJob<AX> cell_job(const StepArgs<double>& A, const SmallGeom& S, int p0, int count, int i) {
  const Dims& d = A.d;
  CellJob<AX> J;
  J.live = i < count;
  if (!J.live) return J;
  J.p = p0 + i;
  int c[6];
  cell_coords(S.G, (unsigned)J.p, c);
  J.bottom = c[2] == 0;
#pragma unroll
  for (int f = 0; f < AX; f++) {
    if (f >= S.axes) break;
    const int a = S.axis[f];
    int ca = 0;
#pragma unroll
    for (int b = 0; b < 6; b++) ca = b == a ? c[b] : ca;
    J.right[f] = S.start[f] + S.sh[f] + i;
    J.left[f] = ca > 0 ? S.start[f] + i : (face0_is_copy(d, a) ? -1 : S.start[S.axes] + i);
    J.v0[f] = J.left[f] < 0 ? A.vlo[a][plane32(S.G, a, c)] : 0.0;
    J.dd[f] = A.g.d[a][pidx(ca + 1)];
  }
#pragma unroll
  for (int k = 0; k < 3; k++) J.lam[k] = d.n[k] > 1 ? A.lam[k][J.p] : 0.0;
  return J;
}
template <int AX>
__device__ __forceinline__ void cell_run(const StepArgs<double>& A, const SmallGeom& S, const Forcing& W,
                                         const CellJob<AX>& J, const double* E, double* En, const double* sF,
                                         bool force) {
  if (!J.live) return;
  const Dims& d = A.d;
  const double e0 = __ldcg(E + J.p);
  double fl[AX], q[AX];   // the axes' quotients do not depend on one another
  bool easy = mid_range(split64(e0));
#pragma unroll
  for (int f = 0; f < AX; f++) {
    if (f >= S.axes) break;
    fl[f] = J.left[f] >= 0 ? sF[J.left[f]] : dmul(J.v0[f], e0);
    easy = easy && mid_range(split64(J.v0[f]));
  }
  if (!easy) {   // one branch to face0_flux's slow path, ahead of the quotients, for one
                 // per axis among them: 40x120 columns 188 -> 186 us per 50 steps, a host
                 // step of 7x5x6x4x4x4 36.3 -> 35.4 us
#pragma unroll
    for (int f = 0; f < AX; f++) {
      if (f >= S.axes) break;
      if (J.left[f] < 0) fl[f] = face0_flux(J.v0[f], e0);
    }
  }
#pragma unroll
  for (int f = 0; f < AX; f++) {
    if (f >= S.axes) break;
    q[f] = div_rn(dsub(sF[J.right[f]], fl[f]), J.dd[f]);
  }
  double dE = 0.;
#pragma unroll
  for (int f = 0; f < AX; f++) {
    if (f >= S.axes) break;
    dE = dsub(dE, q[f]);
  }
  double mf = 0.;
  if (d.n[0] > 1) mf = dmul(e0, J.lam[0]);
  if (d.n[1] > 1) mf = dadd(mf, dmul(e0, J.lam[1]));
  if (d.n[2] > 1) mf = dadd(mf, dmul(e0, J.lam[2]));
  double e = dadd(e0, dmul(A.dt, dsub(dE, mf)));
  if (force && J.bottom) e = forced(A, W, J.p, e);
  En[J.p] = e;
}

// nsteps steps from A.E (and back and forth between the two buffers); with
// more than one the launch is cooperative and `counter` starts at zero.  The
// forcing acts before every step: on A.E at the start, then on each new
// state but the last as it is stored.
// K > 0: a thread has at most K faces and one cell (and the field at most AX
// axes), whose indices and coefficients it keeps in registers from step to
// step; K = 0: it works them out anew.
template <int K, int AX>
__global__ void __launch_bounds__(512) exact_small_kernel(const __grid_constant__ StepArgs<double> A,
                                                          const __grid_constant__ SmallGeom S,
                                                          const __grid_constant__ Forcing W, int nsteps,
                                                          unsigned* counter) {
  extern __shared__ double sF[];
  __shared__ int ok;
  const int p0 = (int)blockIdx.x * S.C;
  const int count = (int)S.G.ncell - p0 < S.C ? (int)S.G.ncell - p0 : S.C;
  double* E = const_cast<double*>(A.E);
  double* En = A.Enew;
  unsigned round = 0;
  const bool forcing = W.kind != RT_FORCING_NONE;
  FaceJob face[K > 0 ? K : 1];
  CellJob<AX> cell;
  if constexpr (K > 0) {
#pragma unroll
    for (int k = 0; k < K; k++) face[k] = face_job(A, S, p0, count, (int)(threadIdx.x + k * blockDim.x));
    cell = cell_job<AX>(A, S, p0, count, (int)threadIdx.x);
  }
  if (nsteps > 1 && forcing) {
    for (int i = threadIdx.x; i < count; i += blockDim.x)
      if (coord(S, 2, (unsigned)(p0 + i)) == 0) E[p0 + i] = forced(A, W, p0 + i, E[p0 + i]);
    if (!grid_wait(counter, ++round, A.status, &ok)) return;
  }
  for (int t = 0; t < nsteps; t++) {
    const bool force = forcing && t + 1 < nsteps;
    if constexpr (K > 0) {
#pragma unroll
      for (int k = 0; k < K; k++) face_run(face[k], E, sF);
      __syncthreads();
      cell_run<AX>(A, S, W, cell, E, En, sF, force);
    } else {
      for (int j = threadIdx.x; j < S.start[S.axes + 1]; j += blockDim.x) face_run(face_job(A, S, p0, count, j), E, sF);
      __syncthreads();
      for (int i = threadIdx.x; i < count; i += blockDim.x)
        cell_run<AX>(A, S, W, cell_job<AX>(A, S, p0, count, i), E, En, sF, force);
    }
    if (t + 1 == nsteps) return;
    if (!grid_wait(counter, ++round, A.status, &ok)) return;
    double* x = E;
    E = En;
    En = x;
  }
}

// ---- the two passes over a slab: values [c0, c0 + count) of the slowest
// axis with n > 1 (axis `ax`), which are contiguous cells [base, end) ----
struct Slab {
  unsigned base, end;   // cells
  int ax, s_ax;         // slab axis and its stride
  int ring;             // planes of the flux ring along the slab axis
  int q0;               // first entry of the slab in the face-0 plane of z
  int c0, c1;           // values of the slab axis
};

__device__ __forceinline__ int ring_at(const Slab& L, int p, int c) {
  return p - c * L.s_ax + (c % L.ring) * L.s_ax;
}

// uCFL of a face, |v*dt/d| (superbee_fluxes.f90:19), where no cached one is at hand
__device__ __forceinline__ double face_ucfl(const StepArgs<double>& A, int a, int f, double v) {
  return fabs(div_rn(dmul(v, A.dt), A.g.d[a][pidx(f)]));
}

// 0 - q, on the integer pipes
__device__ __forceinline__ double zero_minus(double q) {
  const Bits64 b = split64(q);
  return __hiloint2double((int)(is_zero(b) ? 0u : b.hi ^ 0x80000000u), (int)b.lo);
}

// the launches of a step come one upon the other: a launch gets its blocks
// ready while the one ahead drains, and each block waits until that one is
// complete (a no-op where the launch was not told so)
__device__ __forceinline__ void after_launch_ahead() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
}

// CACHED: uc holds the uCFL (it holds the fast step's h otherwise)
template <bool CACHED>
__global__ void __launch_bounds__(256, 8) exact_flux_kernel(StepArgs<double> A, SplitFluxes F, CellGeom G, Slab L) {
  after_launch_ahead();
  const Dims& d = A.d;
  unsigned pu = L.base + blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = pu < L.end;
  if (!valid) pu = L.end - 1;   // whole warps vote below
  const int p = (int)pu;
  int c[6];
  cell_coords(G, pu, c);
  const double e0 = A.E[p];
#pragma unroll
  for (int a = 0; a < 6; a++) {
    if (d.n[a] <= 1) continue;
    const int ca = c[a];
    const double v = __ldcs(A.vel[a] + p);
    const double u = CACHED ? __ldcs(A.uc[a] + p) : face_ucfl(A, a, ca + 1, v);
    const bool pos = f64_pos(v);
    const double Ep1 = A.E[nb32(d, G, p, a, ca, +1, c[5])];
    const double w = A.E[nb32(d, G, p, a, ca, pos ? -1 : +2, c[5])];
    double f;
    if (__all_sync(0xffffffffu, flux_is_near(v, u, e0, Ep1, w))) f = flux_near(v, u, e0, Ep1, w, pos);
    else f = flux_exact(v, u, w, e0, Ep1, w);
    if (valid) F.f[a][a == L.ax ? ring_at(L, p, ca) : p - (int)L.base] = f;
    if (ca == 0 && valid && !face0_is_copy(d, a)) {
      const int q = plane32(G, a, c);
      const double v0 = A.vlo[a][q], u0 = CACHED ? A.ucl[a][q] : face_ucfl(A, a, 0, v0);
      F.f0[a][q - L.q0] = flux_exact(v0, u0, A.E[nb32(d, G, p, a, ca, -2, c[5])],
                                     A.E[nb32(d, G, p, a, ca, -1, c[5])], e0, Ep1);
    }
  }
}

__global__ void __launch_bounds__(256, 8) exact_update_kernel(StepArgs<double> A, SplitFluxes F, CellGeom G, Slab L) {
  after_launch_ahead();
  const Dims& d = A.d;
  const unsigned pu = L.base + blockIdx.x * blockDim.x + threadIdx.x;
  if (pu >= L.end) return;
  const int p = (int)pu;
  int c[6];
  cell_coords(G, pu, c);
  const double e0 = A.E[p];
  double dE = 0.;
  bool first = true;
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
      fl = face0_is_copy(d, a) ? face0_flux(A.vlo[a][q0], e0) : F.f0[a][q0 - L.q0];
    }
    const double quo = div_rn(dsub(fr, fl), A.g.d[a][pidx(ca + 1)]);
    dE = first ? zero_minus(quo) : dsub(dE, quo);
    first = false;
  }
  __stcs(A.Enew + p, exact_update(A, p, e0, dE));
}

// Cells of a slab (at least one plane of the slab axis).  The flux fields of
// a slab are 48 bytes per cell: 100 MB here, 15% of a 4 M-cell field and
// nothing beside a large one.  Smaller slabs pay more launches and last
// waves: a step of 8x8x16x16^3 measured 809 us at 2^19 cells, 739 at 2^20,
// 703 at 2^22; 18x14x20x10x12x14 1587, 1587 and 1439 us.
constexpr long long kSlabCells = 1ll << 21;
// Blocks from which on the flux launch, too, gets ready beside the launch ahead.
// A step of 10x20x60x60 (2813 blocks) measured 83.1 us with neither, 82.2
// with the update's and 78.9 with both, 16x32x30x32 (1920) 57.7, 57.3 and
// 53.8; of smaller ones some lose: 10x20x30x40 (938) 36.9, 34.8 and 36.4,
// 5x6x7x12x10x8 (788) 43.7, 41.2 and 49.5, 10x20x24x24 (450) 20.5, 18.5 and
// 16.7.  32x32x32x12^3: 7.65 and 7.57 ms.  (Fluxes and update of neighbouring
// slabs side by side in one launch, as the fast step has them: 7.84 ms, and
// three slabs of scratch.)
constexpr unsigned kReadyBlocks = 1024;
// Largest field stepped in one launch.  us per step in one launch / in two
// passes, as single steps and, behind the comma, in a run of 200: 160x300
// 10.3 / 12.3, 8.0 / 12.3; 64x1024 12.3 / 12.3, 9.0 / 12.3; 6x6x8x6^3 (62,208
// cells) 24.0 / 20.5, 21.1 / 22.5; 4^3x8^2x16 (65,536) 24.6 / 21.3, 21.6 / 22.5;
// 100x1000 16.4 / 14.4, 13.5 / 14.4.  Just beyond the line a CTA's lists of a 6D
// field no longer fit 48 KB, the CTAs take two rounds, and 4^3x8^2x20 (81,920)
// measures 45 / 24.6, 45 / 26.7.
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

// cells per CTA: one CTA per SM, so that the binary64 work spreads evenly;
// fewer where the face lists would outgrow the 48 KB of shared memory that a
// launch may have without asking (GPUs of less than 139 SMs).  Asking is by an
// attribute of the kernel that all handles and host threads share.
int exact_small_cells(const Dims& d, int sms) {
  int lists = 1;   // slots per cell: two per active axis, one for the z face 0
  for (int a = 0; a < 6; a++) lists += d.n[a] > 1 ? 2 : 0;
  const int most = (48 * 1024 - 64) / 8 / lists;
  return (int)std::min<long long>(most, (d.ncell + sms - 1) / sms);
}

namespace {

SmallGeom make_small(const Dims& d, int sms) {
  SmallGeom S;
  S.G = make_cells(d);
  S.C = exact_small_cells(d, sms);
  S.axes = 0;
  int at = 0;
  for (int a = 0; a < 6; a++) {
    S.sdiv[a] = make_div((unsigned)d.s[a]);
    S.ndiv[a] = make_div((unsigned)d.n[a]);
    if (d.n[a] <= 1) continue;
    const int f = S.axes++;
    S.axis[f] = a;
    S.sh[f] = d.s[a] < S.C ? (int)d.s[a] : S.C;
    S.start[f] = at;
    at += S.sh[f] + S.C;
  }
  S.start[S.axes] = at;
  if (d.n[2] > 1 && d.lower_refl) at += S.C;
  S.start[S.axes + 1] = at;
  return S;
}

int sm_count() {
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n;
}

}  // namespace

cudaError_t launch_step_exact_small(const StepArgs<double>& A, int nsteps, int forcing, const double* F, double dz,
                                    unsigned* counter, cudaStream_t st) {
  const SmallGeom S = make_small(A.d, sm_count());
  const int jobs = S.start[S.axes + 1];
  const int threads = jobs <= 128 ? 128 : (jobs <= 256 ? 256 : 512);
  const size_t sm = (size_t)jobs * sizeof(double);
  Forcing W{forcing, F, dz, make_div((unsigned)A.d.s[3])};
  const unsigned ctas = (unsigned)((A.d.ncell + S.C - 1) / S.C);
  // many steps keep what they know where it fits: fields of two active axes
  // (columns, whose steps are all latency)
  void (*kernel)(StepArgs<double>, SmallGeom, Forcing, int, unsigned*) = exact_small_kernel<0, 6>;
  if (nsteps > 1 && S.axes <= 2 && S.C <= threads) {
    if (jobs <= threads) kernel = exact_small_kernel<1, 2>;
    else if (jobs <= 2 * threads) kernel = exact_small_kernel<2, 2>;
  }
  if (nsteps == 1) {
    kernel<<<ctas, threads, sm, st>>>(A, S, W, 1, nullptr);
    return cudaGetLastError();
  }
  cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(unsigned), st);
  if (e != cudaSuccess) return e;
  StepArgs<double> a = A;
  SmallGeom s = S;
  void* args[] = {&a, &s, &W, &nsteps, &counter};
  return cudaLaunchCooperativeKernel((const void*)kernel, dim3(ctas), dim3((unsigned)threads), args, sm, st);
}

namespace {

// values [c0, c0 + m) of axis ax
Slab make_slab(const Dims& d, int ax, int m, int c0) {
  const int count = c0 + m <= d.n[ax] ? m : d.n[ax] - c0;
  Slab L;
  L.base = (unsigned)(c0 * d.s[ax]);
  L.end = (unsigned)((c0 + count) * d.s[ax]);
  L.ax = ax;
  L.s_ax = (int)d.s[ax];
  L.ring = m == d.n[ax] ? m : m + 1;
  L.q0 = ax == 2 ? 0 : (int)(c0 * (d.s[ax] / d.n[2]));
  L.c0 = c0;
  L.c1 = c0 + count;
  return L;
}

}  // namespace

cudaError_t launch_step_exact_slabs(const StepArgs<double>& A, const SplitFluxes& F, cudaStream_t st, int* nlaunch) {
  const Dims& d = A.d;
  const CellGeom G = make_cells(d);
  const int ax = slab_axis(d), m = exact_slab_planes(d);
  *nlaunch = 0;
  for (int c0 = 0; c0 < d.n[ax]; c0 += m) {
    const Slab L = make_slab(d, ax, m, c0);
    const unsigned blocks = (L.end - L.base + 255) / 256;
    cudaLaunchAttribute ready;
    ready.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    ready.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cfg.attrs = &ready;
    cfg.numAttrs = blocks >= kReadyBlocks ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, exact_flux_kernel<true>, A, F, G, L);
    cfg.numAttrs = 1;
    if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, exact_update_kernel, A, F, G, L);
    if (e != cudaSuccess) return e;
    *nlaunch += 2;
  }
  return cudaSuccess;
}

// ---------------------------------------------------------------------------
// energy budget (diagnose.f90:46-277) of the step from A.E to Ecur, over the
// same slabs: the fluxes once per face, then
//   budget_cells_kernel   per cell dE and meanfl as the update forms them, the
//                         scalar sums and maxima, and the terms of E_int and
//                         meanfl_int (products of the reference's order);
//   budget_tail_kernel    the boundary-flux sums, and beside them the eight
//                         wavenumber integrals of every spatial cell, each a
//                         chain of additions in the reference's order.
// The fluxes and cells are bound by the binary64 pipe (about 105 instructions
// per cell).  A chain is bound by the 64 cycles that a binary64 instruction
// takes a warp whatever its lanes do, so it adds and does nothing else that
// could be done elsewhere.
// ---------------------------------------------------------------------------
namespace {

constexpr int kBudgetBlocks = 8 * 152;

// max of two non-negative doubles by their bits (NaN above all)
__device__ __forceinline__ double max_bits(double a, double b) {
  const unsigned long long x = (unsigned long long)__double_as_longlong(a), y = (unsigned long long)__double_as_longlong(b);
  return x > y ? a : b;
}

__global__ void __launch_bounds__(256, 3) budget_cells_kernel(StepArgs<double> A, const double* __restrict__ Ecur,
                                                              SplitFluxes F, CellGeom G, Slab L,
                                                              double* __restrict__ te, double* __restrict__ tm,
                                                              double* __restrict__ partial) {
  __shared__ double red[8][DIAG_CELL_NV];
  const Dims& d = A.d;
  double acc[DIAG_CELL_NV];
#pragma unroll
  for (int k = 0; k < DIAG_CELL_NV; k++) acc[k] = 0.0;
  for (unsigned pu = L.base + blockIdx.x * blockDim.x + threadIdx.x; pu < L.end; pu += gridDim.x * blockDim.x) {
    const int p = (int)pu, q = p - (int)L.base;
    int c[6];
    cell_coords(G, pu, c);
    const double e0 = A.E[p];
    double dE = 0., w[6];
#pragma unroll
    for (int a = 0; a < 6; a++) {
      const int ca = c[a];
      w[a] = A.g.d[a][pidx(ca + 1)];
      acc[3 + a] = max_bits(acc[3 + a], fabs(__ldcs(A.vel[a] + p)));
      if (d.n[a] <= 1) continue;
      const double fr = F.f[a][a == L.ax ? ring_at(L, p, ca) : q];
      double fl;
      if (ca > 0) {
        fl = F.f[a][a == L.ax ? ring_at(L, p - L.s_ax, ca - 1) : q - G.s[a]];
      } else {
        const int q0 = plane32(G, a, c);
        fl = face0_is_copy(d, a) ? face0_flux(A.vlo[a][q0], e0) : F.f0[a][q0 - L.q0];
      }
      dE = dsub(dE, div_rn(dsub(fr, fl), w[a]));
    }
    double mf = 0.;
    if (d.n[0] > 1) mf = dmul(e0, __ldcs(A.lam[0] + p));
    if (d.n[1] > 1) mf = dadd(mf, dmul(e0, __ldcs(A.lam[1] + p)));
    if (d.n[2] > 1) mf = dadd(mf, dmul(e0, __ldcs(A.lam[2] + p)));
    double vol = w[0];
#pragma unroll
    for (int a = 1; a < 6; a++) vol = dmul(vol, w[a]);
    acc[0] = dadd(acc[0], dmul(dsub(dE, mf), vol));
    acc[1] = dadd(acc[1], dmul(mf, vol));
    const double ec = Ecur[p];
    const Bits64 eb = split64(ec);
    const long long ebits = (long long)(((uint64_t)eb.hi << 32) | eb.lo);
    const double floor_e = ebits > __double_as_longlong(RT_LIT_1EM12) ? ec : RT_LIT_1EM12;   // diagnose.f90:56
    acc[2] = max_bits(acc[2], div_rn(fabs(mf), floor_e));
    te[q] = dmul(dmul(dmul(ec, w[4]), w[5]), w[3]);   // E*dlt*dmt*dkt, diagnose.f90:90
    tm[q] = dmul(dmul(dmul(mf, w[3]), w[4]), w[5]);
  }
  // block partials in a fixed order: lanes, then warps; they add to those of
  // the slabs before
#pragma unroll
  for (int k = 0; k < DIAG_CELL_NV; k++) {
    double x = acc[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double y = __shfl_down_sync(0xffffffffu, x, o);
      x = k < 2 ? dadd(x, y) : max_bits(x, y);
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][k] = x;
  }
  __syncthreads();
  if (threadIdx.x < DIAG_CELL_NV) {
    const int k = threadIdx.x;
    double* out = partial + (long long)blockIdx.x * DIAG_CELL_NV + k;
    double x = L.base == 0 ? red[0][k] : (k < 2 ? dadd(*out, red[0][k]) : max_bits(*out, red[0][k]));
    for (int wi = 1; wi < 8; wi++) x = k < 2 ? dadd(x, red[wi][k]) : max_bits(x, red[wi][k]);
    *out = x;
  }
}

// flux through face 0 (hi = false) or face n of axis a at the boundary cell p
template <int a>
__device__ __forceinline__ double face_at(const StepArgs<double>& A, const SplitFluxes& F, const CellGeom& G,
                                          const Slab& L, bool hi, int p, const int c[6]) {
  if (hi) return F.f[a][a == L.ax ? ring_at(L, p, c[a]) : p - (int)L.base];
  const int q0 = plane32(G, a, c);
  return face0_is_copy(A.d, a) ? face0_flux(A.vlo[a][q0], A.E[p]) : F.f0[a][q0 - L.q0];
}

// a thread's share of the boundary sum through face 0 / n of axis a
template <int a>
__device__ __forceinline__ double plane_share(const StepArgs<double>& A, const SplitFluxes& F, const CellGeom& G,
                                              const Slab& L, bool hi, unsigned blk, unsigned nblk) {
  const Dims& d = A.d;
  const int cb = hi ? d.n[a] - 1 : 0;
  double acc = 0.0;
  if (d.n[a] <= 1 || (a == L.ax && (cb < L.c0 || cb >= L.c1))) return acc;
  // boundary cells of the slab: the slab's cells with axis a at cb
  const unsigned cells = a == L.ax ? (unsigned)L.s_ax : (L.end - L.base) / (unsigned)d.n[a];
  const unsigned s = (unsigned)G.s[a];
  for (unsigned q = blk * blockDim.x + threadIdx.x; q < cells; q += nblk * blockDim.x) {
    const unsigned p = a == L.ax ? (unsigned)cb * s + q
                                 : L.base + (q / s) * (s * (unsigned)d.n[a]) + (unsigned)cb * s + q % s;
    int c[6];
    cell_coords(G, p, c);
    double area = 0.0;
    bool first = true;
#pragma unroll
    for (int b = 0; b < 6; b++) {
      if (b == a) continue;
      const double db = A.g.d[b][pidx(c[b] + 1)];
      area = first ? db : dmul(area, db);
      first = false;
    }
    acc = dadd(acc, dmul(face_at<a>(A, F, G, L, hi, (int)p, c), area));
  }
  return acc;
}

// block b of nblk of boundary `which` = 2*axis + (0: face 0, 1: face n);
// partial layout [axis][block][2]
__device__ __forceinline__ void budget_planes(const StepArgs<double>& A, const SplitFluxes& F, const CellGeom& G,
                                              const Slab& L, int which, unsigned b, unsigned nblk, double* partial,
                                              double red[4]) {
  const int a = which >> 1;
  const bool hi = which & 1;
  double acc = a == 0   ? plane_share<0>(A, F, G, L, hi, b, nblk)
               : a == 1 ? plane_share<1>(A, F, G, L, hi, b, nblk)
               : a == 2 ? plane_share<2>(A, F, G, L, hi, b, nblk)
               : a == 3 ? plane_share<3>(A, F, G, L, hi, b, nblk)
               : a == 4 ? plane_share<4>(A, F, G, L, hi, b, nblk)
                        : plane_share<5>(A, F, G, L, hi, b, nblk);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc = dadd(acc, __shfl_down_sync(0xffffffffu, acc, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double* out = partial + ((long long)a * nblk + b) * 2 + (hi ? 1 : 0);
    double x = L.base == 0 ? 0.0 : *out;
    for (int w = 0; w < 4; w++) x = dadd(x, red[w]);
    *out = x;
  }
}

// diss_{a}s / diss_{a}e of a spatial cell: the boundary fluxes over the two
// other spectral axes, the slower one outside (diagnose.f90:186-277)
template <int a>
__device__ __forceinline__ double diss_chain(const StepArgs<double>& A, const SplitFluxes& F, const CellGeom& G,
                                             const Slab& L, bool hi, int v3, double acc) {
  const Dims& d = A.d;
  const int cb = hi ? d.n[a] - 1 : 0;
  if (d.n[a] <= 1 || (a == L.ax && (cb < L.c0 || cb >= L.c1))) return acc;
  constexpr int b1 = a == 3 ? 4 : 3, b2 = a == 5 ? 4 : 5;
  int c[6];
  cell_coords(G, (unsigned)v3, c);
  c[a] = cb;
  const int lo1 = b1 == L.ax ? L.c0 : 0, hi1 = b1 == L.ax ? L.c1 : d.n[b1];
  const int lo2 = b2 == L.ax ? L.c0 : 0, hi2 = b2 == L.ax ? L.c1 : d.n[b2];
  const bool copy = !hi && face0_is_copy(d, a);   // edge fluxes, which are stored nowhere
  for (int i2 = lo2; i2 < hi2; i2++) {
    c[b2] = i2;
    const double w2 = A.g.d[b2][pidx(i2 + 1)];
    if (!copy) {
#pragma unroll 4
      for (int i1 = lo1; i1 < hi1; i1++) {
        c[b1] = i1;
        const int p = v3 + c[3] * G.s[3] + c[4] * G.s[4] + c[5] * G.s[5];
        acc = dadd(acc, dmul(dmul(face_at<a>(A, F, G, L, hi, p, c), A.g.d[b1][pidx(i1 + 1)]), w2));
      }
      continue;
    }
    // four at a time, so that the loads of all stand before the one branch to
    // face0_flux's slow path: a budget of 8x5x13x4x8x16 takes 164 us, 174 with a
    // branch per value (160 without any), one of 8x8x16x16^3 1216 and 1208 (1267)
    constexpr int U = 4;
    for (int i1 = lo1; i1 < hi1; i1 += U) {
      double v[U], e[U], f[U];
      bool easy = true;
#pragma unroll
      for (int k = 0; k < U; k++) {
        c[b1] = i1 + k < hi1 ? i1 + k : hi1 - 1;
        v[k] = A.vlo[a][plane32(G, a, c)];
        e[k] = A.E[v3 + c[3] * G.s[3] + c[4] * G.s[4] + c[5] * G.s[5]];
        easy = easy && mid_range(split64(v[k])) && mid_range(split64(e[k]));
      }
#pragma unroll
      for (int k = 0; k < U; k++) f[k] = dmul(v[k], e[k]);
      if (!easy) {
#pragma unroll
        for (int k = 0; k < U; k++) f[k] = face0_flux(v[k], e[k]);
      }
#pragma unroll
      for (int k = 0; k < U; k++)
        if (i1 + k < hi1) acc = dadd(acc, dmul(dmul(f[k], A.g.d[b1][pidx(i1 + k + 1)]), w2));
    }
  }
  return acc;
}

// 32 spatial cells (group `g` of them) and the integral f: E_int, meanfl_int,
// diss_ks, diss_ke, diss_ls, diss_le, diss_ms, diss_me; carried from slab to
// slab in out
__device__ __forceinline__ void budget_chain(const StepArgs<double>& A, const SplitFluxes& F, const CellGeom& G,
                                             const Slab& L, const double* __restrict__ te,
                                             const double* __restrict__ tm, unsigned g, int f, double* out) {
  const unsigned nvol3 = (unsigned)A.d.nvol3;
  const unsigned v3 = g * 32 + (threadIdx.x & 31);
  if (v3 >= nvol3) return;
  if (L.ax < 3 && (v3 < L.base || v3 >= L.end)) return;   // a slab of space holds whole spatial cells
  const bool fresh = L.ax < 3 || L.base == 0;
  double acc = fresh ? 0.0 : out[(long long)f * nvol3 + v3];
  if (f < 2) {
    const double* t = (f == 0 ? te : tm) + (L.ax < 3 ? v3 - L.base : v3);
    const int n = L.ax < 3 ? 1 : (int)((L.end - L.base) / nvol3);
    constexpr int U = 16;
    int i = 0;
    double x[U];
    if (n >= U) {
#pragma unroll
      for (int k = 0; k < U; k++) x[k] = __ldcg(t + (long long)k * nvol3);
      for (; i + 2 * U <= n; i += U) {
        double y[U];
#pragma unroll
        for (int k = 0; k < U; k++) y[k] = __ldcg(t + (long long)(i + U + k) * nvol3);
#pragma unroll
        for (int k = 0; k < U; k++) acc = dadd(acc, x[k]);
#pragma unroll
        for (int k = 0; k < U; k++) x[k] = y[k];
      }
#pragma unroll
      for (int k = 0; k < U; k++) acc = dadd(acc, x[k]);
      i += U;
    }
    for (; i < n; i++) acc = dadd(acc, __ldcg(t + (long long)i * nvol3));
  } else if (f < 4) {
    acc = diss_chain<3>(A, F, G, L, f & 1, (int)v3, acc);
  } else if (f < 6) {
    acc = diss_chain<4>(A, F, G, L, f & 1, (int)v3, acc);
  } else {
    acc = diss_chain<5>(A, F, G, L, f & 1, (int)v3, acc);
  }
  out[(long long)f * nvol3 + v3] = acc;
}

// blocks [0, 2*groups): the chains of 32 spatial cells, four integrals each,
// one a warp (the four schedulers' binary64 paths are separate: 76 cycles an
// instruction for four warps, 64 for one, 128 for two on one scheduler); the
// others the boundary sums, which fill the pipe beside them
__global__ void __launch_bounds__(128) budget_tail_kernel(StepArgs<double> A, SplitFluxes F, CellGeom G, Slab L,
                                                          const double* __restrict__ te, const double* __restrict__ tm,
                                                          unsigned groups, unsigned nblk, double* vol3,
                                                          double* partial) {
  __shared__ double red[4];
  const unsigned b = blockIdx.x;
  if (b < 2 * groups)
    budget_chain(A, F, G, L, te, tm, b >> 1, (int)((b & 1) + 2 * (threadIdx.x >> 5)), vol3);
  else
    budget_planes(A, F, G, L, (int)((b - 2 * groups) / nblk), (b - 2 * groups) % nblk, nblk, partial, red);
}

}  // namespace

long long budget_terms(const Dims& d) { return 2 * exact_slab_planes(d) * d.s[slab_axis(d)]; }

cudaError_t launch_budget_exact(const StepArgs<double>& A, const double* Ecur, const SplitFluxes& F, bool ucfl_cached,
                                double* terms, double* scratch, double* vol3, double* result, int* nlaunch,
                                cudaStream_t st) {
  const Dims& d = A.d;
  const CellGeom G = make_cells(d);
  const int ax = slab_axis(d), m = exact_slab_planes(d);
  const DiagSizes sizes = diag_sizes(d);
  double* te = terms;
  double* tm = terms + budget_terms(d) / 2;
  const unsigned cb = (unsigned)std::min<long long>(kBudgetBlocks, (std::min<long long>(m * d.s[ax], d.ncell) + 255) / 256);
  const unsigned pb = (unsigned)std::min<long long>(sizes.plane_blocks, (m * d.s[ax] + 1023) / 1024);
  const unsigned groups = (unsigned)((d.nvol3 + 31) / 32);
  double* pc = scratch;
  double* pp = scratch + (long long)cb * DIAG_CELL_NV;
  *nlaunch = 0;
  cudaError_t e;
  for (int c0 = 0; c0 < d.n[ax]; c0 += m) {
    const Slab L = make_slab(d, ax, m, c0);
    const unsigned blocks = (L.end - L.base + 255) / 256;
    if (ucfl_cached) exact_flux_kernel<true><<<blocks, 256, 0, st>>>(A, F, G, L);
    else exact_flux_kernel<false><<<blocks, 256, 0, st>>>(A, F, G, L);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    budget_cells_kernel<<<cb, 256, 0, st>>>(A, Ecur, F, G, L, te, tm, pc);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    budget_tail_kernel<<<2 * groups + 12 * pb, 128, 0, st>>>(A, F, G, L, te, tm, groups, pb, vol3, pp);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    *nlaunch += 3;
  }
  *nlaunch += 1;
  return launch_diag_finish(pc, cb, pp, pb, result, st);
}

}  // namespace rt
