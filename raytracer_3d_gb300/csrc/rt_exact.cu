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
// The bound is the binary64 pipe: 10 instructions per face flux, two per
// axis in the divergence and eight in the update, 80 per cell with six axes
// in the two passes (290 with the divisions on that pipe).  32x32x32x12^3
// measured 9.46 ms per step, 5.98 G cells/s and 478 G binary64
// instructions/s, 90% of the measured rate; the TMA plane kernel took 39.9
// ms, and a CTA of 512 threads per x-y plane 280 us for a 40x120 column
// (one launch here: 8.2 us), 6.3 ms for a 10x20x60x60 section (97 us) and
// 8.7 ms for 8x8x16x16^3 (0.74 ms).
#include <algorithm>

#include "../../include/rt_gb300.h"
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
  double q[AX];   // the axes' quotients do not depend on one another
#pragma unroll
  for (int f = 0; f < AX; f++) {
    if (f >= S.axes) break;
    const double fl = J.left[f] >= 0 ? sF[J.left[f]] : dmul(J.v0[f], e0);
    q[f] = div_rn(dsub(sF[J.right[f]], fl), J.dd[f]);
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

namespace {

// cells per CTA: one CTA per SM, so that the binary64 work spreads evenly
SmallGeom make_small(const Dims& d, int ctas) {
  SmallGeom S;
  S.G = make_cells(d);
  S.C = (int)((d.ncell + ctas - 1) / ctas);
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
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  if (nsteps == 1) {
    kernel<<<ctas, threads, sm, st>>>(A, S, W, 1, nullptr);
    return cudaGetLastError();
  }
  e = cudaMemsetAsync(counter, 0, sizeof(unsigned), st);
  if (e != cudaSuccess) return e;
  StepArgs<double> a = A;
  SmallGeom s = S;
  void* args[] = {&a, &s, &W, &nsteps, &counter};
  return cudaLaunchCooperativeKernel((const void*)kernel, dim3(ctas), dim3((unsigned)threads), args, sm, st);
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
