// rt_coeff.cu -- coefficients of a field (calc_parameter.f90:13-261): the
// twelve face velocities of every cell, the growth rates and the CFL rate.
//
// Every velocity is a difference of averages of the dispersion relation at
// up to four points, so a direct evaluation takes some 25 dispersion
// relations (a division and a square root each, about 900 binary64
// instructions) per cell; the binary64 pipe bounds it.  Here
//   omega_kernel   evaluates the relation once per grid point into a scratch
//                  ring of m planes (omega_e), with 1/omega_i of the interior
//                  beside it;
//   coeff_kernel   forms, walking along k, the pair sums of each axis pair,
//                  both faces' velocities of all six axes from them (the left
//                  faces of the first cells are the face-0 planes, all of
//                  them enter the CFL rate), and the growth rates, and stores
//                  them in the form's precision.
// Divisions, square roots, comparisons, changes of sign and the conversion to
// binary32 run on the integer pipes (rt_exact.cuh).  About 62 binary64
// instructions and 26 integer quotients per cell, both pipes near 70% busy; registers, not warps:
// 2 to 4 CTAs per SM measure the same.  The values are those of the
// reference's sequence bit for bit (rt_coeff.cuh states it).  24^3x12x12x16
// (31.9 M cells) in binary32: 6.2 ms for all of it (omega_kernel 1.0, 1.75
// with the square root on the binary64 pipe; 8.8 with a thread per cell and
// those operations there), against 60 ms for the direct evaluation and its
// separate face-0, rate and conversion passes.
#include <algorithm>

#include "rt_coeff.cuh"
#include "rt_exact.cuh"
#include "rt_kernels.h"

namespace rt {

namespace {

// points of the scratch: spatial indices 0..n, spectral indices 0..n+1
// (Fortran); of an x/k or y/l pair whose velocities are analytic 1..n of both
struct OmegaGeom {
  int sx, sy, sz;        // spatial points per axis
  int wk, wl;            // spectral points along k and l
  int lo[2];             // first index of the x/k and y/l pairs
  unsigned s3;           // sx*sy*sz
  long long plane;       // doubles of one m plane: s3*wk*wl
  int ring;              // planes of the ring; plane m at m % ring
};

__device__ __forceinline__ double sign_times(double sgn, double x) {
  return sgn == 1.0 ? x : (sgn == -1.0 ? -x : dmul(sgn, x));
}

// m planes [m0, m0 + gridDim.z): block (b, u, j) takes the spectral points u,
// u + gridDim.y, ... of plane m0 + j and walks the spatial points
__global__ void __launch_bounds__(256) omega_kernel(Dims d, Background bg, Grid g, Phys ph, OmegaGeom G, int m0,
                                                    double* __restrict__ om, double* __restrict__ inv) {
  const int m = m0 + (int)blockIdx.z;
  const double mtv = g.mt[pidx(m)];
  const double m2 = dmul(mtv, mtv);
  const double f2m2 = dmul(dmul(ph.f0, ph.f0), m2);
  for (unsigned u = blockIdx.y; u < (unsigned)(G.wk * G.wl); u += gridDim.y) {
    const int l = G.lo[0] + (int)(u % (unsigned)G.wk), n = G.lo[1] + (int)(u / (unsigned)G.wk);
    const double ktv = g.kt[pidx(l)], ltv = g.lt[pidx(n)];
    const double kh2 = dadd(dmul(ltv, ltv), dmul(ktv, ktv));
    const double den = dadd(m2, kh2);
    double* out = om + (long long)(m % G.ring) * G.plane + (long long)u * G.s3;
    const bool inside = l >= 1 && l <= d.n[3] && n >= 1 && n <= d.n[4] && m >= 1 && m <= d.n[5];
    double* outi = inv + (long long)(m % G.ring) * d.s[5] + (long long)((l - 1) + d.n[3] * (n - 1)) * d.nvol3;
    for (unsigned v = blockIdx.x * blockDim.x + threadIdx.x; v < G.s3; v += gridDim.x * blockDim.x) {
      const int i = G.lo[0] + (int)(v % (unsigned)G.sx);
      const unsigned r = v / (unsigned)G.sx;
      const int j = G.lo[1] + (int)(r % (unsigned)G.sy), k = (int)(r / (unsigned)G.sy);
      const long long q = bg_idx(bg, i, j, k);
      const double oi = sign_times(ph.sgn, sqrt_rn(div_rn(dadd(dmul(bg.Nsqr[q], kh2), f2m2), den)));
      out[v] = dadd(dadd(oi, dmul(ktv, bg.U[q])), dmul(ltv, bg.V[q]));
      if (inside && i > 0 && j > 0 && k > 0)
        outi[(i - 1) + d.n[0] * ((j - 1) + (long long)d.n[1] * (k - 1))] = div_rn(1.0, oi);
    }
  }
}

// 0.5*A/d - 0.5*B/d of the reference's averages, from the pair sums: the
// halves are exact, so (0.5*A - 0.5*B)/d = 0.5*((A - B)/d) unless a result
// is near the denormals (then in the reference's order)
__device__ __forceinline__ double half_slope(double A, double B, double dd) {
  const double D = dsub(A, B);
  const Bits64 db = split64(D);
  const double q = div_rn(D, dd);
  const Bits64 qb = split64(q);
  if (is_zero(db)) return q;
  if ((unsigned)(expo(db) - 100) < 1900u && (unsigned)(expo(qb) - 100) < 1900u)
    return __hiloint2double((int)(qb.hi - 0x00100000u), (int)qb.lo);
  return __ddiv_rn(dsub(dmul(0.5, A), dmul(0.5, B)), dd);
}

// -x: written as such it becomes a binary64 instruction
__device__ __forceinline__ double minus(double x) {
  double r;
  asm("{\n\t.reg .b64 t;\n\tmov.b64 t, %1;\n\txor.b64 t, t, 0x8000000000000000;\n\tmov.b64 %0, t;\n\t}" : "=d"(r) : "d"(x));
  return r;
}

// outflow-only ends (calc_parameter.f90:55-66 etc.): max(0, v) and
// -max(0, -v), compared as bit patterns (a NaN stays)
__device__ __forceinline__ double clamp_face(double v, int f, int n, bool hi, bool lo) {
  const uint64_t u = (uint64_t)__double_as_longlong(v);
  const bool neg = u > 0x8000000000000000ull && u <= 0xfff0000000000000ull, pos = u - 1 < 0x7ff0000000000000ull;
  if (f == n && hi && neg) v = 0.0;
  if (f == 0 && lo && pos) v = __longlong_as_double((long long)0x8000000000000000ull);
  return v;
}

// fmax2 of two magnitudes (a > b ? a : b, NaN included)
__device__ __forceinline__ double max_abs(double x, double y) {
  const uint64_t a = (uint64_t)__double_as_longlong(x) & 0x7fffffffffffffffull;
  const uint64_t b = (uint64_t)__double_as_longlong(y) & 0x7fffffffffffffffull;
  return __longlong_as_double((long long)(a > b && a <= 0x7ff0000000000000ull ? a : b));
}

template <class T>
__device__ __forceinline__ T as(double x);
template <>
__device__ __forceinline__ double as<double>(double x) { return x; }
template <>
__device__ __forceinline__ float as<float>(double x) { return float_rn(x); }

// cells of the m planes [m0, m0 + gridDim.z) (Fortran m from 1): a thread
// takes a spatial cell at one (l,m) and walks klen values of k.  From one k to
// the next it keeps what they share: omega at k + 1, the pair sums over the k
// face between them and that face's spectral velocity; and what does not
// depend on k (the shears of the growth rate, the indices) is formed once.
template <class T>
__global__ void __launch_bounds__(256, 2) coeff_kernel(Dims d, Background bg, Grid g, Phys ph, OmegaGeom G, int m0,
                                                       int segs, int klen, const double* __restrict__ om,
                                                       const double* __restrict__ inv, CoeffOut<T> out,
                                                       unsigned long long* rate) {
  unsigned long long best = 0;
  const bool xk = d.n[0] > 1 && d.n[3] > 1;
  int c[6];
  c[5] = m0 + (int)blockIdx.z;
  const double* plane = om + (long long)(c[5] % G.ring) * G.plane;
  const double* below = om + (long long)((c[5] - 1) % G.ring) * G.plane;
  const double* above = om + (long long)((c[5] + 1) % G.ring) * G.plane;
  for (unsigned u = blockIdx.y; u < (unsigned)(d.n[4] * segs); u += gridDim.y) {
    c[4] = (int)(u / (unsigned)segs) + 1;
    const int k0 = (int)(u % (unsigned)segs) * klen + 1, k1 = min(k0 + klen - 1, d.n[3]);
    const double ltv = g.lt[pidx(c[4])];
    for (unsigned v3 = blockIdx.x * blockDim.x + threadIdx.x; v3 < (unsigned)d.nvol3; v3 += gridDim.x * blockDim.x) {
      c[0] = (int)(v3 % (unsigned)d.n[0]) + 1;
      const unsigned r3 = v3 / (unsigned)d.n[0];
      c[1] = (int)(r3 % (unsigned)d.n[1]) + 1;
      c[2] = (int)(r3 / (unsigned)d.n[1]) + 1;
      const int w = c[0] - G.lo[0] + G.sx * (c[1] - G.lo[1] + G.sy * c[2]);
      const int back[3] = {1, G.sx, G.sx * G.sy};
      const long long q = bg_idx(bg, c[0], c[1], c[2]);
      const long long st[3] = {1, bg.px, (long long)bg.px * bg.py};
      double dU[3], dV[3];
  #pragma unroll
      for (int s = 0; s < 3; s++) {
        dU[s] = dsub(bg.U[q + st[s]], bg.U[q - st[s]]);
        dV[s] = dsub(bg.V[q + st[s]], bg.V[q - st[s]]);
      }
      long long o = (long long)(k0 - G.lo[0] + G.wk * (c[4] - G.lo[1])) * G.s3;   // (k, l) of the walk in an omega plane
      double e0 = plane[o + w], ebx = 0.0, A01x = 0.0, A11x = 0.0, hk = 0.0;
      if (xk) {
        ebx = plane[o + w - 1];
        A01x = dadd(plane[o - G.s3 + w], e0);
        A11x = dadd(plane[o - G.s3 + w - 1], ebx);
        hk = half_slope(A01x, A11x, g.d[0][pidx(c[0])]);
      }
      for (c[3] = k0; c[3] <= k1; c[3]++, o += G.s3) {
        const double ktv = g.kt[pidx(c[3])];
        const long long p = v3 + d.nvol3 * ((long long)(c[3] - 1) + d.n[3] * ((c[4] - 1) + (long long)d.n[4] * (c[5] - 1)));
        double vr[6], vl[6], e1 = 0.0;
        if (xk) {
          e1 = plane[o + G.s3 + w];
          const double eb1 = plane[o + G.s3 + w - 1];
          // pair sums of aloc (twice the average over the wavenumber neighbours)
          const double A00 = dadd(e0, e1), A10 = dadd(ebx, eb1);   // at (cell, k), (the cell below, k)
          const double dw = g.d[3][pidx(c[3])], hr = half_slope(A00, A10, g.d[0][pidx(c[0])]);
          vr[0] = clamp_face(half_slope(A00, A01x, dw), c[0], d.n[0], true, true);
          vl[0] = clamp_face(half_slope(A10, A11x, dw), c[0] - 1, d.n[0], true, true);
          vr[3] = clamp_face(minus(hr), c[3], d.n[3], true, true);
          vl[3] = clamp_face(minus(hk), c[3] - 1, d.n[3], true, true);
          A01x = A00;
          A11x = A10;
          ebx = eb1;
          hk = hr;
        }
  #pragma unroll
        for (int s = 0; s < 3; s++) {
          const int a = s, b = s + 3;
          if (s < 2 && !(d.n[a] > 1 && d.n[b] > 1)) {
            // collapsed x/k or y/l pair: analytic spatial velocity on interior cells
            const int cl[6] = {c[0] - (s == 0), c[1] - (s == 1), c[2], c[3], c[4], c[5]};
            vr[a] = analytic_vel(bg, g, ph, c, s);
            vl[a] = cl[a] >= 1 ? analytic_vel(bg, g, ph, cl, s) : 0.0;
            vr[b] = vl[b] = 0.0;
            continue;
          }
          if (s == 0) continue;
          const double* lo = s == 1 ? plane + o - (long long)G.wk * G.s3 : below + o;
          const double* hi = s == 1 ? plane + o + (long long)G.wk * G.s3 : above + o;
          const int wb = w - back[s];
          const double eb = plane[o + wb];
          const double A00 = dadd(e0, hi[w]), A01 = dadd(lo[w], e0);     // at (cell, w), (cell, w - 1)
          const double A10 = dadd(eb, hi[wb]), A11 = dadd(lo[wb], eb);   // at the spatial neighbour below
          const double ds = g.d[a][pidx(c[a])], dw = g.d[b][pidx(c[b])];
          const bool up = s < 2 || !d.upper_refl, dn = s < 2 || !d.lower_refl;
          vr[a] = clamp_face(half_slope(A00, A01, dw), c[a], d.n[a], up, dn);
          vl[a] = clamp_face(half_slope(A10, A11, dw), c[a] - 1, d.n[a], up, dn);
          vr[b] = clamp_face(minus(half_slope(A00, A10, ds)), c[b], d.n[b], true, true);
          vl[b] = clamp_face(minus(half_slope(A01, A11, ds)), c[b] - 1, d.n[b], true, true);
        }
        e0 = xk ? e1 : (c[3] < k1 ? plane[o + G.s3 + w] : 0.0);
        double r = 0.0;
        bool first = true;   // (0 + x = x: no binary64 instruction for the first)
  #pragma unroll
        for (int a = 0; a < 6; a++) {
          out.vel[a][p] = as<T>(vr[a]);
          if (c[a] == 1) {
            long long f = 0;
  #pragma unroll
            for (int b = 0; b < 6; b++) f += (long long)(c[b] - 1) * d.ps[a][b];
            out.vlo[a][f] = as<T>(vl[a]);
          }
          if (d.n[a] > 1) {
            const double t = div_rn(max_abs(vl[a], vr[a]), g.d[a][pidx(c[a])]);
            r = first ? t : dadd(r, t);
            first = false;
          }
        }
        const unsigned long long rb = (unsigned long long)__double_as_longlong(r) & 0x7fffffffffffffffull;
        best = rb > best ? rb : best;
        // growth rates, calc_parameter.f90:246-254
        const double iv = inv[(long long)(c[5] % G.ring) * d.s[5] + (p - (long long)(c[5] - 1) * d.s[5])];
        const double xu = dsub(vr[0], bg.U[q]), yv = dsub(vr[1], bg.V[q]);
        double lam[3];
  #pragma unroll
        for (int s = 0; s < 3; s++) {
          const double d2 = dmul(2.0, g.d[s][pidx(c[s])]);
          const double f1 = s < 2 ? xu : ktv, f2 = s < 2 ? yv : ltv;
          const double head = dmul(iv, s == 0 ? ktv : (s == 1 ? ltv : vr[2]));
          lam[s] = dmul(head, dadd(div_rn(dmul(f1, dU[s]), d2), div_rn(dmul(f2, dV[s]), d2)));
        }
        if constexpr (sizeof(T) == 8) {
  #pragma unroll
          for (int s = 0; s < 3; s++) out.lam[s][p] = lam[s];
        } else {   // one combined rate, summed in binary64 before rounding
          double sum = 0.0;
  #pragma unroll
          for (int s = 0; s < 3; s++)
            if (d.n[s] > 1) sum += lam[s];
          out.lam[0][p] = as<T>(sum);
        }
      }
    }
  }
  // the largest CFL rate: rates are >= 0, so their bit patterns order as
  // unsigned integers (NaN above all of them)
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) {
    const unsigned long long o = __shfl_xor_sync(0xffffffffu, best, w);
    best = o > best ? o : best;
  }
  if ((threadIdx.x & 31) == 0) atomicMax(rate, best);
}

OmegaGeom make_omega(const Dims& d, int ring) {
  OmegaGeom G;
  const int xk = d.n[0] > 1 && d.n[3] > 1, yl = d.n[1] > 1 && d.n[4] > 1;
  G.lo[0] = 1 - xk;
  G.lo[1] = 1 - yl;
  G.sx = d.n[0] + xk;
  G.sy = d.n[1] + yl;
  G.sz = d.n[2] + 1;
  G.wk = d.n[3] + 2 * xk;
  G.wl = d.n[4] + 2 * yl;
  G.s3 = (unsigned)G.sx * G.sy * G.sz;
  G.plane = (long long)G.s3 * G.wk * G.wl;
  G.ring = ring;
  return G;
}

constexpr long long kBusy = 152 * 2 * 6;   // blocks

unsigned walk_blocks(long long points) { return (unsigned)std::min<long long>((points + 255) / 256, 16); }

}  // namespace

// m planes of the scratch ring: three at least, more while it stays within
// `bytes` (two neighbours stay from one batch of planes to the next)
int coeff_ring(const Dims& d, long long bytes) {
  const long long per = (make_omega(d, 1).plane + d.s[5]) * (long long)sizeof(double);
  return (int)std::max<long long>(3, std::min<long long>(std::min(d.n[5] + 2, 60000), bytes / per));
}
long long coeff_scratch(const Dims& d, int ring) { return ring * (make_omega(d, ring).plane + d.s[5]); }

template <class T>
cudaError_t launch_coeff(const Dims& d, const Background& bg, const Grid& g, const Phys& ph, const CoeffOut<T>& out,
                         double* scratch, int ring, double* rate, int* nlaunch, cudaStream_t st) {
  const OmegaGeom G = make_omega(d, ring);
  double* om = scratch;
  double* inv = scratch + ring * G.plane;
  cudaError_t e = cudaMemsetAsync(rate, 0, sizeof(double), st);
  if (e != cudaSuccess) return e;
  *nlaunch = 0;
  const int batch = ring - 2;
  const unsigned wspec = (unsigned)std::min(G.wk * G.wl, 65535);
  for (int m0 = 1; m0 <= d.n[5]; m0 += batch) {
    const int cnt = std::min(batch, d.n[5] - m0 + 1);
    // planes 0 and 1 come with the first batch; then one beyond the last cell plane
    const int w0 = m0 == 1 ? 0 : m0 + 1, wn = m0 + cnt + 1 - w0;
    omega_kernel<<<dim3(walk_blocks(G.s3), wspec, (unsigned)wn), 256, 0, st>>>(d, bg, g, ph, G, w0, om, inv);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    // walks along k as long as the GPU stays busy for a few rounds
    const long long blocks = (d.nvol3 + 255) / 256 * d.n[4] * cnt;
    const int want = (int)std::max(1ll, std::min<long long>(d.n[3], (kBusy + blocks - 1) / blocks));
    const int klen = (d.n[3] + want - 1) / want, segs = (d.n[3] + klen - 1) / klen;
    const dim3 grid((unsigned)((d.nvol3 + 255) / 256), (unsigned)std::min<long long>((long long)d.n[4] * segs, 65535),
                    (unsigned)cnt);
    coeff_kernel<T><<<grid, 256, 0, st>>>(d, bg, g, ph, G, m0, segs, klen, om, inv, out,
                                          reinterpret_cast<unsigned long long*>(rate));
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    *nlaunch += 2;
  }
  return cudaSuccess;
}
template cudaError_t launch_coeff<double>(const Dims&, const Background&, const Grid&, const Phys&,
                                          const CoeffOut<double>&, double*, int, double*, int*, cudaStream_t);
template cudaError_t launch_coeff<float>(const Dims&, const Background&, const Grid&, const Phys&,
                                         const CoeffOut<float>&, double*, int, double*, int*, cudaStream_t);

}  // namespace rt
