// rt_march.cu -- launchers of the binary32 step that marches along k
// (rt_march.cuh): one field, or the members of a batch in one launch.
#include <algorithm>

#include "rt_kernels.h"
#include "rt_march.cuh"

namespace rt {

namespace {

template <int V>
__global__ void __launch_bounds__(RT_MARCH_THREADS, 1) march_kernel(const __grid_constant__ MarchArgs A) {
  march_cta<V>(A, blockIdx.x);
}

// V = 0: members of several widths
template <int V>
__global__ void __launch_bounds__(RT_MARCH_THREADS, 1) march_batch_kernel(const __grid_constant__ MarchBatch B) {
  int lo = 0, hi = B.nmem;   // first[lo] <= blockIdx.x < first[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (blockIdx.x >= B.first[mid]) lo = mid;
    else hi = mid;
  }
  const MarchArgs& A = B.mem[lo];
  const unsigned item = blockIdx.x - B.first[lo];
  if constexpr (V > 0) {
    march_cta<V>(A, item);
  } else {
    if (A.V == 4) march_cta<4>(A, item);
    else if (A.V == 2) march_cta<2>(A, item);
    else march_cta<1>(A, item);
  }
}

int march_width(const Dims& d) { return d.n[0] % 4 == 0 ? 4 : (d.n[0] % 2 == 0 ? 2 : 1); }

// want: CTAs the field should have at least, if k has that many segments.  A
// segment's start costs three loads and one flux, so walks are as long as
// the number of CTAs allows.
MarchArgs make_march(const StepArgs<float>& S, int band, int sweep, long long want) {
  const Dims& d = S.d;
  MarchArgs A;
  A.E = S.E;
  A.Enew = S.Enew;
  int len = 0;
  for (int a = 0; a < 6; a++) {
    A.vel[a] = S.vel[a];
    A.vlo[a] = S.vlo[a];
    A.n[a] = d.n[a];
    A.pre[a] = len;
    len += d.n[a] + 2 * RT_ONX;
  }
  A.len = len;
  A.lam = S.lam[0];
  A.tab = S.t32.inv_d[0];
  A.seed_in = S.seed_in;
  A.seed_out = S.seed_out;
  A.dthi = S.dthi;
  A.dtlo = S.dtlo;
  A.upper_refl = d.upper_refl;
  A.lower_refl = d.lower_refl;
  A.V = march_width(d);
  A.nvol3 = (unsigned)d.nvol3;
  A.nvec = (unsigned)(d.nvol3 / A.V);
  A.hx = make_div((unsigned)(d.n[0] / A.V));
  A.ny = make_div((unsigned)d.n[1]);
  const long long blocks = (A.nvec + RT_MARCH_THREADS - 1) / RT_MARCH_THREADS;
  const long long lm = (long long)d.n[4] * d.n[5];
  long long segs = (want + lm * blocks - 1) / (lm * blocks);
  segs = std::max(1ll, std::min<long long>(segs, d.n[3]));
  A.klen = (int)((d.n[3] + segs - 1) / segs);
  segs = (d.n[3] + A.klen - 1) / A.klen;
  A.segs = make_div((unsigned)segs);
  A.per_vol = make_div((unsigned)(blocks * segs));
  A.sweep = sweep ? 1 : 0;
  const int nb = sweep ? d.n[4] : d.n[5], no = sweep ? d.n[5] : d.n[4];
  const int B = std::max(1, std::min(band, nb));
  A.band = make_div((unsigned)B);
  A.band_full = make_div((unsigned)(B * no));
  A.items = (unsigned)(lm * blocks * segs);
  return A;
}

template <class K>
cudaError_t allow_smem(K kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}
template <class K, class P>
cudaError_t go(K kernel, int V, unsigned ctas, const P& args, cudaStream_t st) {
  const size_t sm = march_smem(V);
  const cudaError_t e = allow_smem(kernel, sm);
  if (e != cudaSuccess) return e;
  kernel<<<ctas, RT_MARCH_THREADS, sm, st>>>(args);
  return cudaGetLastError();
}

// CTAs a field should have: two rounds of what the GPU holds.  More segments
// cost more starts than their even end saves: four rounds measured 76.6 us
// per step at 16^3x12^3 against 73.8, 30.8 against 26.9 at 16^3x8^3, 20.5
// against 16.4 at 8^3x12^3; one round 28.8 and 16.4 us.  From 20 M cells on
// walks are whole either way.
constexpr long long kBusy = 152 * 3 * 2;

}  // namespace

bool march_ok(const Dims& d) { return d.ncell <= (1ll << 30); }

cudaError_t launch_march(const StepArgs<float>& S, const StepTuning& tn, cudaStream_t st) {
  const MarchArgs A = make_march(S, tn.band, tn.sweep, kBusy);
  if (A.V == 4) return go(march_kernel<4>, 4, A.items, A, st);
  if (A.V == 2) return go(march_kernel<2>, 2, A.items, A, st);
  return go(march_kernel<1>, 1, A.items, A, st);
}

// of n fields, those that one launch takes: what its arguments hold, and no
// more CTAs than a grid may have (2^31 - 1; fields of one spatial point have a
// CTA per (l,m), so two of 2^30 cells are beyond it)
int march_batch_take(const StepArgs<float>* S, int n) {
  long long ctas = 0;
  int m = 0;
  for (; m < std::min(n, RT_MARCH_MEMBERS); m++) {
    const Dims& d = S[m].d;
    const long long nvec = d.nvol3 / march_width(d);
    // an upper bound of MarchArgs::items
    ctas += (long long)d.n[4] * d.n[5] * ((nvec + RT_MARCH_THREADS - 1) / RT_MARCH_THREADS) + kBusy;
    if (m > 0 && ctas > 0x7fffffffll) break;
  }
  return m;
}

int march_batch_launches(const StepArgs<float>* S, int n) {
  int k = 0;
  for (int j = 0; j < n; j += march_batch_take(S + j, n - j)) k++;
  return k;
}

cudaError_t launch_march_batch(const StepArgs<float>* S, int n, int band, int sweep, cudaStream_t st) {
  long long cells = 0;
  for (int j = 0; j < n; j++) cells += S[j].d.ncell;
  for (int j0 = 0, take; j0 < n; j0 += take) {
    MarchBatch B;
    B.nmem = take = march_batch_take(S + j0, n - j0);
    unsigned total = 0;
    int V = 0;
    for (int j = 0; j < B.nmem; j++) {
      const StepArgs<float>& s = S[j0 + j];
      B.mem[j] = make_march(s, band, sweep, kBusy * s.d.ncell / cells);
      B.first[j] = total;
      total += B.mem[j].items;
      V = j == 0 ? B.mem[j].V : (V == B.mem[j].V ? V : 0);
    }
    B.first[B.nmem] = total;
    cudaError_t e;
    if (V == 4) e = go(march_batch_kernel<4>, 4, total, B, st);
    else if (V == 2) e = go(march_batch_kernel<2>, 2, total, B, st);
    else if (V == 1) e = go(march_batch_kernel<1>, 1, total, B, st);
    else e = go(march_batch_kernel<0>, 4, total, B, st);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace rt
