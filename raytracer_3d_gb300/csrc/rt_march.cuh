// rt_march.cuh -- binary32 step: threads of V x-cells marching along k.
//
// A thread owns V consecutive cells of an x row (V = 4, 2 or 1, whichever
// divides nx) at one (y,z) and walks k at one (l,m).  What the walk shares
// stays in registers: the four k values of E, the difference of the k face
// ahead and the flux through the k face just passed, so a k face is evaluated
// once; the faces of a row once too, but for the one a row's parts meet at.
// The y, z, l and m faces are evaluated from both sides, on four differences
// instead of six.  Everything else a cell needs is copied ahead: while the
// thread works on one k, cp.async brings its operands of the next k into
// slots of shared memory that it alone uses, so no barrier is needed and any
// extents do: a field of odd or small planes runs like a large one.
//
// A part of the loop waits for its own copies only (one group of copies per
// part, the six younger ones still under way), so each has a whole step of
// the walk to arrive; one group for all, waited for right after its last
// copy was issued, cost 12% (94 against 107 G cells/s).  Registers matter more
// than resident warps: compiled without a lower bound on the CTAs per SM
// (154, 116 and 96 registers; 12 to 20 warps) the widths V = 4, 2, 1 run at
// 111.7, 83.5 and 47.9 G cells/s, with bounds of 3, 6 and 5 at 107.2, 64.9
// and 44.1.  (V = 4 on rows that 4 does not divide, in copies of 8 or 4 bytes:
// 50 and 29, L1 wavefronts.)
//
// What bounds it: 32x32x32x12x16x12 has the issue slots 66% and the ALU pipe
// (selects, minima, sign logic) 62% busy, DRAM 67% at 50 bytes per cell (36
// algorithmic).  Loads straight into registers left issue at 35% (61 G
// cells/s).  Steps measured: 32^6 9.85 ms, 109 G cells/s (z march 15.9 ms);
// 32x32x32x12x16x12 0.68 ms (1.27); 24x24x24x12x12x16 0.29 (0.87, TMA planes
// 3.0); 30x18x20x14x10x12 0.22 (0.55, TMA planes 1.69).
// The boundary maps are offsets fixed for the walk (a ghost that copies the
// edge cell makes the difference zero and the flux v*E exactly), the face-0
// velocities another base pointer.  Arithmetic per face and cell is that of
// flux_fp32, div32 and upd32 in the axis order x,y,z,k,l,m: the same bits as
// the other binary32 kernels.
#pragma once
#include "rt_fast.cuh"
#include "rt_step2.cuh"

namespace rt {

// What a walk needs to know of its field, small enough that the members of a
// batch travel as kernel arguments (constant memory).  Fields up to 2^30
// cells: byte offsets into E fit 32 bits.
struct MarchArgs {
  const float* E;
  float* Enew;
  const float* vel[6];
  const float* vlo[6];
  const float* lam;
  const float* tab;         // the tables of Tab32, group g of axis a at g*len + pre[a]
  const unsigned* seed_in;
  unsigned* seed_out;
  float dthi, dtlo;
  int n[6];
  int pre[6], len;          // starts of the axes in a group of tables, and a group's length
  int upper_refl, lower_refl;
  int V;                    // cells per thread along x
  unsigned nvec;            // vectors per (x,y,z) volume: nvol3 / V
  unsigned nvol3;
  DivU32 hx, ny;            // vector of the volume -> x part, y, z
  DivU32 per_vol;           // CTAs of one (l,m): CTAs per volume * segs -> (l,m) index
  DivU32 segs;              // k segments
  int klen;                 // k values per segment
  DivU32 band_full, band;   // band order of (l,m): outer*band, band
  int sweep;
  unsigned items;           // CTAs of the field
};

#define RT_MARCH_THREADS 128
// members per launch: the argument block of a kernel holds 32,764 bytes
#define RT_MARCH_MEMBERS 80
struct MarchBatch {
  int nmem;
  unsigned first[RT_MARCH_MEMBERS + 1];   // CTAs [first[j], first[j+1]) belong to member j
  MarchArgs mem[RT_MARCH_MEMBERS];
};
static_assert(sizeof(MarchBatch) <= 32764, "the members of a batch must fit a kernel's arguments");

template <int V>
struct Vec {
  float a[V];
};

template <int V>
__device__ __forceinline__ Vec<V> ldv(const float* base, unsigned byte) {
  const char* q = reinterpret_cast<const char*>(base) + byte;
  Vec<V> r;
  if constexpr (V == 4) {
    const float4 t = __ldg(reinterpret_cast<const float4*>(q));
    r.a[0] = t.x; r.a[1] = t.y; r.a[2] = t.z; r.a[3] = t.w;
  } else if constexpr (V == 2) {
    const float2 t = __ldg(reinterpret_cast<const float2*>(q));
    r.a[0] = t.x; r.a[1] = t.y;
  } else {
    r.a[0] = __ldg(reinterpret_cast<const float*>(q));
  }
  return r;
}
__device__ __forceinline__ float ld1(const float* base, unsigned byte) {
  return __ldg(reinterpret_cast<const float*>(reinterpret_cast<const char*>(base) + byte));
}

// max(0, min(2*min(a, t), max(a, t))) for a = |Rj| and t = sign(Rj)*up, given
// 2*Rj and 2*t: the doubling commutes with min, and the three-input minimum
// is one instruction (the ALU pipe bounds this kernel)
__device__ __forceinline__ float superbee32(float Rj, float t, float Rj2, float t2) {
  float q;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(q) : "f"(fabsf(Rj2)), "f"(t2), "f"(fmaxf(fabsf(Rj), t)));
  return fmaxf(0.f, q);
}

// the limited flux from its differences: Rj over the face, up1 / up2 over the
// faces behind and ahead, Eb / Ec on the two sides (flux_fp32's operations)
__device__ __forceinline__ float flux_d(float v, float nhcfl, float Rjm, float Rj, float Rjp, float Eb, float Ec) {
  const bool pos = v > 0.f;
  const float up = pos ? Rjm : Rjp;
  const float Eu = pos ? Eb : Ec;
  const unsigned s = __float_as_uint(Rj) & 0x80000000u;
  const float t = __uint_as_float(__float_as_uint(up) ^ s);
  const float ph = superbee32(Rj, t, 2.f * Rj, 2.f * t);
  const float psi = __uint_as_float(__float_as_uint(ph) ^ s);
  const float av = fabsf(v);
  const float h = av * fmaf(nhcfl, av, 0.5f);
  return fmaf(h, psi, v * Eu);
}
// two cells at once: the products and sums on the packed f32x2 instructions
__device__ __forceinline__ float2 flux_d2(float2 v, float2 nhcfl, float2 Rjm, float2 Rj, float2 Rjp, float2 Eb,
                                          float2 Ec) {
  const bool px = v.x > 0.f, py = v.y > 0.f;
  const float2 up = make_float2(px ? Rjm.x : Rjp.x, py ? Rjm.y : Rjp.y);
  const float2 Eu = make_float2(px ? Eb.x : Ec.x, py ? Eb.y : Ec.y);
  const unsigned sx = __float_as_uint(Rj.x) & 0x80000000u, sy = __float_as_uint(Rj.y) & 0x80000000u;
  const float2 t = make_float2(__uint_as_float(__float_as_uint(up.x) ^ sx), __uint_as_float(__float_as_uint(up.y) ^ sy));
  const float2 Rj2 = pk_add(Rj, Rj), t2 = pk_add(t, t);
  const float phx = superbee32(Rj.x, t.x, Rj2.x, t2.x), phy = superbee32(Rj.y, t.y, Rj2.y, t2.y);
  const float2 psi = make_float2(__uint_as_float(__float_as_uint(phx) ^ sx), __uint_as_float(__float_as_uint(phy) ^ sy));
  const float2 av = pk_abs(v);
  const float2 h = pk_mul(av, pk_fma(nhcfl, av, make_float2(0.5f, 0.5f)));
  return pk_fma(h, psi, pk_mul(v, Eu));
}

template <int V>
__device__ __forceinline__ Vec<V> vsub(const Vec<V>& a, const Vec<V>& b) {
  Vec<V> r;
  if constexpr (V == 1) {
    r.a[0] = a.a[0] - b.a[0];
  } else {
#pragma unroll
    for (int j = 0; j < V; j += 2) {
      const float2 t = pk_sub(make_float2(a.a[j], a.a[j + 1]), make_float2(b.a[j], b.a[j + 1]));
      r.a[j] = t.x;
      r.a[j + 1] = t.y;
    }
  }
  return r;
}
template <int V>
__device__ __forceinline__ Vec<V> vflux(const Vec<V>& v, float nhcfl, const Vec<V>& Rjm, const Vec<V>& Rj,
                                        const Vec<V>& Rjp, const Vec<V>& Eb, const Vec<V>& Ec) {
  Vec<V> r;
  if constexpr (V == 1) {
    r.a[0] = flux_d(v.a[0], nhcfl, Rjm.a[0], Rj.a[0], Rjp.a[0], Eb.a[0], Ec.a[0]);
  } else {
#pragma unroll
    for (int j = 0; j < V; j += 2) {
      const float2 t = flux_d2(make_float2(v.a[j], v.a[j + 1]), make_float2(nhcfl, nhcfl),
                               make_float2(Rjm.a[j], Rjm.a[j + 1]), make_float2(Rj.a[j], Rj.a[j + 1]),
                               make_float2(Rjp.a[j], Rjp.a[j + 1]), make_float2(Eb.a[j], Eb.a[j + 1]),
                               make_float2(Ec.a[j], Ec.a[j + 1]));
      r.a[j] = t.x;
      r.a[j + 1] = t.y;
    }
  }
  return r;
}
// acc += (fl - fr) * (chi + clo), div32 per cell
template <int V>
__device__ __forceinline__ void vdiv(Vec<V>& acc, const Vec<V>& fr, const Vec<V>& fl, float chi, float clo) {
  if constexpr (V == 1) {
    acc.a[0] = div32(acc.a[0], fr.a[0], fl.a[0], chi, clo);
  } else {
#pragma unroll
    for (int j = 0; j < V; j += 2) {
      const float2 t = div2<true>(make_float2(acc.a[j], acc.a[j + 1]), make_float2(fr.a[j], fr.a[j + 1]),
                                  make_float2(fl.a[j], fl.a[j + 1]), make_float2(chi, chi), make_float2(clo, clo));
      acc.a[j] = t.x;
      acc.a[j + 1] = t.y;
    }
  }
}

// group g of the tables (1: dt/(2d), 2 and 3: dt/d as hi + lo) at Fortran index f
__device__ __forceinline__ float tab_at(const MarchArgs& A, int g, int a, int f) {
  return A.tab[g * A.len + A.pre[a] + pidx(f)];
}
// constants of a cell along one axis: -dt/(2d) of the right and left face,
// dt/d as hi + lo
struct AxisK {
  float r, l, hi, lo;
  __device__ __forceinline__ void load(const MarchArgs& A, int a, int c) {
    r = -tab_at(A, 1, a, c + 1);
    l = -tab_at(A, 1, a, c);
    hi = tab_at(A, 2, a, c + 1);
    lo = tab_at(A, 3, a, c + 1);
  }
};

// an axis of which both faces are evaluated
template <int V>
__device__ __forceinline__ void both_faces(Vec<V>& acc, const AxisK& k, const Vec<V>& vr, const Vec<V>& vl,
                                           const Vec<V>& Em2, const Vec<V>& Em1, const Vec<V>& E0, const Vec<V>& Ep1,
                                           const Vec<V>& Ep2) {
  const Vec<V> D0 = vsub<V>(Em1, Em2), D1 = vsub<V>(E0, Em1), D2 = vsub<V>(Ep1, E0), D3 = vsub<V>(Ep2, Ep1);
  const Vec<V> fr = vflux<V>(vr, k.r, D1, D2, D3, E0, Ep1);
  const Vec<V> fl = vflux<V>(vl, k.l, D0, D1, D2, Em1, E0);
  vdiv<V>(acc, fr, fl, k.hi, k.lo);
}

// offsets (bytes) of the -2, -1, +1, +2 neighbours along an axis of n cells
// with stride s from coordinate c, by the rules of map_coord; z walls
// mirror and reverse m (flip: the offset of the reversed m)
__device__ __forceinline__ void nb_bytes(int n, int s, int c, bool mirror_lo, bool mirror_hi, int flip,
                                         unsigned o[4]) {
  const int off[4] = {-2, -1, 1, 2};
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int t = c + off[j];
    int c2 = t, q = 0;
    if (t < 0) {
      c2 = mirror_lo ? -t - 1 : 0;
      q = mirror_lo ? flip : 0;
    } else if (t >= n) {
      c2 = mirror_hi ? 2 * n - 1 - t : n - 1;
      q = mirror_hi ? flip : 0;
    }
    o[j] = (unsigned)((c2 - c) * s + q) * 4u;
  }
}

// ---- operands of the next k, copied ahead into the thread's own slots ----
// slot j of thread t lies at (j*threads + t)*V floats
template <int V>
__device__ __forceinline__ void slot_fill(uint32_t slot, const float* base, unsigned byte) {
  const void* g = reinterpret_cast<const char*>(base) + byte;
  if constexpr (V == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(slot), "l"(g));
  else if constexpr (V == 2) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(slot), "l"(g));
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(slot), "l"(g));
}
template <int V>
__device__ __forceinline__ Vec<V> slot_take(uint32_t slot) {
  Vec<V> r;
  if constexpr (V == 4)
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(r.a[0]), "=f"(r.a[1]), "=f"(r.a[2]), "=f"(r.a[3]) : "r"(slot));
  else if constexpr (V == 2)
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(r.a[0]), "=f"(r.a[1]) : "r"(slot));
  else
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(r.a[0]) : "r"(slot));
  return r;
}
#define RT_MARCH_SLOTS 28
__host__ __device__ constexpr size_t march_smem(int V) { return (size_t)RT_MARCH_SLOTS * RT_MARCH_THREADS * V * sizeof(float); }

// CTA `item` of the field
template <int V>
__device__ __forceinline__ void march_cta(const MarchArgs& A, unsigned item) {
  const unsigned lm = A.per_vol.div(item);
  const unsigned rest = item - lm * A.per_vol.d;
  const unsigned b = A.segs.div(rest);
  const unsigned seg = rest - b * A.segs.d;
  const unsigned vec = b * RT_MARCH_THREADS + threadIdx.x;
  if (item == 0) advance_seed(A.seed_in, A.seed_out, 0);
  if (vec >= A.nvec) return;
  const int nx = A.n[0], nk = A.n[3], nl = A.n[4], nm = A.n[5];
  const unsigned nvol3 = A.nvol3;
  // (l,m) in band order: bands of `band` values of the banded axis, the other
  // axis outside, the band's values inside
  const unsigned nb = (unsigned)(A.sweep ? nl : nm);
  const unsigned bi = A.band_full.div(lm);
  const unsigned r = lm - bi * A.band_full.d;
  const unsigned first = bi * A.band.d;
  const unsigned width = first + A.band.d <= nb ? A.band.d : nb - first;
  const unsigned outer = width == A.band.d ? A.band.div(r) : r / width;
  const unsigned banded = first + (r - outer * width);
  const int l = (int)(A.sweep ? banded : outer), m = (int)(A.sweep ? outer : banded);
  // the thread's cells
  const unsigned row = A.hx.div(vec);
  const int x0 = (int)(vec - row * A.hx.d) * V;
  const int z = (int)A.ny.div(row);
  const int y = (int)(row - (unsigned)z * A.ny.d);
  const int k0 = (int)seg * A.klen, k1 = k0 + A.klen < nk ? k0 + A.klen : nk;
  const int sl = (int)nvol3 * nk, sm = sl * nl;
  unsigned p = (unsigned)(m * nl + l) * (unsigned)sl + (unsigned)k0 * nvol3 + row * (unsigned)nx + (unsigned)x0;
  const unsigned kstep = nvol3 * 4u;

  unsigned oy[4], oz[4], ol[4], om[4];
  nb_bytes(A.n[1], nx, y, false, false, 0, oy);
  nb_bytes(A.n[2], nx * A.n[1], z, A.lower_refl != 0, A.upper_refl != 0, (nm - 1 - 2 * m) * sm, oz);
  nb_bytes(nl, sl, l, false, false, 0, ol);
  nb_bytes(nm, sm, m, false, false, 0, om);
  const bool ay = A.n[1] > 1, az = A.n[2] > 1, ak = nk > 1, al = nl > 1, am = nm > 1, ax = nx > 1;
  // left-face velocities: the cell below, or at coordinate 0 the face-0
  // plane, the cell's index with the axis (and so the part of the index
  // above it, divided by n) left out
  const int c[6] = {x0, y, z, k0, l, m};
  const unsigned st[6] = {1u, (unsigned)nx, (unsigned)(nx * A.n[1]), nvol3, (unsigned)sl, (unsigned)sm};
  const float* lp[6];
  unsigned ls[6];
  unsigned below = 0;   // the part of the index below axis a
#pragma unroll
  for (int a = 0; a < 6; a++) {
    if (c[a] > 0) {
      lp[a] = A.vel[a] + (p - st[a]);
      ls[a] = nvol3;
    } else {
      lp[a] = A.vlo[a] + (below + (p - below) / (unsigned)A.n[a]);
      ls[a] = a < 3 ? nvol3 / (unsigned)A.n[a] : nvol3;
    }
    below += (unsigned)c[a] * st[a];
  }
  AxisK Ky, Kz, Kl, Km;
  Ky.load(A, 1, y);
  Kz.load(A, 2, z);
  Kl.load(A, 4, l);
  Km.load(A, 5, m);
  float xr[V], xh[V], xo[V];
#pragma unroll
  for (int j = 0; j < V; j++) {
    xr[j] = -tab_at(A, 1, 0, x0 + j + 1);
    xh[j] = tab_at(A, 2, 0, x0 + j + 1);
    xo[j] = tab_at(A, 3, 0, x0 + j + 1);
  }
  const float xl = -tab_at(A, 1, 0, x0);
  const bool inl = x0 > 0, inl2 = x0 > 1, inr = x0 + V < nx, inr2 = x0 + V + 1 < nx;
  const float dthi = A.dthi, dtlo = A.dtlo;
  const unsigned seed = *A.seed_in;

  extern __shared__ __align__(16) unsigned char smem_raw[];
  const uint32_t slot0 = (uint32_t)__cvta_generic_to_shared(smem_raw) + threadIdx.x * (V * 4u);
  constexpr uint32_t SS = RT_MARCH_THREADS * V * 4u;   // bytes from slot to slot
  unsigned pb = p * 4u;
  Vec<V> Ec = ldv<V>(A.E, pb), E1 = Ec, Dm = Ec, D0 = Ec, fk = Ec;   // E(k), E(k+1), D(k-1/2), D(k+1/2), left k flux
  // slots: 0 E(k+2); 1-4 y, 5-8 z, 9-12 l, 13-16 m neighbours; 17-22 right, 23-26 left velocities; 27 rate
  // one group of copies per part of the loop below, in its order
  const auto commit = [] { asm volatile("cp.async.commit_group;"); };
  const auto fill4 = [&](int first, const unsigned o[4]) {
#pragma unroll
    for (int j = 0; j < 4; j++) slot_fill<V>(slot0 + (first + j) * SS, A.E, pb + o[j]);
  };
  if (ax) slot_fill<V>(slot0 + 17 * SS, A.vel[0], pb);
  commit();
  if (ay) fill4(1, oy), slot_fill<V>(slot0 + 18 * SS, A.vel[1], pb), slot_fill<V>(slot0 + 23 * SS, lp[1], 0u);
  commit();
  if (az) fill4(5, oz), slot_fill<V>(slot0 + 19 * SS, A.vel[2], pb), slot_fill<V>(slot0 + 24 * SS, lp[2], 0u);
  commit();
  if (ak) {
    slot_fill<V>(slot0, A.E, k0 + 2 < nk ? pb + 2u * kstep : (k0 + 1 < nk ? pb + kstep : pb));
    slot_fill<V>(slot0 + 20 * SS, A.vel[3], pb);
  }
  commit();
  if (al) fill4(9, ol), slot_fill<V>(slot0 + 21 * SS, A.vel[4], pb), slot_fill<V>(slot0 + 25 * SS, lp[4], 0u);
  commit();
  if (am) fill4(13, om), slot_fill<V>(slot0 + 22 * SS, A.vel[5], pb), slot_fill<V>(slot0 + 26 * SS, lp[5], 0u);
  commit();
  slot_fill<V>(slot0 + 27 * SS, A.lam, pb);
  commit();
  float X0 = 0.f, X1 = 0.f, X2 = 0.f, X3 = 0.f, vxl = 0.f;   // E beside the row's part and its left x velocity
  if (ax) {
    X1 = ld1(A.E, inl ? pb - 4u : pb);
    X0 = ld1(A.E, inl2 ? pb - 8u : (inl ? pb - 4u : pb));
    X2 = ld1(A.E, inr ? pb + 4u * V : pb + 4u * (V - 1));
    X3 = ld1(A.E, inr2 ? pb + 4u * V + 4u : (inr ? pb + 4u * V : pb + 4u * (V - 1)));
    vxl = __ldg(lp[0]);
  }
  if (ak) {
    const Vec<V> Em1 = ldv<V>(A.E, k0 > 0 ? pb - kstep : pb);
    const Vec<V> Em2 = ldv<V>(A.E, k0 > 1 ? pb - 2u * kstep : (k0 > 0 ? pb - kstep : pb));
    E1 = ldv<V>(A.E, k0 + 1 < nk ? pb + kstep : pb);
    Dm = vsub<V>(Ec, Em1);
    D0 = vsub<V>(E1, Ec);
    fk = vflux<V>(ldv<V>(lp[3], 0u), -tab_at(A, 1, 3, k0), vsub<V>(Em1, Em2), Dm, D0, Em1, Ec);
  }
#pragma unroll 1
  for (int k = k0; k < k1; k++) {
    const bool more = k + 1 < k1;
    const unsigned pn = pb + kstep;
    // the part's copies of a k ago are there: six groups are younger
    const auto filled = [] { asm volatile("cp.async.wait_group 6;" ::: "memory"); };
    Vec<V> E2 = Ec;
    AxisK Kk;
    if (V == 1 && ak) Kk.load(A, 3, k);   // (V = 4: 3% slower here than beside its use, V = 1: 8% faster)
    filled();
    Vec<V> acc;
#pragma unroll
    for (int j = 0; j < V; j++) acc.a[j] = 0.f;
    // ---- x: the faces x0-1/2 ... x0+V-1/2 of the row's part ----
    if (ax) {
      float X[V + 4];
#pragma unroll
      for (int j = 0; j < V; j++) X[j + 2] = Ec.a[j];
      X[1] = X1;
      X[0] = X0;
      X[V + 2] = X2;
      X[V + 3] = X3;
      const float vl = vxl;
      const Vec<V> vx = slot_take<V>(slot0 + 17 * SS);
      if (more) {
        slot_fill<V>(slot0 + 17 * SS, A.vel[0], pn);
        X1 = ld1(A.E, inl ? pn - 4u : pn);
        X0 = ld1(A.E, inl2 ? pn - 8u : (inl ? pn - 4u : pn));
        X2 = ld1(A.E, inr ? pn + 4u * V : pn + 4u * (V - 1));
        X3 = ld1(A.E, inr2 ? pn + 4u * V + 4u : (inr ? pn + 4u * V : pn + 4u * (V - 1)));
        lp[0] += ls[0];
        vxl = __ldg(lp[0]);
      }
      float D[V + 3];
#pragma unroll
      for (int j = 0; j < V + 3; j++) D[j] = X[j + 1] - X[j];
      float f[V + 1];
      f[0] = flux_d(vl, xl, D[0], D[1], D[2], X[1], X[2]);
      if constexpr (V == 1) {
        f[1] = flux_d(vx.a[0], xr[0], D[1], D[2], D[3], X[2], X[3]);
      } else {
#pragma unroll
        for (int j = 0; j < V; j += 2) {
          const float2 t = flux_d2(make_float2(vx.a[j], vx.a[j + 1]), make_float2(xr[j], xr[j + 1]),
                                   make_float2(D[j + 1], D[j + 2]), make_float2(D[j + 2], D[j + 3]),
                                   make_float2(D[j + 3], D[j + 4]), make_float2(X[j + 2], X[j + 3]),
                                   make_float2(X[j + 3], X[j + 4]));
          f[j + 1] = t.x;
          f[j + 2] = t.y;
        }
      }
#pragma unroll
      for (int j = 0; j < V; j++) acc.a[j] = div32(acc.a[j], f[j + 1], f[j], xh[j], xo[j]);
    }
    commit();
    auto axis = [&](int a, int se, int sv, int sf, const unsigned o[4], const AxisK& K) {
      Vec<V> e[4];
#pragma unroll
      for (int j = 0; j < 4; j++) e[j] = slot_take<V>(slot0 + (se + j) * SS);
      const Vec<V> vr = slot_take<V>(slot0 + sv * SS), vl = slot_take<V>(slot0 + sf * SS);
      if (more) {
#pragma unroll
        for (int j = 0; j < 4; j++) slot_fill<V>(slot0 + (se + j) * SS, A.E, pn + o[j]);
        slot_fill<V>(slot0 + sv * SS, A.vel[a], pn);
        lp[a] += ls[a];
        slot_fill<V>(slot0 + sf * SS, lp[a], 0u);
      }
      both_faces<V>(acc, K, vr, vl, e[0], e[1], Ec, e[2], e[3]);
    };
    filled();
    if (ay) axis(1, 1, 18, 23, oy, Ky);
    commit();
    filled();
    if (az) axis(2, 5, 19, 24, oz, Kz);
    commit();
    filled();
    if (ak) {
      if (V > 1) Kk.load(A, 3, k);
      E2 = slot_take<V>(slot0);
      const Vec<V> vk = slot_take<V>(slot0 + 20 * SS);
      if (more) {
        slot_fill<V>(slot0, A.E, k + 3 < nk ? pn + 2u * kstep : (k + 2 < nk ? pn + kstep : pn));
        slot_fill<V>(slot0 + 20 * SS, A.vel[3], pn);
      }
      const Vec<V> D1 = vsub<V>(E2, E1);
      const Vec<V> fr = vflux<V>(vk, Kk.r, Dm, D0, D1, Ec, E1);
      vdiv<V>(acc, fr, fk, Kk.hi, Kk.lo);
      fk = fr;
      Dm = D0;
      D0 = D1;
    }
    commit();
    filled();
    if (al) axis(4, 9, 21, 25, ol, Kl);
    commit();
    filled();
    if (am) axis(5, 13, 22, 26, om, Km);
    commit();
    filled();
    const Vec<V> lam = slot_take<V>(slot0 + 27 * SS);
    if (more) slot_fill<V>(slot0 + 27 * SS, A.lam, pn);
    commit();
    // ---- mean-flow term and update ----
    Vec<V> out;
    if constexpr (V == 1) {
      out.a[0] = upd32(Ec.a[0], acc.a[0], Ec.a[0] * lam.a[0], dthi, dtlo, sr_bits(p, seed));
    } else {
#pragma unroll
      for (int j = 0; j < V; j += 2) {
        const float2 t = upd2<true>(make_float2(Ec.a[j], Ec.a[j + 1]), make_float2(acc.a[j], acc.a[j + 1]),
                                    make_float2(lam.a[j], lam.a[j + 1]), dthi, dtlo,
                                    make_uint2(sr_bits(p + j, seed), sr_bits(p + j + 1, seed)));
        out.a[j] = t.x;
        out.a[j + 1] = t.y;
      }
    }
    float* o = reinterpret_cast<float*>(reinterpret_cast<char*>(A.Enew) + pb);
    if constexpr (V == 4) __stcs(reinterpret_cast<float4*>(o), make_float4(out.a[0], out.a[1], out.a[2], out.a[3]));
    else if constexpr (V == 2) __stcs(reinterpret_cast<float2*>(o), make_float2(out.a[0], out.a[1]));
    else __stcs(o, out.a[0]);
    Ec = E1;
    E1 = E2;
    p += nvol3;
    pb = pn;
  }
}

}  // namespace rt
