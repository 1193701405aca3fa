// rt_cells.cuh -- 32-bit index arithmetic of the one-thread-per-cell binary64
// passes (rt_exact.cu, rt_fast.cu): fields below 2^31 cells.
#pragma once
#include "rt_fast.cuh"
#include "rt_step.cuh"

namespace rt {

// strides and the divisors of the coordinates
struct CellGeom {
  unsigned ncell;
  int s[6];
  int ps[6][6];
  DivU32 n[5];     // divisors of the coordinates, x..l
};

inline CellGeom make_cells(const Dims& d) {
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

// face 0 of an axis whose lower ghosts copy the edge cell: no limited slope
__device__ __forceinline__ bool face0_is_copy(const Dims& d, int a) { return a != 2 || !d.lower_refl; }

}  // namespace rt
