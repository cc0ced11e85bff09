// Cell indices of the plain form: the reference's double arithmetic, and the
// float forms that give the same integers.
#pragma once

#include "common.h"

namespace spb {

// The double product (x - start) * inv, limited to [-8, n + 8] so that the
// int conversion below never overflows (NaN maps to -8). Exact for every
// position inside the grid, where the limit does not bite.
__device__ __forceinline__ double cell_coord(float p, double start, float inv, int n) {
  const double d = ((double)p - start) * (double)inv;
  return fmin(fmax(d, -8.0), (double)n + 8.0);
}

// Reference cell index of the mover: 2 + int((x - xStart) * invdx), the
// product in double, truncated toward zero (src/Mover.cpp:39-41).
__device__ __forceinline__ int cell_trunc(float p, double start, float inv, int n) {
  return 2 + __double2int_rz(cell_coord(p, start, inv, n));
}

// Reference cell index of the deposit: 2 + int(floor(...)) (src/Mover.cpp:399-401).
__device__ __forceinline__ int cell_floor(float p, double start, float inv, int n) {
  return 2 + __double2int_rd(cell_coord(p, start, inv, n));
}

// Keeps the node pair (i-1, i) inside [0, n-1]. The reference reads out of
// bounds for such particles; here they are flagged and clamped.
__device__ __forceinline__ int clamp_cell(int i, int n, int &bad) {
  if (i < 1) { bad = 1; return 1; }
  if (i > n - 1) { bad = 1; return n - 1; }
  return i;
}

// The deposit's three cell indices, clamped to the node array. FLOAT_CELLS
// (GeomDev::float_cells): the reference's double product of two floats is
// exact, so a float product rounded down has the same floor (every integer
// below 2^24 is a float, and rounding down cannot cross one), and compares
// alike with the integers -1 and n - 2; cells outside the node array (and NaN)
// take the general path, which flags them. The floor itself is an add rounded
// down against 1.5 * 2^23, whose neighbouring floats are the integers (no axis
// has 2^22 nodes): a conversion per axis kept the conversion unit half busy.
template <bool FLOAT_CELLS>
__device__ __forceinline__ void deposit_cell(const GeomDev &g, float x, float y, float z, int &ix,
                                             int &iy, int &iz, int &bad) {
  if (FLOAT_CELLS) {
    const float px = __fmul_rd(x, g.invdx), py = __fmul_rd(y, g.invdy),
                pz = __fmul_rd(z, g.invdz);
    if (px >= -1.0f && px < g.nxf && py >= -1.0f && py < g.nyf && pz >= -1.0f && pz < g.nzf) {
      constexpr float M = 12582912.0f;   // 1.5 * 2^23
      ix = 2 + __float_as_int(__fadd_rd(px, M)) - __float_as_int(M);
      iy = 2 + __float_as_int(__fadd_rd(py, M)) - __float_as_int(M);
      iz = 2 + __float_as_int(__fadd_rd(pz, M)) - __float_as_int(M);
      return;
    }
  }
  ix = clamp_cell(cell_floor(x, g.xStart, g.invdx, g.nxn), g.nxn, bad);
  iy = clamp_cell(cell_floor(y, g.yStart, g.invdy, g.nyn), g.nyn, bad);
  iz = clamp_cell(cell_floor(z, g.zStart, g.invdz, g.nzn), g.nzn, bad);
}

}  // namespace spb
