// applyBCids (src/BC.cpp:362-615) on moment arrays, FP32 and FP64: the
// boundary planes 1 and n - 2 of every axis are folded into one another
// (periodic axes, in the order X, Y, Z) and then doubled (the other axes).
//
// One launch. The nodes that the steps mix form closed groups: a node on the
// boundary planes of some axes, with those indices running over {1, n - 2}
// (2, 4 or 8 nodes). One thread reads a whole group, takes the steps in the
// reference's order in registers and writes the group back, so the sums are
// the ones that a launch per step gives, bit for bit. What bounds it is the
// latency of one read and one write, not the bytes (2 % of the node arrays):
// a thread per group and moment has them all in flight at once. On the GEM
// grid (131x67x67 nodes, FP64) 7 us against 32 us for three launches whose threads
// took the ten moments one after another.
#pragma once

#include "common.h"

namespace spb {

// A launch's grid: groups with x on its boundary planes, then those with y
// (x inside), then those with z (x and y inside).
struct FoldGroups {
  int n[3];           // nodes per axis
  int periodic[3];
  int cj, ck;         // group representatives along y and z: 1 (the pair) .. n - 3
  int ix, iy;         // inner x and y indices: 2 .. n - 3
  long fx, fy, fz;    // groups per region
};

inline FoldGroups fold_groups(int nxn, int nyn, int nzn, const int periodic[3]) {
  FoldGroups g;
  const int n[3] = {nxn, nyn, nzn};
  for (int a = 0; a < 3; ++a) {
    g.n[a] = n[a];
    g.periodic[a] = periodic[a] ? 1 : 0;
  }
  g.cj = nyn > 4 ? nyn - 3 : 1;
  g.ck = nzn > 4 ? nzn - 3 : 1;
  g.ix = nxn > 4 ? nxn - 4 : 0;
  g.iy = nyn > 4 ? nyn - 4 : 0;
  g.fx = (long)g.cj * g.ck;
  g.fy = (long)g.ix * g.ck;
  g.fz = (long)g.ix * g.iy;
  return g;
}

// One group t < fx + fy + fz of the array a.
template <typename T>
__device__ __forceinline__ void fold_group(const FoldGroups &g, T *__restrict__ a, long t) {
  int i = 1, j = 1, k = 1;
  bool pi = false, pj = false, pk = false;   // index on the boundary planes of its axis
  if (t < g.fx) {
    pi = true;
    j = 1 + (int)(t / g.ck);
    k = 1 + (int)(t % g.ck);
    pj = j == 1;
    pk = k == 1;
  } else if ((t -= g.fx) < g.fy) {
    pj = true;
    i = 2 + (int)(t / g.ck);
    k = 1 + (int)(t % g.ck);
    pk = k == 1;
  } else {
    t -= g.fy;
    pk = true;
    i = 2 + (int)(t / g.iy);
    j = 2 + (int)(t % g.iy);
  }
  const int hi = pi ? g.n[0] - 2 : i, hj = pj ? g.n[1] - 2 : j, hk = pk ? g.n[2] - 2 : k;
  long at[8];
  T v[8];
  bool in[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const bool x = e & 4, y = e & 2, z = e & 1;
    in[e] = (!x || pi) && (!y || pj) && (!z || pk);
    at[e] = ((long)(x ? hi : i) * g.n[1] + (y ? hj : j)) * g.n[2] + (z ? hk : k);
    v[e] = in[e] ? a[at[e]] : (T)0;
  }
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) {
    const int bit = 4 >> ax;
    if (g.periodic[ax] && (ax == 0 ? pi : ax == 1 ? pj : pk)) {
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (!(e & bit)) {
          const T sum = v[e] + v[e | bit];
          v[e] = sum;
          v[e | bit] = sum;
        }
    }
  }
#pragma unroll
  for (int ax = 0; ax < 3; ++ax)
    if (!g.periodic[ax] && (ax == 0 ? pi : ax == 1 ? pj : pk)) {
      const T f = g.n[ax] == 3 ? (T)4 : (T)2;   // three nodes: both planes are one
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] *= f;
    }
#pragma unroll
  for (int e = 0; e < 8; ++e)
    if (in[e]) a[at[e]] = v[e];
}

}  // namespace spb
