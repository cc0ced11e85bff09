// Plain-form kernels: the reference's mover_PC / interpP2G / mover_interp /
// applyBCids on device-resident SoA particles with the reference's precision
// types (float particles, fields and moments).
//
// Bit-exactness. The mover reproduces src/Mover.cpp:31-157 operation by
// operation: float arithmetic in the reference's evaluation order, the double
// promotions where the reference mixes float with double (cell index,
// denominator, final velocity, boundary tests), truncating (mover) and
// flooring (P2G) double-to-int conversions. This file is compiled with
// -fmad=false so no multiply-add pair is contracted into an FMA, matching a
// baseline x86-64 build of the reference. Particle outputs are therefore
// bit-identical to the reference CPU code; moments differ only by the order
// of the FP32 additions.
//
// Launch shape. One thread per particle: the particle SoA streams through once
// (coalesced 4-byte loads per array per warp), the 8-node gathers hit the packed
// fields, which stay L2-resident (28 MB at 128x64x64 cells).
#include "bc_fold.cuh"
#include "grid_ctx.h"
#include "kernels.h"
#include "plain_cells.cuh"
#include "warp_sum.cuh"

#include <atomic>
#include <type_traits>

namespace spb {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int TPB = 256;

struct Moments10 {
  float *m[10];
};

// x * y on a pair of floats, each half rounded to nearest on its own, as a
// scalar float multiply rounds it. The mover adds the two halves with scalar
// adds: a packed product that feeds a packed add came out rounded once with
// its sum, which the reference's float code does not do.
__device__ __forceinline__ float2 mul2_rn(float2 x, float2 y) {
  float2 d;
  asm("{\n\t.reg .b64 a, b, c;\n\t"
      "mov.b64 a, {%2, %3};\n\t"
      "mov.b64 b, {%4, %5};\n\t"
      "mul.rn.f32x2 c, a, b;\n\t"
      "mov.b64 {%0, %1}, c;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(x.x), "f"(x.y), "f"(y.x), "f"(y.y));
  return d;
}

// Particle boundary condition on one axis (src/Mover.cpp:103-157): an
// "above L" test in double, then a separate "below 0" test in float.
__device__ __forceinline__ void bc_axis(float &pos, float &vel, double L, int periodic) {
  if ((double)pos > L) {
    if (periodic) {
      pos = (float)((double)pos - L);
    } else {
      vel = -vel;
      pos = (float)(2.0 * L - (double)pos);
    }
  }
  if (pos < 0.0f) {
    if (periodic) {
      pos = (float)((double)pos + L);
    } else {
      vel = -vel;
      pos = -pos;
    }
  }
}

// Particle boundary condition of mover_PC_V (src/Mover.cpp:296-379): the
// periodic branch is mover_PC's; the reflecting branch first mirrors the
// position, then flips the velocity only if the MIRRORED position is still
// outside [0, L].
__device__ __forceinline__ void bc_axis_v(float &pos, float &vel, double L, int periodic) {
  if (periodic) {
    if ((double)pos > L) pos = (float)((double)pos - L);
    if (pos < 0.0f) pos = (float)((double)pos + L);
  } else {
    if ((double)pos > L) pos = (float)(2.0 * L - (double)pos);
    if (pos < 0.0f) pos = -pos;
    if ((double)pos > L) vel = -vel;
    if (pos < 0.0f) vel = -vel;
  }
}

// The mover's three cell indices, clamped to the node array. FLOAT_CELLS
// (GeomDev::float_cells): the reference's double product of two floats is
// exact, so a float product rounded toward zero has the same integer part
// (every integer below 2^24 is a float, and rounding cannot cross one), and
// the same comparisons with the integers -2 and n - 2 hold: cells outside the
// node array (and NaN) take the general path, which flags them.
template <bool FLOAT_CELLS>
__device__ __forceinline__ void cell_index(const GeomDev &g, float x, float y, float z, int &ix,
                                           int &iy, int &iz, int &bad) {
  if (FLOAT_CELLS) {
    const float px = __fmul_rz(x, g.invdx), py = __fmul_rz(y, g.invdy),
                pz = __fmul_rz(z, g.invdz);
    if (px > -2.0f && px < g.nxf && py > -2.0f && py < g.nyf && pz > -2.0f && pz < g.nzf) {
      ix = 2 + __float2int_rz(px);
      iy = 2 + __float2int_rz(py);
      iz = 2 + __float2int_rz(pz);
      return;
    }
  }
  ix = clamp_cell(cell_trunc(x, g.xStart, g.invdx, g.nxn), g.nxn, bad);
  iy = clamp_cell(cell_trunc(y, g.yStart, g.invdy, g.nyn), g.nyn, bad);
  iz = clamp_cell(cell_trunc(z, g.zStart, g.invdz, g.nzn), g.nzn, bad);
}

// (float)(1.0 / (1.0 + (double)o)), bit for bit, o >= 0. An approximate float
// reciprocal r of d = 1 + o and one third-order Newton step in double,
// r (1 + e + e^2) with e = 1 - d r, give the quotient to within one unit in
// its last place (e < 2^-21, so e^3 is far below it). Rounded to float that is
// the rounded quotient unless the quotient lies within two units of the
// midpoint of two floats; those, and o so large that r loses its precision
// (or NaN), take the division itself.
__device__ __forceinline__ float inv_one_plus(float o) {
  const double d = 1.0 + (double)o;
  float r0;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(1.0f + o));
  const double r = (double)r0;
  const double e = __fma_rn(-d, r, 1.0);
  double q = __fma_rn(r, __fma_rn(e, e, e), r);
  // the bits of a double below a float's last one
  const unsigned low = (unsigned)__double2loint(q) & 0x1fffffffu;
  if (!(o < 1e18f) || low - 0x0ffffffeu <= 4u) q = 1.0 / d;
  return (float)q;
}

// One particle of mover_PC (src/Mover.cpp:33-157); BCV = 1 gives mover_PC_V's
// boundary handling instead.
//
// Every result is the reference's, bit for bit; what its mixed arithmetic
// computes in double is formed in float where that is provably the same:
//   - the cell index: cell_index; 1 / (1 + omdtsq): inv_one_plus;
//   - 2 upt - u in double, then to float: the difference of two floats is
//     exact in double unless their exponents lie 30 or more apart, and then
//     both roundings give the larger one, so one fused multiply-add (which
//     rounds the exact difference once) is the same;
//   - x > L: a float is above L exactly if it is above the largest float not
//     above L.
// The six field sums add c = 0 (the upper z node) before c = 1, as the
// reference's loop does, and each product is rounded before it is added: the
// products come from packed multiplies over the two z nodes, the sums from
// scalar adds.
//
// The cell's eight nodes stay in registers over the iterations: most predicted
// positions stay in the particle's cell, and only the lanes that left it load
// again. The L1's data stage delivers 48 passes per warp and gather when the
// lanes share a cell and two to three times that when the arrays have drifted
// from cell order (it was 95 % busy then), so what the later iterations do not
// load counts twice.
template <int BCV, bool FLOAT_CELLS, int NITER>
__device__ __forceinline__ void move_one(const GeomDev &g, const PushDev &p,
                                         const PackedFields &F, float &x, float &y,
                                         float &z, float &u, float &v, float &w,
                                         int &bad) {
  const float xpt = x, ypt = y, zpt = z;
  const float qomdt2 = p.qomdt2, q2 = qomdt2 * qomdt2;
  float upt = 0.0f, vpt = 0.0f, wpt = 0.0f;
  float xc = x, yc = y, zc = z;
  const int sx = g.nyn * g.nzn, sy = g.nzn;   // nodes < 2^31 (spb_grid_create)
  const float2 inv2 = make_float2(g.invVOL, g.invVOL);
  int held = -1;        // cell whose eight nodes f holds
  float4 f[12];
#pragma unroll
  for (int i = 0; i < 12; ++i) f[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  const int niter = NITER ? NITER : p.niter;
#pragma unroll(NITER ? NITER : 1)
  for (int it = 0; it < niter; ++it) {
    int ix, iy, iz;
    cell_index<FLOAT_CELLS>(g, xc, yc, zc, ix, iy, iz, bad);
    const float2 xp = __ldg(g.xp + ix), yp = __ldg(g.yp + iy), zp = __ldg(g.zp + iz);
    const float xi[2] = {xc - xp.x, xp.y - xc};
    const float2 eta = make_float2(yc - yp.x, yp.y - yc);
    const float2 zeta = make_float2(zc - zp.x, zp.y - zc);
    float Ex = 0.0f, Ey = 0.0f, Ez = 0.0f, Bx = 0.0f, By = 0.0f, Bz = 0.0f;
    const int base = ix * sx + iy * sy + iz;
    if (base != held) {
      held = base;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float4 *row = F.eb + 3 * (long)(base - (r >> 1) * sx - (r & 1) * sy);
#pragma unroll
        for (int k = 0; k < 3; ++k) f[3 * r + k] = __ldg(row + k);
      }
    }
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      const float2 xe = mul2_rn(make_float2(xi[a], xi[a]), eta);
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        const float s = b ? xe.y : xe.x;
        // the weights of the two z nodes
        const float2 w2 = mul2_rn(mul2_rn(make_float2(s, s), zeta), inv2);
        const float4 f0 = f[6 * a + 3 * b], f1 = f[6 * a + 3 * b + 1], f2 = f[6 * a + 3 * b + 2];
        const float2 ex = mul2_rn(w2, make_float2(f0.x, f0.y));
        const float2 ey = mul2_rn(w2, make_float2(f0.z, f0.w));
        const float2 ez = mul2_rn(w2, make_float2(f1.x, f1.y));
        const float2 bx = mul2_rn(w2, make_float2(f1.z, f1.w));
        const float2 by = mul2_rn(w2, make_float2(f2.x, f2.y));
        const float2 bz = mul2_rn(w2, make_float2(f2.z, f2.w));
        Ex = Ex + ex.x + ex.y;
        Ey = Ey + ey.x + ey.y;
        Ez = Ez + ez.x + ez.y;
        Bx = Bx + bx.x + bx.y;
        By = By + by.x + by.y;
        Bz = Bz + bz.x + bz.y;
      }
    }
    const float omdtsq = q2 * (Bx * Bx + By * By + Bz * Bz);
    const float denom = inv_one_plus(omdtsq);
    const float ut = u + qomdt2 * Ex;
    const float vt = v + qomdt2 * Ey;
    const float wt = w + qomdt2 * Ez;
    const float udotb = ut * Bx + vt * By + wt * Bz;
    upt = (ut + qomdt2 * (vt * Bz - wt * By + qomdt2 * udotb * Bx)) * denom;
    vpt = (vt + qomdt2 * (wt * Bx - ut * Bz + qomdt2 * udotb * By)) * denom;
    wpt = (wt + qomdt2 * (ut * By - vt * Bx + qomdt2 * udotb * Bz)) * denom;
    xc = xpt + upt * p.dto2;
    yc = ypt + vpt * p.dto2;
    zc = zpt + wpt * p.dto2;
  }
  u = __fmaf_rn(2.0f, upt, -u);
  v = __fmaf_rn(2.0f, vpt, -v);
  w = __fmaf_rn(2.0f, wpt, -w);
  x = xpt + upt * p.dt_sub;
  y = ypt + vpt * p.dt_sub;
  z = zpt + wpt * p.dt_sub;
  // a particle inside [0, L] is left alone by both boundary conditions
  auto bc = [&](float &pos, float &vel, float Lf, double L, int periodic) {
    if (pos > Lf || pos < 0.0f) {
      if (BCV == 0)
        bc_axis(pos, vel, L, periodic);
      else
        bc_axis_v(pos, vel, L, periodic);
    }
  };
  bc(x, u, g.Lfx, g.Lx, p.periodic[0]);
  bc(y, v, g.Lfy, g.Ly, p.periodic[1]);
  bc(z, w, g.Lfz, g.Lz, p.periodic[2]);
}

// The 40 summands of one x half of a particle (src/Mover.cpp:399-570), each
// computed as the reference does (weight = q * xi * eta * zeta * invVOL,
// then e.g. (u * weight) * invVOL, no FMA), in the packed, lane-permuted
// layout of warp_sum80: t[(b * 2 + c) * 5 + k] = (moment k, moment k + 5) of
// node slot (a, b, c), slot a = `a` given, with physical node (a ^ bit4(lane),
// b ^ bit3(lane), c ^ bit2(lane)); the physical node (a, b, c) is (ix - a,
// iy - b, iz - c). ADD: added to t (else stored).
template <bool ADD>
__device__ __forceinline__ void half_terms(const GeomDev &g, float x, float y, float z, float u,
                                           float v, float w, float q, float2 (&t)[20], int lane,
                                           int a) {
  int ignored = 0;   // the range flag was raised when the cell key was formed
  const int ix = clamp_cell(cell_floor(x, g.xStart, g.invdx, g.nxn), g.nxn, ignored);
  const int iy = clamp_cell(cell_floor(y, g.yStart, g.invdy, g.nyn), g.nyn, ignored);
  const int iz = clamp_cell(cell_floor(z, g.zStart, g.invdz, g.nzn), g.nzn, ignored);
  const float xi0 = x - __ldg(g.xn + ix - 1), xi1 = __ldg(g.xn + ix) - x;
  const float eta0 = y - __ldg(g.yn + iy - 1), eta1 = __ldg(g.yn + iy) - y;
  const float zeta0 = z - __ldg(g.zn + iz - 1), zeta1 = __ldg(g.zn + iz) - z;
  const bool pb = lane & 8, pc = lane & 4;
  const float xia = (a ^ ((lane >> 4) & 1)) ? xi1 : xi0;
  const float eta[2] = {pb ? eta1 : eta0, pb ? eta0 : eta1};
  const float zeta[2] = {pc ? zeta1 : zeta0, pc ? zeta0 : zeta1};
  const float uu = u * u, uv = u * v, uw = u * w, vv = v * v, vw = v * w, ww = w * w;
  const float inv = g.invVOL;
#pragma unroll
  for (int b = 0; b < 2; ++b)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const float wgt = q * xia * eta[b] * zeta[c] * inv;
      float2 *o = t + (b * 2 + c) * 5;
      const float2 n[5] = {make_float2(wgt * inv, (uv * wgt) * inv),
                           make_float2((u * wgt) * inv, (uw * wgt) * inv),
                           make_float2((v * wgt) * inv, (vv * wgt) * inv),
                           make_float2((w * wgt) * inv, (vw * wgt) * inv),
                           make_float2((uu * wgt) * inv, (ww * wgt) * inv)};
#pragma unroll
      for (int k = 0; k < 5; ++k) o[k] = ADD ? __fadd2_rn(o[k], n[k]) : n[k];
    }
}

struct Particle {
  float x, y, z, u, v, w, q;
};

// One 16-byte add to global memory (p 16-byte aligned): one L2 atomic
// operation for four floats.
__device__ __forceinline__ void red_v4(float *p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b),
               "f"(c), "f"(d)
               : "memory");
}

// The plain deposit's accumulator: the ten moments of node n side by side,
// acc[n * ACC_STRIDE + m] (m = rhon, Jx, Jy, Jz, pxx, pxy, pxz, pyy, pyz, pzz;
// two pad floats keep every node's record on a 16-byte boundary). A
// particle's 80 terms then land in about a dozen 32-byte sectors instead of
// the forty that ten separate arrays take; k_fold_acc adds it into the ten
// arrays afterwards.
constexpr int ACC_STRIDE = 12;

// Where a plain deposit adds: the accumulator (ACC) or, when none could be
// allocated, the ten moment arrays themselves.
struct DepTarget {
  float *acc;
  Moments10 mom;
};

// Adds v to moment m of node n.
template <bool ACC>
__device__ __forceinline__ void dep_add(const DepTarget &T, long n, int m, float v) {
  if (ACC)
    atomicAdd(T.acc + n * ACC_STRIDE + m, v);
  else
    atomicAdd(T.mom.m[m] + n, v);
}

// Adds v0..v3 to moments 4 grp .. 4 grp + 3 of node n (moments below 10).
template <bool ACC>
__device__ __forceinline__ void dep_add4(const DepTarget &T, long n, int grp, float v0, float v1,
                                         float v2, float v3) {
  if (ACC) {
    red_v4(T.acc + n * ACC_STRIDE + 4 * grp, v0, v1, v2, v3);
  } else {
    const float v[4] = {v0, v1, v2, v3};
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (4 * grp + i < 10) atomicAdd(T.mom.m[4 * grp + i] + n, v[i]);
  }
}

// Adds one warp's deposits to the accumulator. For each of up to four
// distinct cells among the warp's particles (cell-ordered particles give one
// or two), the members compute their terms and the warp sums them (the steps
// of warp_sum80, one x half of the terms at a time) and adds the 80 totals;
// each lone particle of a further cell (a particle that moved, unordered
// input) is spread over 24 lanes, four moments of one node each, added with
// one 16-byte add per lane. Terms are recomputed per round rather than kept,
// which keeps the registers down. All 32 lanes call.
template <bool ACC>
__device__ __forceinline__ void deposit_warp(const GeomDev &g, const DepTarget &T, bool valid,
                                             const Particle &p, int &bad) {
  const int lane = threadIdx.x & 31;
  const int sx = g.nyn * g.nzn, sy = g.nzn;   // nodes < 2^31 (spb_grid_create)
  int key = 0;
  if (valid) {
    const int ix = clamp_cell(cell_floor(p.x, g.xStart, g.invdx, g.nxn), g.nxn, bad);
    const int iy = clamp_cell(cell_floor(p.y, g.yStart, g.invdy, g.nyn), g.nyn, bad);
    const int iz = clamp_cell(cell_floor(p.z, g.zStart, g.invdz, g.nzn), g.nzn, bad);
    key = (ix * g.nyn + iy) * g.nzn + iz;
  }
  // this lane's totals after warp_sum80: physical node (bit4, bit3, bit2),
  // moments mbase + [lo, hi)
  const int na = (lane >> 4) & 1, nb = (lane >> 3) & 1, nc = (lane >> 2) & 1;
  const int mbase = 5 * ((lane >> 1) & 1);
  const int lo = (lane & 1) ? 3 : 0, hi = (lane & 1) ? 5 : 3;
  unsigned remaining = __ballot_sync(FULL, valid);
#pragma unroll 1
  for (int round = 0; round < 4 && remaining; ++round) {
    const int leader = __ffs(remaining) - 1;
    const int k = __shfl_sync(FULL, key, leader);
    const bool member = valid && key == k;
    const unsigned members = __ballot_sync(FULL, member);
    remaining &= ~members;
    if (__popc(members) < 2 && round > 0) continue;   // lone particle: direct atomics below
    // warp_sum80 in halves: the slot a = 1 terms go to lane ^ 16, whose slot
    // a = 0 holds the same physical x node, and each lane adds its own slot
    // a = 0 terms to what it received (40 live values instead of 80)
    float2 t[20];
    if (member) {
      half_terms<false>(g, p.x, p.y, p.z, p.u, p.v, p.w, p.q, t, lane, 1);
    } else {
#pragma unroll
      for (int j = 0; j < 20; ++j) t[j] = make_float2(0.0f, 0.0f);
    }
#pragma unroll
    for (int j = 0; j < 20; ++j) t[j] = shfl_xor2(t[j], 16);
    if (member) half_terms<true>(g, p.x, p.y, p.z, p.u, p.v, p.w, p.q, t, lane, 0);
    float r[5];
    warp_sum80_tail(t, r, lane);
    const int node = k - na * sx - nb * sy - nc;
#pragma unroll
    for (int i = 0; i < 5; ++i)
      if (i >= lo && i < hi) dep_add<ACC>(T, node, mbase + i, r[i]);
    if (member) valid = false;   // done
  }
  // lone particles of further cells, one at a time: lane j < 24 takes node
  // j / 3 and moments 4 (j % 3) .. 4 (j % 3) + 3 of the particle, each term
  // computed as half_terms does, and adds them with one 16-byte add
  unsigned lone = __ballot_sync(FULL, valid);
  if (lone) {
    const int ix = (int)(key / sx), iy = (int)((key / sy) % g.nyn), iz = (int)(key % sy);
    float d[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};   // xi0, xi1, eta0, eta1, zeta0, zeta1
    if (valid) {
      d[0] = p.x - __ldg(g.xn + ix - 1);
      d[1] = __ldg(g.xn + ix) - p.x;
      d[2] = p.y - __ldg(g.yn + iy - 1);
      d[3] = __ldg(g.yn + iy) - p.y;
      d[4] = p.z - __ldg(g.zn + iz - 1);
      d[5] = __ldg(g.zn + iz) - p.z;
    }
    const float inv = g.invVOL;
    while (lone) {
      const int L = __ffs(lone) - 1;
      lone &= lone - 1;
      float e[6];
#pragma unroll
      for (int j = 0; j < 6; ++j) e[j] = __shfl_sync(FULL, d[j], L);
      const float q = __shfl_sync(FULL, p.q, L), u = __shfl_sync(FULL, p.u, L);
      const float v = __shfl_sync(FULL, p.v, L), w = __shfl_sync(FULL, p.w, L);
      const int k = __shfl_sync(FULL, key, L);
      if (lane < 24) {
        const int node = lane / 3, grp = lane % 3;
        const int a = node >> 2, b = (node >> 1) & 1, c = node & 1;
        const float wgt = q * (a ? e[1] : e[0]) * (b ? e[3] : e[2]) * (c ? e[5] : e[4]) * inv;
        // moment factors of the group: (1, u, v, w), (uu, uv, uw, vv) or
        // (vw, ww, 0, 0) (rhon's (1 * wgt) * inv is the reference's wgt * inv
        // exactly; the pad slots add zeros)
        const float f0 = grp == 0 ? 1.0f : (grp == 1 ? u * u : v * w);
        const float f1 = grp == 0 ? u : (grp == 1 ? u * v : w * w);
        const float f2 = grp == 0 ? v : (grp == 1 ? u * w : 0.0f);
        const float f3 = grp == 0 ? w : (grp == 1 ? v * v : 0.0f);
        dep_add4<ACC>(T, k - a * sx - b * sy - c, grp, (f0 * wgt) * inv, (f1 * wgt) * inv,
                      (f2 * wgt) * inv, (f3 * wgt) * inv);
      }
    }
  }
}

// One lone particle (its cell's only member in a group) of a warp's
// deposit: lane j < 24 takes node j / 3 and moments 4 (j % 3) .. 4 (j % 3) + 3,
// each term computed as half_terms does, added with one 16-byte add. Every
// lane passes the same particle and key. All 32 lanes call.
template <bool ACC>
__device__ __forceinline__ void deposit_lone(const GeomDev &g, const DepTarget &T,
                                             const Particle &p, int key) {
  const int lane = threadIdx.x & 31;
  const int sx = g.nyn * g.nzn, sy = g.nzn;
  if (lane >= 24) return;
  const int ix = key / sx, iy = (key / sy) % g.nyn, iz = key % sy;
  const float e[6] = {p.x - __ldg(g.xn + ix - 1), __ldg(g.xn + ix) - p.x,
                      p.y - __ldg(g.yn + iy - 1), __ldg(g.yn + iy) - p.y,
                      p.z - __ldg(g.zn + iz - 1), __ldg(g.zn + iz) - p.z};
  const float inv = g.invVOL, u = p.u, v = p.v, w = p.w;
  const int node = lane / 3, grp = lane % 3;
  const int a = node >> 2, b = (node >> 1) & 1, c = node & 1;
  const float wgt = p.q * (a ? e[1] : e[0]) * (b ? e[3] : e[2]) * (c ? e[5] : e[4]) * inv;
  const float f0 = grp == 0 ? 1.0f : (grp == 1 ? u * u : v * w);
  const float f1 = grp == 0 ? u : (grp == 1 ? u * v : w * w);
  const float f2 = grp == 0 ? v : (grp == 1 ? u * w : 0.0f);
  const float f3 = grp == 0 ? w : (grp == 1 ? v * v : 0.0f);
  dep_add4<ACC>(T, key - a * sx - b * sy - c, grp, (f0 * wgt) * inv, (f1 * wgt) * inv,
                (f2 * wgt) * inv, (f3 * wgt) * inv);
}

// The grouped plain deposit. A CTA takes a chunk of GP_CHUNK consecutive
// particles into shared memory and groups them by cell (a shared-memory hash
// table of GP_SLOTS cells; each warp inserts each of its distinct cells once),
// then every group is deposited by one warp: its lanes take the group's
// particles in turn and accumulate their terms in the packed layout of
// warp_sum80 (one x half of the terms at a time), and one warp reduction and
// 80 adds serve the whole group instead of one per 32 particles. Groups of up
// to three particles deposit particle by particle (deposit_lone). A chunk
// with more distinct cells than the table holds (unordered input) deposits
// warp by warp (deposit_warp).
constexpr int GP_TPB = 256;
constexpr int GP_PER_THREAD = 4;
constexpr int GP_CHUNK = GP_TPB * GP_PER_THREAD;
constexpr int GP_SLOTS = 256;
static_assert(GP_SLOTS == GP_TPB, "one table slot per thread in the scans");

struct GroupSmem {
  float p[7][GP_CHUNK];                 // x, y, z, u, v, w, q
  int key[GP_CHUNK];                    // node-space cell of each particle
  short slot[GP_CHUNK];                 // its table slot
  unsigned short order[GP_CHUNK];       // chunk indices grouped by slot
  int hkey[GP_SLOTS], hcnt[GP_SLOTS], hstart[GP_SLOTS], hcur[GP_SLOTS];
  int wsum[GP_TPB / 32];
  int full;
};

__device__ __forceinline__ Particle smem_particle(const GroupSmem &S, int j) {
  return Particle{S.p[0][j], S.p[1][j], S.p[2][j], S.p[3][j], S.p[4][j], S.p[5][j], S.p[6][j]};
}

// (Particles in the arrays' own order: interpP2G below P2S_MIN particles, and
// deposits whose scratch for the cell order cannot be had.)
template <bool ACC>
__global__ void __launch_bounds__(GP_TPB) k_plain_p2g_grouped(
    GeomDev g, const float *__restrict__ x, const float *__restrict__ y,
    const float *__restrict__ z, const float *__restrict__ u, const float *__restrict__ v,
    const float *__restrict__ w, const float *__restrict__ q, long n,
    const __grid_constant__ DepTarget T, int *__restrict__ err) {
  __shared__ GroupSmem S;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long base = (long)blockIdx.x * GP_CHUNK;
  const int cnt = (int)min((long)GP_CHUNK, n - base);
  S.hkey[tid] = -1;
  S.hcnt[tid] = 0;
  if (tid == 0) S.full = 0;
  __syncthreads();
  int bad = 0;
  const float *const src[7] = {x, y, z, u, v, w, q};
#pragma unroll
  for (int r = 0; r < GP_PER_THREAD; ++r) {
    const int j = tid + r * GP_TPB;
    const bool valid = j < cnt;
    int key = -1;
    if (valid) {
      const long i = base + j;
#pragma unroll
      for (int a = 0; a < 7; ++a) S.p[a][j] = src[a][i];
      const int ix = clamp_cell(cell_floor(S.p[0][j], g.xStart, g.invdx, g.nxn), g.nxn, bad);
      const int iy = clamp_cell(cell_floor(S.p[1][j], g.yStart, g.invdy, g.nyn), g.nyn, bad);
      const int iz = clamp_cell(cell_floor(S.p[2][j], g.zStart, g.invdz, g.nzn), g.nzn, bad);
      key = (ix * g.nyn + iy) * g.nzn + iz;
      S.key[j] = key;
    }
    // one insertion per distinct cell of the warp (linear probing)
    const unsigned peers = __match_any_sync(FULL, key);
    const int leader = __ffs(peers) - 1;
    int slot = -1;
    if (valid && lane == leader) {
      unsigned h = ((unsigned)key * 2654435761u) >> 24;
      for (int t = 0; t < GP_SLOTS; ++t) {
        const int prev = atomicCAS(&S.hkey[h], -1, key);
        if (prev == -1 || prev == key) {
          slot = (int)h;
          break;
        }
        h = (h + 1) & (GP_SLOTS - 1);
      }
      if (slot < 0)
        S.full = 1;
      else
        atomicAdd(&S.hcnt[slot], __popc(peers));
    }
    slot = __shfl_sync(FULL, slot, leader);
    if (valid) S.slot[j] = (short)slot;
  }
  __syncthreads();
  if (S.full) {
    // more distinct cells than table slots: the per-warp deposit, in order
#pragma unroll 1
    for (int r = 0; r < GP_PER_THREAD; ++r) {
      const int j = tid + r * GP_TPB;
      const bool valid = j < cnt;
      Particle p{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (valid) p = smem_particle(S, j);
      deposit_warp<ACC>(g, T, valid, p, bad);
    }
    if (bad) atomicOr(err, ERRBIT_OUT_OF_GRID);
    return;
  }
  // group starts: exclusive scan of the slot counts
  {
    const int c = S.hcnt[tid];
    int xs = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(FULL, xs, o);
      if (lane >= o) xs += t;
    }
    if (lane == 31) S.wsum[warp] = xs;
    __syncthreads();
    int pre = 0;
    for (int k = 0; k < warp; ++k) pre += S.wsum[k];
    S.hstart[tid] = pre + xs - c;
    S.hcur[tid] = pre + xs - c;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < GP_PER_THREAD; ++r) {
    const int j = tid + r * GP_TPB;
    const bool valid = j < cnt;
    const int slot = valid ? S.slot[j] : -1;
    const unsigned peers = __match_any_sync(FULL, slot);
    const int leader = __ffs(peers) - 1;
    int first = 0;
    if (valid && lane == leader) first = atomicAdd(&S.hcur[slot], __popc(peers));
    first = __shfl_sync(FULL, first, leader);
    if (valid) S.order[first + __popc(peers & ((1u << lane) - 1u))] = (unsigned short)j;
  }
  __syncthreads();
  const int sx = g.nyn * g.nzn, sy = g.nzn;
  const int na = (lane >> 4) & 1, nb = (lane >> 3) & 1, nc = (lane >> 2) & 1;
  const int mbase = 5 * ((lane >> 1) & 1);
  const int lo = (lane & 1) ? 3 : 0, hi = (lane & 1) ? 5 : 3;
#pragma unroll 1
  for (int s = warp; s < GP_SLOTS; s += GP_TPB / 32) {
    const int c = S.hcnt[s];
    if (c == 0) continue;
    const int st = S.hstart[s], key = S.hkey[s];
    if (c <= 3) {
      for (int m = 0; m < c; ++m) deposit_lone<ACC>(g, T, smem_particle(S, S.order[st + m]), key);
      continue;
    }
    float2 t[20];
#pragma unroll
    for (int i = 0; i < 20; ++i) t[i] = make_float2(0.0f, 0.0f);
    for (int m = lane; m < c; m += 32) {
      const Particle p = smem_particle(S, S.order[st + m]);
      half_terms<true>(g, p.x, p.y, p.z, p.u, p.v, p.w, p.q, t, lane, 1);
    }
#pragma unroll
    for (int i = 0; i < 20; ++i) t[i] = shfl_xor2(t[i], 16);
    for (int m = lane; m < c; m += 32) {
      const Particle p = smem_particle(S, S.order[st + m]);
      half_terms<true>(g, p.x, p.y, p.z, p.u, p.v, p.w, p.q, t, lane, 0);
    }
    float r[5];
    warp_sum80_tail(t, r, lane);
    const int node = key - na * sx - nb * sy - nc;
#pragma unroll
    for (int i = 0; i < 5; ++i)
      if (i >= lo && i < hi) dep_add<ACC>(T, node, mbase + i, r[i]);
  }
  if (bad) atomicOr(err, ERRBIT_OUT_OF_GRID);
}

// A CTA's nodes go through shared memory, so that a warp stores 512 consecutive
// bytes at a time and not 32 pieces 48 bytes apart: 256x256x256 cells 273 -> 219 us,
// 128x64x64 25 -> 22 with the launch.
__global__ void __launch_bounds__(TPB) k_pack_fields(const float *__restrict__ ex,
                                                     const float *__restrict__ ey,
                                                     const float *__restrict__ ez,
                                                     const float *__restrict__ bx,
                                                     const float *__restrict__ by,
                                                     const float *__restrict__ bz,
                                                     float4 *__restrict__ eb, long nodes,
                                                     int nzn) {
  __shared__ float4 s[3 * TPB];
  const int t = threadIdx.x;
  const long base = blockIdx.x * (long)TPB, i = base + t;
  if (i < nodes) {
    const long l = i % nzn ? i - 1 : i;   // the node below (a row's first is never read)
    s[3 * t] = make_float4(ex[i], ex[l], ey[i], ey[l]);
    s[3 * t + 1] = make_float4(ez[i], ez[l], bx[i], bx[l]);
    s[3 * t + 2] = make_float4(by[i], by[l], bz[i], bz[l]);
  }
  __syncthreads();
  const int count = 3 * (int)min((long)TPB, nodes - base);
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (t + k * TPB < count) eb[3 * base + t + k * TPB] = s[t + k * TPB];
}

// Seven CTAs of 128 threads per SM (72 registers, 44 bytes of spills): the
// pass is bound by the L1's data stage and by issue alike, and 28 warps keep
// both busier than 24 without spills (3 to 4 % slower near cell order, as much
// faster in long drifted arrays) or 32 with fewer nodes held. 65.5M electrons of
// the GEM workload up to 15 steps after their arrays were in cell order: 2663 ->
// 2300 us with the packing of the fields; 2.4M
// electrons some cycles after the last sort: 166 -> 133 us.
constexpr int MOVER_TPB = 128;
template <int BCV, bool FLOAT_CELLS, int NITER>
__global__ void __launch_bounds__(MOVER_TPB, 7) k_plain_mover(GeomDev g, PushDev p, PackedFields F,
                                                     float *__restrict__ x, float *__restrict__ y,
                                                     float *__restrict__ z, float *__restrict__ u,
                                                     float *__restrict__ v, float *__restrict__ w,
                                                     long n, int *__restrict__ err) {
  const long i = blockIdx.x * (long)MOVER_TPB + threadIdx.x;
  if (i >= n) return;
  float px = x[i], py = y[i], pz = z[i], pu = u[i], pv = v[i], pw = w[i];
  int bad = 0;
  move_one<BCV, FLOAT_CELLS, NITER>(g, p, F, px, py, pz, pu, pv, pw, bad);
  x[i] = px;
  y[i] = py;
  z[i] = pz;
  u[i] = pu;
  v[i] = pv;
  w[i] = pw;
  if (bad) atomicOr(err, ERRBIT_OUT_OF_GRID);
}

// mover_interp in one pass (fused_interp says when): a warp deposits the
// particles that it has just moved.
template <bool ACC, bool FLOAT_CELLS, int NITER>
__global__ void __launch_bounds__(TPB) k_plain_mover_interp(
    GeomDev g, PushDev p, PackedFields F, float *__restrict__ x, float *__restrict__ y,
    float *__restrict__ z, float *__restrict__ u, float *__restrict__ v,
    float *__restrict__ w, const float *__restrict__ q, long n,
    const __grid_constant__ DepTarget T, int *__restrict__ err) {
  const long i = blockIdx.x * (long)TPB + threadIdx.x;
  const bool valid = i < n;
  Particle pt{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  int bad = 0;
  if (valid) {
    pt = Particle{x[i], y[i], z[i], u[i], v[i], w[i], q[i]};
    move_one<0, FLOAT_CELLS, NITER>(g, p, F, pt.x, pt.y, pt.z, pt.u, pt.v, pt.w, bad);
    x[i] = pt.x;
    y[i] = pt.y;
    z[i] = pt.z;
    u[i] = pt.u;
    v[i] = pt.v;
    w[i] = pt.w;
  }
  deposit_warp<ACC>(g, T, valid, pt, bad);
  if (bad) atomicOr(err, ERRBIT_OUT_OF_GRID);
}

// sumOverSpecies (src/InterpDensNet.cpp:120-146) on the device: net moment m
// of node i = the species' values added in species order, from zero, as the
// reference's loop does (so the float sums are bit-identical).
constexpr int SUM_MAX_SPECIES = 32;
struct SpeciesBases {
  const float *b[SUM_MAX_SPECIES];   // [10][nodes] moments of each species
};

__global__ void __launch_bounds__(TPB) k_sum_species(SpeciesBases S, int ns, long nodes,
                                                     float *__restrict__ net) {
  const long total = 10 * nodes;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total;
       i += (long)gridDim.x * blockDim.x) {
    float acc = 0.0f;
    for (int s = 0; s < ns; ++s) acc += S.b[s][i];
    net[i] = acc;
  }
}

// mom[m][n] += acc[n * ACC_STRIDE + m] for the non-zero entries (atomically:
// the pipeline streams of the drop-in fold into the same arrays).
__global__ void __launch_bounds__(TPB) k_fold_acc(const float4 *__restrict__ acc, long nodes,
                                                  Moments10 M) {
  for (long n = blockIdx.x * (long)blockDim.x + threadIdx.x; n < nodes;
       n += (long)gridDim.x * blockDim.x) {
    const float4 a = acc[3 * n], b = acc[3 * n + 1], c = acc[3 * n + 2];
    const float v[10] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y};
#pragma unroll
    for (int m = 0; m < 10; ++m)
      if (v[m] != 0.0f) atomicAdd(M.m[m] + n, v[m]);
  }
}

// applyBCids on the ten moments (blockIdx.y), see bc_fold.cuh.
__global__ void __launch_bounds__(TPB) k_bc_fold(const __grid_constant__ Moments10 M,
                                                 FoldGroups g) {
  const long t = blockIdx.x * (long)TPB + threadIdx.x;
  if (t < g.fx + g.fy + g.fz) fold_group(g, M.m[blockIdx.y], t);
}

inline unsigned blocks_for(long n) { return (unsigned)ceil_div(n, TPB); }

// Deposits of at least this many particles sort them by cell first.
constexpr long P2S_MIN = SORTED_P2G_MIN;

}  // namespace

int launch_pack_fields(const float *const f[6], float4 *eb, long nodes, int nzn,
                       cudaStream_t s) {
  k_pack_fields<<<blocks_for(nodes), TPB, 0, s>>>(f[0], f[1], f[2], f[3], f[4], f[5], eb, nodes,
                                                  nzn);
  SPB_CUDA(cudaGetLastError());
  g_launches++;
  return SPB_OK;
}

int launch_plain_mover(const GeomDev &g, const PushDev &p, const PackedFields &F, float *x,
                       float *y, float *z, float *u, float *v, float *w, long n, int *err,
                       cudaStream_t s, int bc_variant) {
  if (n <= 0) return SPB_OK;
  // three iterations, the usual number, unrolled
  auto pick = [&](auto bcv) {
    constexpr int B = decltype(bcv)::value;
    if (!g.float_cells) return k_plain_mover<B, false, 0>;
    return p.niter == 3 ? k_plain_mover<B, true, 3> : k_plain_mover<B, true, 0>;
  };
  auto *const kernel = bc_variant == 0 ? pick(std::integral_constant<int, 0>())
                                       : pick(std::integral_constant<int, 1>());
  kernel<<<(unsigned)ceil_div(n, MOVER_TPB), MOVER_TPB, 0, s>>>(g, p, F, x, y, z, u, v, w, n,
                                                              err);
  SPB_CUDA(cudaGetLastError());
  g_launches++;
  return SPB_OK;
}

int launch_sum_species(const float *const *bases, int ns, long nodes, float *net,
                       cudaStream_t s) {
  if (ns < 1 || ns > SUM_MAX_SPECIES) return fail(SPB_ERR_UNSUPPORTED, "1..32 species");
  SpeciesBases S{};
  for (int i = 0; i < ns; ++i) S.b[i] = bases[i];
  k_sum_species<<<(unsigned)std::min<long>(ceil_div(10 * nodes, TPB), 4096), TPB, 0, s>>>(
      S, ns, nodes, net);
  SPB_CUDA(cudaGetLastError());
  g_launches++;
  return SPB_OK;
}

namespace {
// The device's stream-ordered pool keeps freed memory for reuse (once per
// device), so the per-deposit accumulators map nothing after the first.
void keep_pool_memory() {
  static std::atomic<unsigned long long> done{0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64 || ((done.load() >> dev) & 1ull)) {
    cudaGetLastError();
    return;
  }
  cudaMemPool_t pool;
  if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
    unsigned long long keep = ~0ull;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  }
  cudaGetLastError();
  done |= 1ull << dev;
}

}  // namespace

namespace {
std::atomic<int> g_deposit_mode{SPB_DEPOSIT_ACCUMULATOR};
}  // namespace

void *pool_alloc(size_t bytes, cudaStream_t s) {
  keep_pool_memory();
  void *p = nullptr;
  if (cudaMallocAsync(&p, std::max<size_t>(bytes, 1), s) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return p;
}

void pool_free(void *p, cudaStream_t s) {
  if (p) cudaFreeAsync(p, s);
}

float *plain_acc_alloc(const GeomDev &g, cudaStream_t s) {
  if (g_deposit_mode.load() == SPB_DEPOSIT_DIRECT) return nullptr;
  keep_pool_memory();
  const size_t bytes = (size_t)g.nxn * g.nyn * g.nzn * ACC_STRIDE * sizeof(float);
  float *acc = nullptr;
  if (cudaMallocAsync(reinterpret_cast<void **>(&acc), bytes, s) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  // the 16-byte adds need the alignment (pool allocations have it)
  if ((reinterpret_cast<uintptr_t>(acc) & 15u) || cudaMemsetAsync(acc, 0, bytes, s) != cudaSuccess) {
    cudaGetLastError();
    cudaFreeAsync(acc, s);
    cudaGetLastError();
    return nullptr;
  }
  return acc;
}

int plain_acc_fold(float *acc, const GeomDev &g, float *const mom[10], cudaStream_t s) {
  if (!acc) return SPB_OK;
  const long nodes = (long)g.nxn * g.nyn * g.nzn;
  Moments10 M;
  for (int m = 0; m < 10; ++m) M.m[m] = mom[m];
  k_fold_acc<<<(unsigned)std::min<long>(ceil_div(nodes, TPB), 4096), TPB, 0, s>>>(
      reinterpret_cast<const float4 *>(acc), nodes, M);
  const cudaError_t e = cudaGetLastError();
  cudaFreeAsync(acc, s);
  if (e != cudaSuccess) return fail_cuda(e, "k_fold_acc");
  g_launches++;
  return SPB_OK;
}

namespace {
DepTarget target(float *acc, float *const mom[10]) {
  DepTarget T;
  T.acc = acc;
  for (int m = 0; m < 10; ++m) T.mom.m[m] = mom[m];
  return T;
}
}  // namespace

int launch_plain_p2g_into(const GeomDev &g, const float *x, const float *y, const float *z,
                          const float *u, const float *v, const float *w, const float *q, long n,
                          float **acc, float *const mom[10], int *err, cudaStream_t s) {
  if (n <= 0) return SPB_OK;
  long done = 0;   // particles deposited in cell order
  if (n >= P2S_MIN)
    if (int rc = sorted_p2g(g, x, y, z, u, v, w, q, n, mom, err, s, &done)) return rc;
  if (done == n) return SPB_OK;
  if (!*acc) *acc = plain_acc_alloc(g, s);
  const DepTarget T = target(*acc, mom);
  const unsigned chunks = (unsigned)ceil_div(n - done, GP_CHUNK);
  auto *const kernel = *acc ? k_plain_p2g_grouped<true> : k_plain_p2g_grouped<false>;
  kernel<<<chunks, GP_TPB, 0, s>>>(g, x + done, y + done, z + done, u + done, v + done, w + done,
                                   q + done, n - done, T, err);
  SPB_CUDA(cudaGetLastError());
  g_launches++;
  return SPB_OK;
}

namespace {
// Whether mover_interp moves and deposits in one pass: below the sorted
// deposit's threshold, where the grouped deposit takes 105 us however few the
// particles (mover_interp of 30,000 on 64x32x32 cells: 53 us, in two passes
// 115), and for fewer than half a particle per node, where the sorted deposit's
// passes over the cells are its time (cell order, one pass and two: 128x64x64
// cells, 200,000 particles 96 and 109 us, 600,000 152 and 134; 256x256x256,
// 4M 1221 and 2000, 8M 1770 and 2313, 16M 2954 and 2835).
bool fused_interp(const GeomDev &g, long n) {
  return n < P2S_MIN || 2 * n < (long)g.nxn * g.nyn * g.nzn;
}
}  // namespace

int launch_plain_mover_interp_into(const GeomDev &g, const PushDev &p, const PackedFields &F,
                                   float *x, float *y, float *z, float *u, float *v, float *w,
                                   const float *q, long n, float **acc, float *const mom[10],
                                   int *err, cudaStream_t s) {
  if (n > 0 && fused_interp(g, n)) {
    if (!*acc) *acc = plain_acc_alloc(g, s);
    auto pick = [&](auto with_acc) {
      constexpr bool A = decltype(with_acc)::value;
      if (!g.float_cells) return k_plain_mover_interp<A, false, 0>;
      return p.niter == 3 ? k_plain_mover_interp<A, true, 3> : k_plain_mover_interp<A, true, 0>;
    };
    auto *const kernel = *acc ? pick(std::true_type()) : pick(std::false_type());
    kernel<<<blocks_for(n), TPB, 0, s>>>(g, p, F, x, y, z, u, v, w, q, n, target(*acc, mom), err);
    SPB_CUDA(cudaGetLastError());
    g_launches++;
    return SPB_OK;
  }
  if (int rc = launch_plain_mover(g, p, F, x, y, z, u, v, w, n, err, s)) return rc;
  return launch_plain_p2g_into(g, x, y, z, u, v, w, q, n, acc, mom, err, s);
}

int launch_plain_p2g(const GeomDev &g, const float *x, const float *y, const float *z,
                     const float *u, const float *v, const float *w, const float *q, long n,
                     float *const mom[10], int *err, cudaStream_t s) {
  if (n <= 0) return SPB_OK;
  float *acc = nullptr;
  const int rc = launch_plain_p2g_into(g, x, y, z, u, v, w, q, n, &acc, mom, err, s);
  if (rc) {
    if (acc) cudaFreeAsync(acc, s);
    return rc;
  }
  return plain_acc_fold(acc, g, mom, s);
}

int launch_plain_mover_interp(const GeomDev &g, const PushDev &p, const PackedFields &F,
                              float *x, float *y, float *z, float *u, float *v, float *w,
                              const float *q, long n, float *const mom[10], int *err,
                              cudaStream_t s) {
  float *acc = nullptr;
  const int rc =
      launch_plain_mover_interp_into(g, p, F, x, y, z, u, v, w, q, n, &acc, mom, err, s);
  if (rc) {
    if (acc) cudaFreeAsync(acc, s);
    return rc;
  }
  return plain_acc_fold(acc, g, mom, s);
}

int launch_apply_bc_ids(int nxn, int nyn, int nzn, const int periodic[3],
                        float *const mom[10], cudaStream_t s, long *launches) {
  Moments10 M;
  for (int m = 0; m < 10; ++m) M.m[m] = mom[m];
  const FoldGroups g = fold_groups(nxn, nyn, nzn, periodic);
  k_bc_fold<<<dim3(blocks_for(g.fx + g.fy + g.fz), 10), TPB, 0, s>>>(M, g);
  SPB_CUDA(cudaGetLastError());
  g_launches++;
  if (launches) ++*launches;
  return SPB_OK;
}

}  // namespace spb

extern "C" int spb_set_plain_deposit_mode(int mode) {
  if (mode != SPB_DEPOSIT_ACCUMULATOR && mode != SPB_DEPOSIT_DIRECT)
    return spb::fail(SPB_ERR_INVALID, "spb_set_plain_deposit_mode: unknown mode");
  return spb::g_deposit_mode.exchange(mode);
}
