// Pieces of the one-thread-per-cell deposit, shared by the plain form's sorted
// deposit and the precision form's: 32-byte particle records walked cell by
// cell, 80 FP32 sums per cell in registers, the nodes' sums over their cells
// in shared memory.
#pragma once

#include "warp_sum.cuh"

namespace spb {

// Read-only 32-byte load of one particle record (one 256-bit access) that asks
// L2 to fetch the surrounding 256 bytes: a lane walking its cell's bucket then
// finds the next records in L2.
__device__ __forceinline__ void ld_rec(const float4 *p, float4 &a, float4 &b) {
  asm("ld.global.nc.L2::256B.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
      : "l"(p));
}

// One 32-byte record store (one 256-bit access; p 32-byte aligned).
__device__ __forceinline__ void st_rec(float4 *p, float4 a, float4 b) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(a.x),
               "f"(a.y), "f"(a.z), "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
               : "memory");
}

// Deposit terms of one particle added to 40 packed accumulators:
// acc[node*5 + k] += W_node * (mf[k], mf[k+5]) with the moment factors
// mf = 1, u, v, w, uu | uv, uw, vv, vw, ww, i.e. the pairs (1,uv) (u,uw)
// (v,vv) (w,vw) (uu,ww), in the reference order rhon, Jx, Jy, Jz, pxx | pxy,
// pxz, pyy, pyz, pzz (src/Mover.cpp:466-570); node = a*4 + b*2 + c with
// a/b/c = 1 the upper node on that axis, XOR-permuted by bits 4/3/2 of
// `perm` (the lane for warp_sum80, 0 for the plain order). q is folded into
// the x weights; q = 0 adds nothing.
// lox/ox, ...: the weights of the lower and the upper node of each axis.
__device__ __forceinline__ void add_terms(float2 (&acc)[40], float q, float lox, float ox,
                                          float loy, float oy, float loz, float oz, float u,
                                          float v, float w, int perm) {
  const bool px = perm & 16, py = perm & 8, pz = perm & 4;
  const float wx0 = q * (px ? ox : lox), wx1 = q * (px ? lox : ox);
  const float wy0 = py ? oy : loy, wy1 = py ? loy : oy;
  const float wz0 = pz ? oz : loz, wz1 = pz ? loz : oz;
  const float2 mf[5] = {make_float2(1.0f, u * v), make_float2(u, u * w), make_float2(v, v * v),
                        make_float2(w, v * w), make_float2(u * u, w * w)};
  const float wxy[4] = {wx0 * wy0, wx0 * wy1, wx1 * wy0, wx1 * wy1};
#pragma unroll
  for (int ab = 0; ab < 4; ++ab) {
    const float W0 = wxy[ab] * wz0, W1 = wxy[ab] * wz1;
    const float2 W02 = make_float2(W0, W0), W12 = make_float2(W1, W1);
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      acc[(ab * 2 + 0) * 5 + k] = __ffma2_rn(W02, mf[k], acc[(ab * 2 + 0) * 5 + k]);
      acc[(ab * 2 + 1) * 5 + k] = __ffma2_rn(W12, mf[k], acc[(ab * 2 + 1) * 5 + k]);
    }
  }
}

// Per-warp quota of the deposit (all 32 lanes call with their cell's count):
// lanes sum at most Q particles of their own cell, one particle per lane per
// step; the excess of the cells above Q is summed by the whole warp, 32
// particles per step plus one warp reduction per cell. Q minimises the
// estimated issue slots, 60 per lane step and 65 per warp step + 160 per
// excess cell; a warp whose largest count is at most 1.25 x its mean keeps Q =
// its largest count. Counts within 64 of each other: over up to eight values
// between the mean and the largest, two ballots each; else over all the lanes'
// counts, one shuffle each (32 in a row: k_deposit of the GEM grid, 4 species,
// took 310 us with them and 304 us with the ballots at 8 particles per cell,
// 608 and 597 us at 27, 1975 and 1965 us at 125).
__device__ __forceinline__ int deposit_quota(int cnt) {
  const int mx = __reduce_max_sync(0xffffffffu, cnt);
  if (mx > (1 << 24)) return mx;   // keeps the cost sums below 2^32
  const int sum = __reduce_add_sync(0xffffffffu, cnt);
  if ((long long)mx * 32 * 4 <= (long long)sum * 5) return mx;   // max <= 1.25 x mean
  const int mean = sum >> 5;
  if (mx - mean <= 64) {
    const int step = (mx - mean + 7) >> 3;
    int best = mx;
    unsigned least = 60u * (unsigned)mx;
#pragma unroll
    for (int i = 1; i <= 8; ++i) {
      const int q = max(mx - i * step, mean);
      const unsigned over = __popc(__ballot_sync(0xffffffffu, cnt > q));
      const unsigned twice = __popc(__ballot_sync(0xffffffffu, cnt > q + 32));
      const unsigned c = 60u * (unsigned)q + 225u * over + 65u * twice;
      if (c < least) {
        least = c;
        best = q;
      }
    }
    return best;
  }
  unsigned cost = 60u * (unsigned)cnt;
#pragma unroll 4
  for (int i = 0; i < 32; ++i) {
    const int c = __shfl_sync(0xffffffffu, cnt, i);
    if (c > cnt) cost += 65u * (unsigned)((c - cnt + 31) >> 5) + 160u;
  }
  const unsigned lane = threadIdx.x & 31;
  const unsigned best = __reduce_min_sync(0xffffffffu, (min(cost, (1u << 26) - 1) << 5) | lane);
  return __shfl_sync(0xffffffffu, cnt, (int)(best & 31u));
}

// A tile's per-cell totals in shared memory: pairs (moment k, moment k + 5) of
// every corner of every cell, sCell[(corner * 5 + k) * TC + cell].
template <typename T>
struct PairOf;
template <>
struct PairOf<float> {
  using type = float2;
};
template <>
struct PairOf<double> {
  using type = double2;
};
__device__ __forceinline__ float2 add_pair(float2 a, float2 b) { return __fadd2_rn(a, b); }
template <typename T2>
__device__ __forceinline__ double2 add_pair(double2 a, T2 b) {
  return make_double2(a.x + (double)b.x, a.y + (double)b.y);
}

// Each node's sum of the totals of its (up to 8) cells in the tile, handed to
// emit(bx, by, bz, sum[5]) (sum[k]: moments k and k + 5, summed in A; the node's
// position counted from the tile's lower corner). All threads of the CTA call, after a
// barrier behind the totals' stores. A thread takes a node and its ten
// moments: the node's position and which of its cells lie in the tile are
// formed once, the cells' pairs lie at fixed offsets from one address, and one
// load and one packed add take two moments. (A thread per node and moment
// spent most of its instructions on those addresses; the precision form's
// deposit of the GEM grid, 4 species: 396 -> 323 us at 8 particles per cell,
// 697 -> 636 us at 27, 2100 -> 2050 us at 125.)
template <int TX, int TY, int TZ, int NT, typename T, typename A, typename Emit>
__device__ __forceinline__ void node_sums(const typename PairOf<T>::type *sCell, Emit emit) {
  using T2 = typename PairOf<T>::type;
  using A2 = typename PairOf<A>::type;
  constexpr int NX = TX + 1, NY = TY + 1, NZ = TZ + 1, NB = NX * NY * NZ;
  constexpr int TC = TX * TY * TZ;
  for (int nb = threadIdx.x; nb < NB; nb += NT) {
    const int bz = nb % NZ, by = (nb / NZ) % NY, bx = nb / (NZ * NY);
    // the cell above the node on an axis (corner bit 0) or the one below it (1)
    const bool inx[2] = {bx < TX, bx > 0}, iny[2] = {by < TY, by > 0}, inz[2] = {bz < TZ, bz > 0};
    const T2 *at = sCell + (bx * TY + by) * TZ + bz;
    A2 sum[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) sum[k].x = sum[k].y = (A)0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int a = e >> 2, b = (e >> 1) & 1, c = e & 1;
      if (inx[a] && iny[b] && inz[c]) {
#pragma unroll
        for (int k = 0; k < 5; ++k)
          sum[k] = add_pair(sum[k], at[(e * 5 + k) * TC - ((a * TY + b) * TZ + c)]);
      }
    }
    emit(bx, by, bz, sum);
  }
}

}  // namespace spb
