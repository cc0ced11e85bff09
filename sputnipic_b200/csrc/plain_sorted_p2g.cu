// The plain deposit (interpP2G, src/Mover.cpp:385-572) in cell order: the
// particles are copied into 32-byte records grouped by deposit cell, and one
// thread per cell sums its records in registers.
//
// Four launches per chunk of particles: count the particles of every cell;
// give every cell its range of the record array (a scan inside each CTA, one
// atomic per CTA for its place: the cells' ranges need not be in order); copy
// every particle into its cell's range; sum. Records (x, y, z, q, u, v, w, -)
// are written and read whole, one 32-byte sector each, so a particle costs the
// same traffic however far the arrays have drifted from cell order: 12 B read
// to count it, 28 B read and 32 B written to copy it, 32 B read to sum it.
//
// The permutation this replaces (8 B of sort scratch per particle) left the
// deposit 4-byte gathers through it, 4.5 L2 sectors per particle in arrays
// near cell order and up to 7 in others, and a warp reduction per run of a
// cell's particles. 65.5M particles in cell order, 125 per cell, zeroing and
// applyBCids included: 2352 -> 1455 us (count 150, copy 680, sum 600); two
// species of 2.4M some cycles after the last sort, 27 per cell: 432 -> 232 us.
//
// Cells are numbered tile by tile (8 x 4 x 4 cells; a CTA of the last launch
// takes a tile), over the nxn - 1 cells per axis that node pairs (i - 1, i)
// span, guard cells included. The first inner cell starts a tile, so that on a
// grid of whole tiles the guard cells, empty but for particles on a wall, fill
// tiles of their own, which end at once (the GEM grid: 4096 tiles of full cells
// instead of 4913 of which 817 held one layer).
#include "cell_deposit.cuh"
#include "grid_ctx.h"
#include "kernels.h"
#include "plain_cells.cuh"
#include "sim_kernels.cuh"

#include <algorithm>

namespace spb {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int TX = 8, TY = 4, TZ = 4, TC = TX * TY * TZ;
// Positions that cell 0, the lower guard cell, lies into its tile.
constexpr int SX = TX - 1, SY = TY - 1, SZ = TZ - 1;
constexpr int TPB = 256;
// Particles per chunk: bounds the scratch at 2.1 GB of records.
constexpr long CHUNK_MAX = 1L << 26;

struct Moments10 {
  float *m[10];
};

struct Particles7 {
  const float *p[7];   // x, y, z, u, v, w, q
};

// The deposit cell of a particle, as a key.
template <bool FLOAT_CELLS>
__device__ __forceinline__ int cell_key(const GeomDev &g, int nty, int ntz, float x, float y,
                                        float z, int &bad) {
  int ix, iy, iz;
  deposit_cell<FLOAT_CELLS>(g, x, y, z, ix, iy, iz, bad);
  return tile_key<TX, TY, TZ>(ix - 1 + SX, iy - 1 + SY, iz - 1 + SZ, nty, ntz);
}

// Particles per cell (one atomic per distinct cell of a warp).
template <bool FLOAT_CELLS>
__global__ void __launch_bounds__(TPB) k_p2g_count(GeomDev g, int nty, int ntz,
                                                   const float *__restrict__ x,
                                                   const float *__restrict__ y,
                                                   const float *__restrict__ z, long n,
                                                   unsigned *__restrict__ count) {
  const int lane = threadIdx.x & 31;
  int ignored = 0;   // the copy flags cells off the node array
  constexpr int U = 4;   // particles whose loads are in flight per thread
  for (long base = (long)blockIdx.x * (TPB * U); base < n; base += (long)gridDim.x * (TPB * U)) {
    float p[U][3];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const long i = min(base + k * TPB + threadIdx.x, n - 1);
      p[k][0] = x[i];
      p[k][1] = y[i];
      p[k][2] = z[i];
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const bool valid = base + k * TPB + threadIdx.x < n;
      const int key =
          valid ? cell_key<FLOAT_CELLS>(g, nty, ntz, p[k][0], p[k][1], p[k][2], ignored) : -1;
      const unsigned peers = __match_any_sync(FULL, key);
      if (valid && lane == __ffs(peers) - 1) atomicAdd(count + key, (unsigned)__popc(peers));
    }
  }
}

// Every cell's first record: an exclusive scan of the counts inside a CTA, at
// the place in the record array that the CTA takes for its cells.
constexpr int BASES_TPB = 1024;
__global__ void __launch_bounds__(BASES_TPB) k_p2g_bases(const unsigned *__restrict__ count,
                                                         long keys, unsigned *__restrict__ first,
                                                         unsigned *__restrict__ taken) {
  __shared__ unsigned ws[32];
  __shared__ unsigned place;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long i = blockIdx.x * (long)BASES_TPB + threadIdx.x;
  const unsigned v = i < keys ? count[i] : 0u;
  unsigned xs = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned t = __shfl_up_sync(FULL, xs, o);
    if (lane >= o) xs += t;
  }
  if (lane == 31) ws[warp] = xs;
  __syncthreads();
  if (warp == 0) {
    unsigned s = ws[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned t = __shfl_up_sync(FULL, s, o);
      if (lane >= o) s += t;
    }
    ws[lane] = s;
    if (lane == 31) place = s ? atomicAdd(taken, s) : 0u;
  }
  __syncthreads();
  if (i < keys) first[i] = place + (warp ? ws[warp - 1] : 0u) + xs - v;
}

// Every particle into its cell's next free record (next: the cells' first
// records, advanced to their ends; the order inside a cell is the atomics').
template <bool FLOAT_CELLS>
__global__ void __launch_bounds__(TPB) k_p2g_records(GeomDev g, int nty, int ntz,
                                                     const __grid_constant__ Particles7 P, long n,
                                                     unsigned *__restrict__ next,
                                                     float4 *__restrict__ rec,
                                                     int *__restrict__ err) {
  const int lane = threadIdx.x & 31;
  int bad = 0;
  for (long base = (long)blockIdx.x * TPB; base < n; base += (long)gridDim.x * TPB) {
    const bool valid = base + threadIdx.x < n;
    const long i = valid ? base + threadIdx.x : n - 1;   // every lane loads: no branch
    const float4 a = make_float4(P.p[0][i], P.p[1][i], P.p[2][i], P.p[6][i]);
    const float4 b = make_float4(P.p[3][i], P.p[4][i], P.p[5][i], 0.f);
    const int key = valid ? cell_key<FLOAT_CELLS>(g, nty, ntz, a.x, a.y, a.z, bad) : -1;
    const unsigned peers = __match_any_sync(FULL, key);
    const int leader = __ffs(peers) - 1;
    unsigned at = 0;
    if (valid && lane == leader) at = atomicAdd(next + key, (unsigned)__popc(peers));
    at = __shfl_sync(FULL, at, leader) + __popc(peers & ((1u << lane) - 1u));
    if (valid) st_rec(rec + 2 * (long)at, a, b);
  }
  if (bad) atomicOr(err, ERRBIT_OUT_OF_GRID);
}

// Particles that a lane sums before they are added to the cell's totals (by the
// warp, above the quota): sums of n terms one after another lose about n / 2
// rounding errors' variance, sums of runs of 16 of them 8 + n / 32, less than
// the warp's tree they replace.
constexpr int SUM_RUN = 16;

// One tile of cells (blockIdx.x) and one part of each cell's records
// (blockIdx.y): thread t sums the records of cell t, the warp those above its
// quota (deposit_quota), and every node of the tile adds its cells' sums into
// the moments. A term is f (q xi) eta (zeta invVOL),
// summed in FP32; the second invVOL multiplies a node's sum once (the reference
// multiplies every term by both): fewer roundings than its own. (q invVOL
// would round alike for all particles of equal charge: a bias, not noise.)
__global__ void __launch_bounds__(TC, 512 / TC) k_p2g_cells(GeomDev g, int nty, int ntz,
                                                            const unsigned *__restrict__ count,
                                                            const unsigned *__restrict__ end,
                                                            const float4 *__restrict__ recs,
                                                            const __grid_constant__ Moments10 M) {
  __shared__ float2 sCell[40 * TC];
  const int tid = threadIdx.x, lane = tid & 31;
  const long key = (long)blockIdx.x * TC + tid;
  // this CTA's part of the cell's records (gridDim.y parts)
  const unsigned all = count[key];
  const unsigned from = (unsigned)((unsigned long long)all * blockIdx.y / gridDim.y);
  const int cnt = (int)((unsigned)((unsigned long long)all * (blockIdx.y + 1) / gridDim.y) - from);
  if (!__syncthreads_or(cnt)) return;
  const float4 *rec = recs + 2 * ((long)end[key] - all + from);
  const int tz = blockIdx.x % ntz, ty = (blockIdx.x / ntz) % nty, tx = blockIdx.x / (ntz * nty);
  // the cell's lower nodes; cells of the tiles off the grid are empty
  const int cx = min(max(tx * TX + tid / (TY * TZ) - SX, 0), g.nxn - 2);
  const int cy = min(max(ty * TY + (tid / TZ) % TY - SY, 0), g.nyn - 2);
  const int cz = min(max(tz * TZ + tid % TZ - SZ, 0), g.nzn - 2);
  const float2 X = __ldg(g.xp + cx + 1), Y = __ldg(g.yp + cy + 1), Z = __ldg(g.zp + cz + 1);
  const float inv = g.invVOL;
  const int Q = deposit_quota(cnt);
  const int n1 = min(cnt, Q);
  const int trips = __reduce_max_sync(FULL, n1);
  float2 acc[40];
#pragma unroll
  for (int i = 0; i < 40; ++i) acc[i] = make_float2(0.f, 0.f);
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a, a1 = a, b1 = a;
  if (n1 > 0) ld_rec(rec, a, b);
  if (n1 > 1) ld_rec(rec + 2, a1, b1);
  // the cell's totals take the sums of SUM_RUN particles at a time
  auto put = [&](bool first) {
#pragma unroll
    for (int i = 0; i < 40; ++i) {
      sCell[i * TC + tid] = first ? acc[i] : __fadd2_rn(sCell[i * TC + tid], acc[i]);
      acc[i] = make_float2(0.f, 0.f);
    }
  };
#pragma unroll 1
  for (int k = 0; k < trips; ++k) {
    // two records in flight while this one is summed
    float4 na = a1, nb = b1;
    if (k + 2 < n1) ld_rec(rec + 2 * (k + 2), na, nb);
    // (after the load is on its way: before it, the totals' round through
    // shared memory kept the loads waiting, 55 us of 65.5M particles' 690)
    if (k && k % SUM_RUN == 0) put(k == SUM_RUN);
    // (lanes past their count add nothing: their last record with a charge of
    // zero would turn an infinite product of its velocities into NaN)
    if (k < n1)
      add_terms(acc, a.w, X.y - a.x, a.x - X.x, Y.y - a.y, a.y - Y.x, (Z.y - a.z) * inv,
                (a.z - Z.x) * inv, b.x, b.y, b.z, 0);
    a = a1;
    b = b1;
    a1 = na;
    b1 = nb;
  }
  put(trips <= SUM_RUN);
  unsigned heavy = __ballot_sync(FULL, cnt > Q);
  if (heavy) {
    __syncwarp();
    const int corner = (lane >> 2) & 7, half = (lane >> 1) & 1;
    const int lo = (lane & 1) ? 3 : 0, hi = (lane & 1) ? 5 : 3;
    while (heavy) {
      const int hl = __ffs(heavy) - 1;
      heavy &= heavy - 1;
      const int hc = __shfl_sync(FULL, cnt, hl);
      const float4 *hrec = reinterpret_cast<const float4 *>(
          __shfl_sync(FULL, reinterpret_cast<unsigned long long>(rec), hl));
      const float2 hX = make_float2(__shfl_sync(FULL, X.x, hl), __shfl_sync(FULL, X.y, hl));
      const float2 hY = make_float2(__shfl_sync(FULL, Y.x, hl), __shfl_sync(FULL, Y.y, hl));
      const float2 hZ = make_float2(__shfl_sync(FULL, Z.x, hl), __shfl_sync(FULL, Z.y, hl));
      float2 *dst = sCell + corner * 5 * TC + (tid & ~31) + hl;
#pragma unroll 1
      for (int o = Q; o < hc;) {
#pragma unroll
        for (int i = 0; i < 40; ++i) acc[i] = make_float2(0.f, 0.f);
        const int stop = min(o + 32 * SUM_RUN, hc);
#pragma unroll 1
        for (; o < stop; o += 32) {
          const int i = o + lane;
          float4 ha = make_float4(0.f, 0.f, 0.f, 0.f), hb = ha;
          if (i < hc) ld_rec(hrec + 2 * (long)i, ha, hb);
          add_terms(acc, i < hc ? ha.w : 0.0f, hX.y - ha.x, ha.x - hX.x, hY.y - ha.y,
                    ha.y - hY.x, (hZ.y - ha.z) * inv, (ha.z - hZ.x) * inv, hb.x, hb.y, hb.z, lane);
        }
        float r[5];
        warp_sum80(acc, r, lane);
#pragma unroll
        for (int k = 0; k < 5; ++k)
          if (k >= lo && k < hi) (half ? dst[k * TC].y : dst[k * TC].x) += r[k];
      }
    }
  }
  __syncthreads();
  node_sums<TX, TY, TZ, TC, float, double>(sCell, [&](int bx, int by, int bz,
                                                      const double2(&sum)[5]) {
    const long n = ((long)(tx * TX + bx - SX) * g.nyn + (ty * TY + by - SY)) * g.nzn +
                   (tz * TZ + bz - SZ);
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      if (sum[k].x != 0.0) atomicAdd(M.m[k] + n, (float)(sum[k].x * (double)inv));
      if (sum[k].y != 0.0) atomicAdd(M.m[k + 5] + n, (float)(sum[k].y * (double)inv));
    }
  });
}

}  // namespace

int sorted_p2g(const GeomDev &g, const float *x, const float *y, const float *z, const float *u,
               const float *v, const float *w, const float *q, long n, float *const mom[10],
               int *err, cudaStream_t s, long *done) {
  *done = 0;
  const int ntx = (int)ceil_div(g.nxn - 1 + SX, TX), nty = (int)ceil_div(g.nyn - 1 + SY, TY),
            ntz = (int)ceil_div(g.nzn - 1 + SZ, TZ);
  const long tiles = (long)ntx * nty * ntz, keys = tiles * TC;
  if (keys >= (1L << 31)) return SPB_OK;   // cell keys are ints: not in cell order
  // records of a chunk, the cells' counts and a counter, the cells' places;
  // chunks are halved until their scratch can be had
  long chunk = ceil_div(n, ceil_div(n, CHUNK_MAX));
  unsigned char *scratch = nullptr;
  for (;; chunk = ceil_div(chunk, 2)) {
    scratch = static_cast<unsigned char *>(
        pool_alloc((size_t)chunk * 32 + (size_t)(2 * keys + 1) * sizeof(unsigned), s));
    if (scratch && (reinterpret_cast<uintptr_t>(scratch) & 31u)) {   // records are 32-byte accesses
      pool_free(scratch, s);
      scratch = nullptr;
    }
    if (scratch) break;
    if (chunk < 2 * SORTED_P2G_MIN) return SPB_OK;
  }
  float4 *rec = reinterpret_cast<float4 *>(scratch);
  unsigned *count = reinterpret_cast<unsigned *>(scratch + (size_t)chunk * 32);
  unsigned *taken = count + keys, *next = taken + 1;
  Moments10 M;
  for (int m = 0; m < 10; ++m) M.m[m] = mom[m];
  // on small grids the cells' records go to several CTAs: a thread walks its
  // cell's one after another, and with fewer tiles than CTAs fit (four per SM)
  // that walk is the launch's time; parts of at least eight records a cell
  // (32x16x16 cells at 27 per cell: 22 -> 13 us)
  const long inner = std::max(1L, ceil_div(g.nxn - 3, TX)) *
                     std::max(1L, ceil_div(g.nyn - 3, TY)) *
                     std::max(1L, ceil_div(g.nzn - 3, TZ));
  const unsigned parts = (unsigned)std::max(
      1L, std::min({4L, 4L * num_sms() / inner, chunk / (8 * inner * TC)}));
  int rc = SPB_OK;
  for (long off = 0; off < n && rc == SPB_OK; off += chunk) {
    const long c = std::min(chunk, n - off);
    const unsigned blocks = (unsigned)std::min<long>(ceil_div(c, TPB), 148L * 32);
    const Particles7 P{{x + off, y + off, z + off, u + off, v + off, w + off, q + off}};
    cudaError_t e = cudaMemsetAsync(count, 0, (size_t)(keys + 1) * sizeof(unsigned), s);
    if (e == cudaSuccess) {
      (g.float_cells ? k_p2g_count<true> : k_p2g_count<false>)<<<blocks, TPB, 0, s>>>(
          g, nty, ntz, P.p[0], P.p[1], P.p[2], c, count);
      k_p2g_bases<<<(unsigned)ceil_div(keys, BASES_TPB), BASES_TPB, 0, s>>>(count, keys, next,
                                                                            taken);
      (g.float_cells ? k_p2g_records<true> : k_p2g_records<false>)<<<blocks, TPB, 0, s>>>(
          g, nty, ntz, P, c, next, rec, err);
      k_p2g_cells<<<dim3((unsigned)tiles, parts), TC, 0, s>>>(g, nty, ntz, count, next, rec, M);
      e = cudaGetLastError();
    }
    if (e != cudaSuccess) rc = fail_cuda(e, "sorted_p2g");
    g_launches += 4;
  }
  pool_free(scratch, s);
  if (rc == SPB_OK) *done = n;
  return rc;
}

}  // namespace spb
