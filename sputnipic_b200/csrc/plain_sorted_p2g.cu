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
// applyBCids included: 2376 -> 1468 us (count 150, copy 680, sum 610); two
// species of 2.4M some cycles after the last sort, 27 per cell: 433 -> 231 us.
//
// Cells are numbered tile by tile (8 x 4 x 4 cells, on thin grids of one layer;
// a CTA of the last launch takes a tile), over the nxn - 1 cells per axis that
// node pairs (i - 1, i) span, guard cells included. The first inner cell starts a
// tile, so that on a grid of whole tiles the guard cells, empty but for particles
// on a wall, fill tiles of their own, which end at once (the GEM grid: 4096 tiles
// of full cells instead of 4913 of which 817 held one layer).
#include "cell_deposit.cuh"
#include "grid_ctx.h"
#include "kernels.h"
#include "plain_cells.cuh"
#include "sim_kernels.cuh"

#include <algorithm>

namespace spb {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int TC = 128;   // cells of a tile, TX x TY x TZ
constexpr int TPB = 256;
// Particles per chunk: bounds the scratch at 2.1 GB of records.
constexpr long CHUNK_MAX = 1L << 26;
// Records from which a cell may be summed apart from its tile.
constexpr int HEAVY_MIN = 1024;

struct Moments10 {
  float *m[10];
};

struct Particles7 {
  const float *p[7];   // x, y, z, u, v, w, q
};

// The deposit cell of a particle, as a key (cell 0 of an axis, the lower guard
// cell, is its tile's last).
template <int TX, int TY, int TZ, bool FLOAT_CELLS>
__device__ __forceinline__ int cell_key(const GeomDev &g, int nty, int ntz, float x, float y,
                                        float z, int &bad) {
  int ix, iy, iz;
  deposit_cell<FLOAT_CELLS>(g, x, y, z, ix, iy, iz, bad);
  return tile_key<TX, TY, TZ>(ix + TX - 2, iy + TY - 2, iz + TZ - 2, nty, ntz);
}

// Particles per cell (one atomic per distinct cell of a warp).
template <int TX, int TY, int TZ, bool FLOAT_CELLS>
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
          valid ? cell_key<TX, TY, TZ, FLOAT_CELLS>(g, nty, ntz, p[k][0], p[k][1], p[k][2], ignored)
                : -1;
      const unsigned peers = __match_any_sync(FULL, key);
      if (valid && lane == __ffs(peers) - 1) atomicAdd(count + key, (unsigned)__popc(peers));
    }
  }
}

// Cells with more than `above` records are summed by warps of their own, in
// segments of about `length` records (k_p2g_cells).
struct Heavy {
  unsigned above, length;
  int4 *segs;   // first record, records, cell key, -
};

// Every cell's first record: an exclusive scan of the counts inside a CTA, at
// the place in the record array that the CTA takes for its cells (taken[0]);
// and the heavy cells' segments (taken[1]: how many).
constexpr int BASES_TPB = 1024;
__global__ void __launch_bounds__(BASES_TPB) k_p2g_bases(const unsigned *__restrict__ count,
                                                         long keys, unsigned *__restrict__ first,
                                                         unsigned *__restrict__ taken, Heavy H) {
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
  const unsigned mine = place + (warp ? ws[warp - 1] : 0u) + xs - v;
  if (i < keys) first[i] = mine;
  if (v > H.above) {
    const unsigned k = (v + H.length - 1) / H.length, len = (v + k - 1) / k;
    const unsigned at = atomicAdd(taken + 1, k);
    for (unsigned j = 0, o = 0; j < k; ++j, o = min(o + len, v))
      H.segs[at + j] = make_int4((int)(mine + o), (int)min(len, v - o), (int)i, 0);
  }
}

// Every particle into its cell's next free record (next: the cells' first
// records, advanced to their ends; the order inside a cell is the atomics').
template <int TX, int TY, int TZ, bool FLOAT_CELLS>
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
    const int key =
        valid ? cell_key<TX, TY, TZ, FLOAT_CELLS>(g, nty, ntz, a.x, a.y, a.z, bad) : -1;
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
// Cells with particles up to which a tile skips the totals and the node sums
// (with no more than SUM_RUN records in any): its cells' sums go straight into
// the moments, at most 2,560 atomics where the node sums make up to 2,250.
// 256x256x256 cells, 1M particles (8 cells a tile) 0.89 ms, 1.63 with node sums;
// 4M (27 cells a tile) 1.5 and 1.8.
constexpr int SPARSE_CELLS = 32;

// The lower nodes' coordinates of a cell and their upper neighbours'.
struct CellNodes {
  float2 x, y, z;
};
__device__ __forceinline__ CellNodes cell_nodes(const GeomDev &g, int cx, int cy, int cz) {
  return {__ldg(g.xp + cx + 1), __ldg(g.yp + cy + 1), __ldg(g.zp + cz + 1)};
}

// Adds record (a, b) to acc (add_terms): a term is f (q xi) eta (zeta invVOL).
__device__ __forceinline__ void add_record(float2 (&acc)[40], const CellNodes &N, float inv,
                                           const float4 &a, const float4 &b, int perm) {
  add_terms(acc, a.w, N.x.y - a.x, a.x - N.x.x, N.y.y - a.y, a.y - N.y.x, (N.z.y - a.z) * inv,
            (a.z - N.z.x) * inv, b.x, b.y, b.z, perm);
}

// The heavy cells' segments, one per warp at a time: neighbouring lanes take
// neighbouring records, and every SUM_RUN of a lane's are summed over the warp
// into doubles (in shared memory, five per thread: the sums at hand fill the
// registers; a record loaded ahead spilled and gained nothing).
template <int TX, int TY, int TZ>
__device__ __forceinline__ void sum_segments(const GeomDev &g, int nty, int ntz, int cta, int ctas,
                                             const unsigned *__restrict__ nsegs,
                                             const int4 *__restrict__ segs,
                                             const float4 *__restrict__ recs,
                                             const Moments10 &M, double *sums) {
  const int lane = threadIdx.x & 31;
  const float inv = g.invVOL;
  const int n = (int)*nsegs;
  for (int s = cta * (TC / 32) + threadIdx.x / 32; s < n; s += ctas * (TC / 32)) {
    const int4 seg = segs[s];
    const int tile = seg.z / TC, c = seg.z % TC;
    const int cx = tile / (ntz * nty) * TX + c / (TY * TZ) - (TX - 1);
    const int cy = (tile / ntz) % nty * TY + (c / TZ) % TY - (TY - 1);
    const int cz = tile % ntz * TZ + c % TZ - (TZ - 1);
    const CellNodes N = cell_nodes(g, cx, cy, cz);
    const float4 *rec = recs + 2 * (long)seg.x;
    double *const sum = sums + threadIdx.x;
#pragma unroll
    for (int k = 0; k < 5; ++k) sum[k * TC] = 0.0;
#pragma unroll 1
    for (int o = 0; o < seg.y;) {
      float2 acc[40];
#pragma unroll
      for (int i = 0; i < 40; ++i) acc[i] = make_float2(0.f, 0.f);
      const int stop = min(o + 32 * SUM_RUN, seg.y);
#pragma unroll 1
      for (; o < stop; o += 32)
        if (o + lane < seg.y) {
          float4 a, b;
          ld_rec(rec + 2 * (o + lane), a, b);
          add_record(acc, N, inv, a, b, lane);
        }
      float r[5];
      warp_sum80(acc, r, lane);
#pragma unroll
      for (int k = 0; k < 5; ++k) sum[k * TC] += (double)r[k];
    }
    const int lo = (lane & 1) ? 3 : 0, hi = (lane & 1) ? 5 : 3, half = (lane >> 1) & 1;
    const long node = ((long)(cx + ((lane >> 4) & 1)) * g.nyn + (cy + ((lane >> 3) & 1))) * g.nzn +
                      (cz + ((lane >> 2) & 1));
#pragma unroll
    for (int k = 0; k < 5; ++k)
      if (k >= lo && k < hi)
        atomicAdd((half ? M.m[k + 5] : M.m[k]) + node, (float)(sum[k * TC] * (double)inv));
  }
}

// The cnt records of the lane's cell, straight into its nodes' moments.
__device__ __forceinline__ void add_cell(const GeomDev &g, const CellNodes &N, int cx, int cy,
                                         int cz, const float4 *rec, int cnt, const Moments10 &M) {
  const float inv = g.invVOL;
  float2 acc[40];
#pragma unroll
  for (int i = 0; i < 40; ++i) acc[i] = make_float2(0.f, 0.f);
#pragma unroll 1
  for (int k = 0; k < cnt; ++k) {
    float4 a, b;
    ld_rec(rec + 2 * k, a, b);
    add_record(acc, N, inv, a, b, 0);
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const long n =
        ((long)(cx + (e >> 2)) * g.nyn + (cy + ((e >> 1) & 1))) * g.nzn + (cz + (e & 1));
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      atomicAdd(M.m[k] + n, acc[e * 5 + k].x * inv);
      atomicAdd(M.m[k + 5] + n, acc[e * 5 + k].y * inv);
    }
  }
}

// The first CTAs take one tile of cells and one of `parts` parts of each cell's
// records, the last ones the heavy cells' segments (none on most input: they
// end as the last tiles are summed). Thread t sums the records of cell t, the
// warp those above its quota (deposit_quota), and every node of the tile adds
// its cells' sums into the moments. A term is f (q xi) eta (zeta invVOL), summed
// in FP32; the second invVOL multiplies a node's sum once (the reference
// multiplies every term by both): fewer roundings than its own. (q invVOL
// would round alike for all particles of equal charge: a bias, not noise.)
template <int TX, int TY, int TZ>
__global__ void __launch_bounds__(TC, 512 / TC) k_p2g_cells(GeomDev g, int nty, int ntz, int tiles,
                                                            int parts,
                                                            const unsigned *__restrict__ count,
                                                            const unsigned *__restrict__ end,
                                                            const unsigned *__restrict__ nsegs,
                                                            Heavy H,
                                                            const float4 *__restrict__ recs,
                                                            const __grid_constant__ Moments10 M) {
  __shared__ float2 sCell[40 * TC];
  const int tid = threadIdx.x, lane = tid & 31;
  if (blockIdx.x >= tiles * parts) {
    sum_segments<TX, TY, TZ>(g, nty, ntz, blockIdx.x - tiles * parts, gridDim.x - tiles * parts,
                             nsegs, H.segs, recs, M, reinterpret_cast<double *>(sCell));
    return;
  }
  const int part = parts > 1 ? blockIdx.x / tiles : 0, tile = blockIdx.x - part * tiles;
  const long key = (long)tile * TC + tid;
  // this CTA's part of the cell's records
  unsigned all = count[key], from = 0;
  if (all > H.above) all = 0;
  int cnt = (int)all;
  if (parts > 1) {
    from = (unsigned)((unsigned long long)all * part / parts);
    cnt = (int)((unsigned)((unsigned long long)all * (part + 1) / parts) - from);
  }
  const int busy = __syncthreads_count(cnt > 0);
  if (!busy) return;
  const unsigned rec = end[key] - all + from;   // its first record
  const int tz = tile % ntz, ty = (tile / ntz) % nty, tx = tile / (ntz * nty);
  // the cell's lower nodes; cells of the tiles off the grid are empty
  const int cx = min(max(tx * TX + tid / (TY * TZ) - (TX - 1), 0), g.nxn - 2);
  const int cy = min(max(ty * TY + (tid / TZ) % TY - (TY - 1), 0), g.nyn - 2);
  const int cz = min(max(tz * TZ + tid % TZ - (TZ - 1), 0), g.nzn - 2);
  const CellNodes N = cell_nodes(g, cx, cy, cz);
  const float inv = g.invVOL;
  if (busy <= SPARSE_CELLS && !__syncthreads_or(cnt > SUM_RUN)) {
    if (cnt) add_cell(g, N, cx, cy, cz, recs + 2 * (long)rec, cnt, M);
    return;
  }
  const int Q = deposit_quota(cnt);
  const int n1 = min(cnt, Q);
  const int trips = __reduce_max_sync(FULL, n1);
  float2 acc[40];
#pragma unroll
  for (int i = 0; i < 40; ++i) acc[i] = make_float2(0.f, 0.f);
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a, a1 = a, b1 = a;
  if (n1 > 0) ld_rec(recs + 2 * (long)rec, a, b);
  if (n1 > 1) ld_rec(recs + 2 * (long)(rec + 1), a1, b1);
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
    if (k + 2 < n1) ld_rec(recs + 2 * (long)(rec + k + 2), na, nb);
    // (after the load is on its way: before it, the totals' round through
    // shared memory kept the loads waiting, 55 us of 65.5M particles' 690)
    if (k && k % SUM_RUN == 0) put(k == SUM_RUN);
    // (lanes past their count add nothing: their last record with a charge of
    // zero would turn an infinite product of its velocities into NaN)
    if (k < n1) add_record(acc, N, inv, a, b, 0);
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
      const unsigned hrec = __shfl_sync(FULL, rec, hl);
      const auto from_hl = [&](float2 v) {
        return make_float2(__shfl_sync(FULL, v.x, hl), __shfl_sync(FULL, v.y, hl));
      };
      const CellNodes hN = {from_hl(N.x), from_hl(N.y), from_hl(N.z)};
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
          if (i < hc) ld_rec(recs + 2 * (long)(hrec + i), ha, hb);
          add_record(acc, hN, inv, ha, hb, lane);
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
    const long n = ((long)(tx * TX + bx - (TX - 1)) * g.nyn + (ty * TY + by - (TY - 1))) * g.nzn +
                   (tz * TZ + bz - (TZ - 1));
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      if (sum[k].x != 0.0) atomicAdd(M.m[k] + n, (float)(sum[k].x * (double)inv));
      if (sum[k].y != 0.0) atomicAdd(M.m[k + 5] + n, (float)(sum[k].y * (double)inv));
    }
  });
}

// Tiles of TX x TY x TZ cells that hold inner cells.
template <int TX, int TY, int TZ>
long inner_tiles(const GeomDev &g) {
  return std::max(1L, ceil_div(g.nxn - 3, TX)) * std::max(1L, ceil_div(g.nyn - 3, TY)) *
         std::max(1L, ceil_div(g.nzn - 3, TZ));
}

template <int TX, int TY, int TZ>
int sorted_p2g_by(const GeomDev &g, const float *x, const float *y, const float *z,
                  const float *u, const float *v, const float *w, const float *q, long n,
                  float *const mom[10], int *err, cudaStream_t s, long *done) {
  *done = 0;
  const int ntx = (int)ceil_div(g.nxn + TX - 2, TX), nty = (int)ceil_div(g.nyn + TY - 2, TY),
            ntz = (int)ceil_div(g.nzn + TZ - 2, TZ);
  const long tiles = (long)ntx * nty * ntz, keys = tiles * TC;
  if (keys >= (1L << 31)) return SPB_OK;   // cell keys are ints: not in cell order
  // records of a chunk, the heavy cells' segments (at most one per HEAVY_MIN
  // particles), the cells' counts and two counters, the cells' places; chunks
  // are halved until their scratch can be had
  long chunk = ceil_div(n, ceil_div(n, CHUNK_MAX));
  unsigned char *scratch = nullptr;
  for (;; chunk = ceil_div(chunk, 2)) {
    scratch = static_cast<unsigned char *>(
        pool_alloc((size_t)chunk * 32 + (size_t)(chunk / HEAVY_MIN + 1) * sizeof(int4) +
                       (size_t)(2 * keys + 2) * sizeof(unsigned),
                   s));
    if (scratch && (reinterpret_cast<uintptr_t>(scratch) & 31u)) {   // records are 32-byte accesses
      pool_free(scratch, s);
      scratch = nullptr;
    }
    if (scratch) break;
    if (chunk < 2 * SORTED_P2G_MIN) return SPB_OK;
  }
  float4 *rec = reinterpret_cast<float4 *>(scratch);
  int4 *segs = reinterpret_cast<int4 *>(scratch + (size_t)chunk * 32);
  unsigned *count = reinterpret_cast<unsigned *>(segs + chunk / HEAVY_MIN + 1);
  unsigned *taken = count + keys, *next = taken + 2;
  Moments10 M;
  for (int m = 0; m < 10; ++m) M.m[m] = mom[m];
  // on small grids the cells' records go to several CTAs: a thread walks its
  // cell's one after another, and with fewer tiles than CTAs fit (four per SM)
  // that walk is the launch's time; parts of at least eight records a cell
  // (32x16x16 cells at 27 per cell: 22 -> 13 us)
  const long inner = inner_tiles<TX, TY, TZ>(g);
  const int places = 4 * num_sms();
  const int parts = (int)std::max(1L, std::min(places / inner, chunk / (8 * inner * TC)));
  // heavy cells: more than eight times the mean of the inner tiles' cells, so
  // that none keeps its tile much longer than the others keep theirs; their
  // segments are as long as leaves every warp of the launch one. 4x4x4 cells with
  // 10M particles 0.63 ms, 23.8 with at most four parts; 128x64x64 cells with 20M
  // of which a third in one cell 1.04 ms, 121 if a warp walks that cell, all in
  // one cell 1.35 ms, 4.6 s
  const Heavy H{(unsigned)std::max<long>(HEAVY_MIN, chunk / (inner * (TC / 8))),
                (unsigned)std::max(2L * HEAVY_MIN, ceil_div(chunk, (long)places * (TC / 32))),
                segs};
  // a warp for every segment that there can be, no more CTAs than fit
  const int seg_ctas = (int)std::min<long>(places, ceil_div(chunk / HEAVY_MIN, TC / 32));
  int rc = SPB_OK;
  for (long off = 0; off < n && rc == SPB_OK; off += chunk) {
    const long c = std::min(chunk, n - off);
    const unsigned blocks = (unsigned)std::min<long>(ceil_div(c, TPB), 32L * num_sms());
    const Particles7 P{{x + off, y + off, z + off, u + off, v + off, w + off, q + off}};
    cudaError_t e = cudaMemsetAsync(count, 0, (size_t)(keys + 2) * sizeof(unsigned), s);
    if (e == cudaSuccess) {
      auto *const k_count = g.float_cells ? k_p2g_count<TX, TY, TZ, true>
                                          : k_p2g_count<TX, TY, TZ, false>;
      auto *const k_records = g.float_cells ? k_p2g_records<TX, TY, TZ, true>
                                            : k_p2g_records<TX, TY, TZ, false>;
      k_count<<<blocks, TPB, 0, s>>>(g, nty, ntz, P.p[0], P.p[1], P.p[2], c, count);
      k_p2g_bases<<<(unsigned)ceil_div(keys, BASES_TPB), BASES_TPB, 0, s>>>(count, keys, next,
                                                                            taken, H);
      k_records<<<blocks, TPB, 0, s>>>(g, nty, ntz, P, c, next, rec, err);
      k_p2g_cells<TX, TY, TZ><<<(unsigned)(tiles * parts + seg_ctas), TC, 0, s>>>(
          g, nty, ntz, (int)tiles, parts, count, next, taken + 1, H, rec, M);
      e = cudaGetLastError();
    }
    if (e != cudaSuccess) rc = fail_cuda(e, "sorted_p2g");
    g_launches += 4;
  }
  pool_free(scratch, s);
  if (rc == SPB_OK) *done = n;
  return rc;
}

}  // namespace

int sorted_p2g(const GeomDev &g, const float *x, const float *y, const float *z, const float *u,
               const float *v, const float *w, const float *q, long n, float *const mom[10],
               int *err, cudaStream_t s, long *done) {
  // on grids a few cells thin, tiles of one layer along that axis, where they
  // hold the cells in two thirds of the tiles or fewer (a layer's tile has 306
  // nodes to sum, not 225). 10M particles, 512x512x1 cells: 557 -> 321 us;
  // 1x512x512: 978 -> 316
  const auto pick = [&]() -> decltype(&sorted_p2g_by<8, 4, 4>) {
    const long most = 2 * inner_tiles<8, 4, 4>(g) / 3;
    if (inner_tiles<1, 16, 8>(g) <= most) return sorted_p2g_by<1, 16, 8>;
    if (inner_tiles<8, 1, 16>(g) <= most) return sorted_p2g_by<8, 1, 16>;
    if (inner_tiles<8, 16, 1>(g) <= most) return sorted_p2g_by<8, 16, 1>;
    return sorted_p2g_by<8, 4, 4>;
  };
  return pick()(g, x, y, z, u, v, w, q, n, mom, err, s, done);
}

}  // namespace spb
