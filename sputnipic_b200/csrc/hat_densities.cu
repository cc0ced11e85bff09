// calculateHatDensities (src/MaxwellSolver.cpp:465-603) on the device: the
// implicit sources of the field solver, J hat on the nodes and rho hat on the
// cell centres, from the species moments, in the reference's arithmetic.
//
// Three launches for all species: the divergence of every species' pressure
// tensor on the inner cells (divSymmTensorN2C, src/Grid.cpp:322-396) scaled by
// -dt/2; one node pass that, species by species, interpolates the centres to
// the nodes (interpC2Ninterp, src/Grid.cpp:122-139), adds the species' J,
// rotates with its omega_c dt/2 and accumulates J hat in registers (the PIdot
// loop, MaxwellSolver.cpp:535-566); one cell pass for rho hat = rho_c - dt
// theta div(J hat) (divN2C, src/Grid.cpp:267-319). The guard cells that the
// reference fills in between (applyBCscalarDensC, src/BC.cpp:623-727, of the
// centre temporaries and of rho hat; applyBCscalarDensN, src/BC.cpp:11-121, of
// J hat) each take the value of one inner cell (guard_source), so they are
// read, or computed, where that cell is: no fill passes.
//
// In place. J hat may be written over J or B, and rho hat over rho_c. A guard
// entry's thread would then read an inner entry that its own thread may already
// have overwritten, so such a call computes the inner entries only, each from
// its own, and copies the guards afterwards (k_hat_guards).
//
// Arithmetic. This file is compiled with -fmad=false and follows the C
// promotions of the reference expressions: the stencils' .25 * (a - b) * inv
// terms and the .125 interpolation scale are double, rounded to the array
// type on assignment; PIdot's denominator is double, the rest of PIdot is in
// the array type. The float instantiation reproduces the reference's FP32
// build bit for bit, the double one its FP64 build.
//
#include <algorithm>
#include <cstring>

#include "../../include/sputnipic_ref_layout.h"
#include "common.h"
#include "grid_ctx.h"
#include "kernels.h"

namespace spb {
namespace {

struct HatGeom {
  int nxc, nyc, nzc;   // cells, guard cells included
  int nxn, nyn, nzn;   // nodes
  double inv[3];       // the grid's inverse spacings
  int per[3];          // periodic axes
};

__device__ __forceinline__ long nidx(const HatGeom &g, int i, int j, int k) {
  return ((long)i * g.nyn + j) * g.nzn + k;
}
__device__ __forceinline__ long cidx(const HatGeom &g, int i, int j, int k) {
  return ((long)i * g.nyc + j) * g.nzc + k;
}

// The four node differences across cell (i, j, k) along `axis`, each times
// .25 and the inverse spacing, summed in double in the reference's order:
// x runs over (j, k), y over (i, k), both with k fastest; z over (i, j) with
// i fastest.
template <typename T>
__device__ __forceinline__ double d4(const HatGeom &g, const T *__restrict__ a, int i, int j,
                                     int k, int axis) {
  double sum = 0.0;
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int hi = t >> 1, lo = t & 1;
    int i0 = i, j0 = j, k0 = k;
    if (axis == 0) {
      j0 += hi;
      k0 += lo;
    } else if (axis == 1) {
      i0 += hi;
      k0 += lo;
    } else {
      j0 += hi;
      i0 += lo;
    }
    const T a0 = a[nidx(g, i0, j0, k0)];
    const T a1 = a[nidx(g, i0 + (axis == 0), j0 + (axis == 1), k0 + (axis == 2))];
    const T diff = a1 - a0;
    const double term = 0.25 * (double)diff * g.inv[axis];
    sum = t ? sum + term : term;
  }
  return sum;
}

constexpr int HAT_MAXS = SPB_HAT_MAX_SPECIES;

// Every species' inputs: pressure tensors (pxx, pxy, pxz, pyy, pyz, pzz), J,
// the centre temporaries (three per species) and beta = qom dt / 2c.
template <typename T>
struct Species6 {
  const T *p[HAT_MAXS][6];
  const T *j[HAT_MAXS][3];
  T *tc[HAT_MAXS][3];
  T beta[HAT_MAXS];
};

// The nodes (i; j, j + 1; k, k + 1) of the six pressure components.
template <typename T>
struct Plane6 {
  T v[6][4];   // [component][2 (j + 1) + (k + 1)]
};

template <typename T>
__device__ __forceinline__ void load_plane(const HatGeom &g, const T *const (&p)[6], long at,
                                           Plane6<T> &P) {
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    P.v[c][0] = __ldg(p[c] + at);
    P.v[c][1] = __ldg(p[c] + at + 1);
    P.v[c][2] = __ldg(p[c] + at + g.nzn);
    P.v[c][3] = __ldg(p[c] + at + g.nzn + 1);
  }
}

// d4 of component c between the planes i (lo) and i + 1 (hi) along `axis`.
template <typename T>
__device__ __forceinline__ double d4_planes(const HatGeom &g, const Plane6<T> &lo,
                                            const Plane6<T> &hi, int c, int axis) {
  double sum = 0.0;
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int a = t >> 1, b = t & 1;   // d4's hi and lo
    T diff;
    if (axis == 0)
      diff = hi.v[c][2 * a + b] - lo.v[c][2 * a + b];
    else if (axis == 1)
      diff = (a ? hi : lo).v[c][2 + b] - (a ? hi : lo).v[c][b];
    else
      diff = (b ? hi : lo).v[c][2 * a + 1] - (b ? hi : lo).v[c][2 * a];
    const double term = 0.25 * (double)diff * g.inv[axis];
    sum = t ? sum + term : term;
  }
  return sum;
}

// Pressure-tensor rows (pxx pxy pxz / pxy pyy pyz / pxz pyz pzz): divergence
// of each row on the inner cells, times alfa = (T)(-dt/2); species blockIdx.y.
// A thread walks `run` cells along x and keeps the nodes of the last plane, so
// a cell costs 24 loads (four nodes of six components) instead of the 72 that
// its nine stencils read one by one: those kept the L1 pipe busy (an unaligned
// row of 32 doubles takes three passes). 128x64x64 cells, 4 species, FP64: 62 ->
// 46 us; with the guard fills gone the whole call 168 -> 106 us. Register caps
// for four (double) and five (float) CTAs per SM: float 83 -> 74 us.
template <typename T>
__global__ void __launch_bounds__(128, sizeof(T) == 8 ? 4 : 5) k_hat_div_tensor(HatGeom g, const __grid_constant__ Species6<T> S, T alfa, int run) {
  const int is = blockIdx.y;
  const int my = g.nyc - 2, mz = g.nzc - 2;
  const unsigned columns = (unsigned)(((long)my * mz + 127) / 128);   // CTAs per run
  const long t = (blockIdx.x % columns) * 128L + threadIdx.x;
  if (t >= (long)my * mz) return;
  const int k = 1 + (int)(t % mz), j = 1 + (int)(t / mz);
  const int first = 1 + (int)(blockIdx.x / columns) * run, last = min(first + run, g.nxc - 1);
  const T *const p[6] = {S.p[is][0], S.p[is][1], S.p[is][2], S.p[is][3], S.p[is][4], S.p[is][5]};
  const long plane = (long)g.nyn * g.nzn;
  long at = nidx(g, first, j, k), to = cidx(g, first, j, k);
  auto cell = [&](const Plane6<T> &lo, const Plane6<T> &hi) {
    // row r, column ax -> tensor component
    const int comp[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const T c0 = (T)d4_planes(g, lo, hi, comp[r][0], 0);
      const T c1 = (T)d4_planes(g, lo, hi, comp[r][1], 1);
      const T c2 = (T)d4_planes(g, lo, hi, comp[r][2], 2);
      const T div = c0 + c1 + c2;
      S.tc[is][r][to] = div * alfa;
    }
    to += (long)g.nyc * g.nzc;
  };
  Plane6<T> A, B;
  load_plane(g, p, at, A);
  for (int i = first; i < last; i += 2) {
    load_plane(g, p, at += plane, B);
    cell(A, B);
    if (i + 1 < last) {
      load_plane(g, p, at += plane, A);
      cell(B, A);
    }
  }
}

// The inner cell whose value a cell holds after the reference's guard-cell
// fill, per axis: x itself inside; on a periodic axis of n cells the guard at 0
// holds cell n - 1 - s and the one at n - 1 cell s (s = 1 for centres, 2 for
// nodes), on another axis the neighbouring cell. The reference fills in phases
// (periodic faces X, Y, Z; edges; corners; the other faces X, Y, Z), each of
// which copies cells by these rules axis by axis; the phases' combined effect
// on a guard cell of several axes is the axes' rules one by one.
__device__ __forceinline__ int guard_source(int x, int n, int s, int periodic) {
  const int e = n - 1;
  if (x == 0) return periodic ? e - s : 1;
  if (x == e) return periodic ? s : e - 1;
  return x;
}

template <typename T>
struct Vec3 {
  const T *v[3];
};
template <typename T>
struct Out3 {
  T *v[3];
};

// Every node: per species in order, the interpolated divergence plus J,
// rotated by the species' beta B and added into J hat, which starts at 0 (the
// reference's per-species accumulation, in registers). A guard node computes
// the node that its value comes from, and guard cells are read where theirs
// does; without `guards` a guard node is left alone. Four CTAs per SM (at most
// 64 registers), for the same reason.
template <typename T>
__global__ void __launch_bounds__(256, 4) k_hat_pidot(HatGeom g, const __grid_constant__ Species6<T> S, int ns, Vec3<T> B,
                            Out3<T> JH, bool guards) {
  const long nodes = (long)g.nxn * g.nyn * g.nzn;
  for (long n = blockIdx.x * (long)blockDim.x + threadIdx.x; n < nodes;
       n += (long)gridDim.x * blockDim.x) {
    const int i = guard_source((int)(n / ((long)g.nzn * g.nyn)), g.nxn, 2, g.per[0]);
    const int j = guard_source((int)((n / g.nzn) % g.nyn), g.nyn, 2, g.per[1]);
    const int k = guard_source((int)(n % g.nzn), g.nzn, 2, g.per[2]);
    const long m = nidx(g, i, j, k);
    if (!guards && m != n) continue;
    // the node's upper cell, and the steps to its lower ones per axis
    const int i0 = guard_source(i, g.nxc, 1, g.per[0]), j0 = guard_source(j, g.nyc, 1, g.per[1]),
              k0 = guard_source(k, g.nzc, 1, g.per[2]);
    const long c0 = cidx(g, i0, j0, k0);
    const long dx = (long)(guard_source(i - 1, g.nxc, 1, g.per[0]) - i0) * g.nyc * g.nzc;
    const int dy = (guard_source(j - 1, g.nyc, 1, g.per[1]) - j0) * g.nzc;
    const int dz = guard_source(k - 1, g.nzc, 1, g.per[2]) - k0;
    const T bx = B.v[0][m], by = B.v[1][m], bz = B.v[2][m];
    T jh[3] = {(T)0, (T)0, (T)0};
    for (int is = 0; is < ns; ++is) {
      T tn[3];
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const T *c = S.tc[is][r] + c0;
        T s8 = c[0] + c[dx];
        s8 = s8 + c[dy];
        s8 = s8 + c[dz];
        s8 = s8 + c[dx + dy];
        s8 = s8 + c[dx + dz];
        s8 = s8 + c[dy + dz];
        s8 = s8 + c[dx + dy + dz];
        tn[r] = (T)(0.125 * (double)s8) + S.j[is][r][m];
      }
      const T beta = S.beta[is];
      const T ox = beta * bx, oy = beta * by, oz = beta * bz;
      const T X = tn[0], Y = tn[1], Z = tn[2];
      const T edotb = X * ox + Y * oy + Z * oz;
      const T oxx = ox * ox, oyy = oy * oy, ozz = oz * oz;
      const T denom = (T)(1 / (1.0 + (double)oxx + (double)oyy + (double)ozz));
      jh[0] = jh[0] + (X + (Y * oz - Z * oy + edotb * ox)) * denom;
      jh[1] = jh[1] + (Y + (Z * ox - X * oz + edotb * oy)) * denom;
      jh[2] = jh[2] + (Z + (X * oy - Y * ox + edotb * oz)) * denom;
    }
    JH.v[0][n] = jh[0];
    JH.v[1][n] = jh[1];
    JH.v[2][n] = jh[2];
  }
}

// rho hat = rho_c - dt theta div(J hat) on every cell; a guard cell computes
// the cell that its value comes from, or nothing without `guards`.
template <typename T>
__global__ void k_hat_rho(HatGeom g, Vec3<T> JH, const T *rhoc, double dt_th, T *rhoh,
                          bool guards) {
  const long cells = (long)g.nxc * g.nyc * g.nzc;
  for (long c = blockIdx.x * (long)blockDim.x + threadIdx.x; c < cells;
       c += (long)gridDim.x * blockDim.x) {
    const int i = guard_source((int)(c / ((long)g.nzc * g.nyc)), g.nxc, 1, g.per[0]);
    const int j = guard_source((int)((c / g.nzc) % g.nyc), g.nyc, 1, g.per[1]);
    const int k = guard_source((int)(c % g.nzc), g.nzc, 1, g.per[2]);
    const long m = cidx(g, i, j, k);
    if (!guards && m != c) continue;
    const T cx = (T)d4(g, JH.v[0], i, j, k, 0);
    const T cy = (T)d4(g, JH.v[1], i, j, k, 1);
    const T cz = (T)d4(g, JH.v[2], i, j, k, 2);
    const T dv = cx + cy + cz;
    rhoh[c] = (T)((double)rhoc[m] - dt_th * (double)dv);
  }
}

// The guard entries of n0 x n1 x n2 arrays, each from the inner entry
// that its value comes from (blockIdx.y: the array).
template <typename T>
__global__ void k_hat_guards(int n0, int n1, int n2, int s, HatGeom g, Out3<T> A) {
  T *const a = A.v[blockIdx.y];
  const long n = (long)n0 * n1 * n2;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n;
       t += (long)gridDim.x * blockDim.x) {
    const long i = guard_source((int)(t / ((long)n2 * n1)), n0, s, g.per[0]);
    const int j = guard_source((int)((t / n2) % n1), n1, s, g.per[1]);
    const int k = guard_source((int)(t % n2), n2, s, g.per[2]);
    const long m = (i * n1 + j) * n2 + k;
    if (m != t) a[t] = a[m];
  }
}

// Whether the na entries at a and the nb at b share memory.
template <typename T>
bool share(const T *a, long na, const T *b, long nb) {
  const uintptr_t x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b);
  return x < y + nb * sizeof(T) && y < x + na * sizeof(T);
}

int blocks_for(long n, int tpb) {
  return (int)std::max<long>(1, std::min<long>((n + tpb - 1) / tpb, 16L * num_sms()));
}

template <typename T>
int hat_densities(const spb_hat_desc *d, const T *const *mom, const T *const B[3], const T *rhoc,
                  T *jxh, T *jyh, T *jzh, T *rhoh, cudaStream_t st) {
  if (!d || !mom || !B || !rhoc || !jxh || !jyh || !jzh || !rhoh)
    return fail(SPB_ERR_INVALID, "spb_hat_densities: null argument");
  if (d->ns < 1 || d->ns > SPB_HAT_MAX_SPECIES)
    return fail(SPB_ERR_INVALID, "spb_hat_densities: ns out of range");
  if (d->nxc < 3 || d->nyc < 3 || d->nzc < 3)
    return fail(SPB_ERR_INVALID, "spb_hat_densities: at least 3 cells per axis (guards included)");
  HatGeom g;
  g.nxc = d->nxc;
  g.nyc = d->nyc;
  g.nzc = d->nzc;
  g.nxn = d->nxc + 1;
  g.nyn = d->nyc + 1;
  g.nzn = d->nzc + 1;
  g.inv[0] = d->invdx;
  g.inv[1] = d->invdy;
  g.inv[2] = d->invdz;
  for (int a = 0; a < 3; ++a) g.per[a] = d->periodic[a] ? 1 : 0;
  const long cells = (long)g.nxc * g.nyc * g.nzc, nodes = (long)g.nxn * g.nyn * g.nzn;
  const int ns = d->ns;
  // three centre temporaries per species (their guard cells are never written)
  T *const tc = static_cast<T *>(pool_alloc(3 * ns * cells * sizeof(T), st));
  if (!tc) return fail(SPB_ERR_CUDA, "spb_hat_densities: scratch allocation failed");
  Species6<T> S;   // kernel parameters (copied at launch)
  std::memset(&S, 0, sizeof(S));
  for (int is = 0; is < ns; ++is) {
    const T *const *M = mom + 10 * is;
    for (int c = 0; c < 6; ++c) S.p[is][c] = M[4 + c];
    for (int r = 0; r < 3; ++r) {
      S.j[is][r] = M[1 + r];
      S.tc[is][r] = tc + (3 * is + r) * cells;
    }
    S.beta[is] = (T)(.5 * d->qom[is] * d->dt / d->c);
  }
  const T alfa = (T)(-d->dt / 2.0);
  const long inner = (long)(g.nxc - 2) * (g.nyc - 2) * (g.nzc - 2);
  int rc = SPB_OK;
  // cells per thread along x: eight, fewer where that would leave SMs without
  // a full set of threads
  const int run = (int)std::max(1L, std::min(8L, inner * ns / (512L * num_sms())));
  const dim3 grid((unsigned)(ceil_div((long)(g.nyc - 2) * (g.nzc - 2), 128) *
                             ceil_div(g.nxc - 2, run)), (unsigned)ns);
  k_hat_div_tensor<T><<<grid, 128, 0, st>>>(g, S, alfa, run);
  const Out3<T> JH{{jxh, jyh, jzh}};
  bool j_over = false;   // J hat over the inputs of its own pass
  for (int r = 0; r < 3; ++r) {
    for (int c = 0; c < 3; ++c) j_over |= share(JH.v[r], nodes, B[c], nodes);
    for (int is = 0; is < ns; ++is)
      for (int c = 0; c < 3; ++c) j_over |= share(JH.v[r], nodes, S.j[is][c], nodes);
  }
  const bool rho_over = share(rhoh, cells, rhoc, cells);
  k_hat_pidot<T><<<blocks_for(nodes, 256), 256, 0, st>>>(g, S, ns, Vec3<T>{{B[0], B[1], B[2]}},
                                                         JH, !j_over);
  if (j_over)
    k_hat_guards<T><<<dim3(blocks_for(nodes, 256), 3), 256, 0, st>>>(g.nxn, g.nyn, g.nzn, 2, g,
                                                                     JH);
  k_hat_rho<T><<<blocks_for(cells, 256), 256, 0, st>>>(g, Vec3<T>{{jxh, jyh, jzh}}, rhoc,
                                                       d->dt * d->th, rhoh, !rho_over);
  if (rho_over)
    k_hat_guards<T><<<blocks_for(cells, 256), 256, 0, st>>>(g.nxc, g.nyc, g.nzc, 1, g,
                                                            Out3<T>{{rhoh, nullptr, nullptr}});
  if (cudaGetLastError() != cudaSuccess) rc = fail(SPB_ERR_CUDA, "spb_hat_densities: launch");
  g_launches += 3 + j_over + rho_over;
  pool_free(tc, st);
  return rc;
}

spb_hat_desc desc_from(const struct grid *grd, const struct parameters *param) {
  spb_hat_desc d;
  std::memset(&d, 0, sizeof(d));
  d.nxc = grd->nxc;
  d.nyc = grd->nyc;
  d.nzc = grd->nzc;
  d.invdx = grd->invdx;
  d.invdy = grd->invdy;
  d.invdz = grd->invdz;
  d.periodic[0] = param->PERIODICX;
  d.periodic[1] = param->PERIODICY;
  d.periodic[2] = param->PERIODICZ;
  d.dt = param->dt;
  d.c = param->c;
  d.th = param->th;
  d.ns = param->ns;
  for (int is = 0; is < param->ns && is < SPB_HAT_MAX_SPECIES; ++is) d.qom[is] = param->qom[is];
  return d;
}

// The drop-in over host arrays: uploads what the computation reads, runs it
// on a library stream, downloads J hat and rho hat.
int hat_dropin(struct interpDens_aux *aux, struct interpDensNet *idn,
               struct interpDensSpecies *ids, struct EMfield *field, struct grid *grd,
               struct parameters *param) {
  if (!aux || !idn || !ids || !field || !grd || !param)
    return fail(SPB_ERR_INVALID, "calculateHatDensities: null argument");
  if (param->ns < 1 || param->ns > SPB_NS_MAX)
    return fail(SPB_ERR_INVALID, "calculateHatDensities: ns out of range");
  const spb_hat_desc d = desc_from(grd, param);
  const long cells = (long)grd->nxc * grd->nyc * grd->nzc;
  const long nodes = (long)grd->nxn * grd->nyn * grd->nzn;
  if (d.nxc < 3 || d.nyc < 3 || d.nzc < 3)
    return fail(SPB_ERR_INVALID, "calculateHatDensities: grid too small");
  typedef spb_FPinterp T;
  static_assert(sizeof(spb_FPinterp) == sizeof(spb_FPfield), "one array type");
  cudaStream_t st;
  SPB_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  // node arrays: 9 per species (Jx..pzz), 3 fields, 3 outputs; centre arrays: rhoc, rhoh
  const int nin = 9 * d.ns + 3;
  T *buf = nullptr;
  const size_t bytes = ((size_t)(nin + 3) * nodes + 2 * (size_t)cells) * sizeof(T);
  int rc = SPB_OK;
  if (!(buf = static_cast<T *>(pool_alloc(bytes, st)))) {
    cudaStreamDestroy(st);
    return fail(SPB_ERR_ALLOC, "calculateHatDensities: device allocation failed");
  }
  const T *mom[10 * SPB_NS_MAX];
  T *p = buf;
  for (int is = 0; is < d.ns && rc == SPB_OK; ++is) {
    const struct interpDensSpecies &s = ids[is];
    const T *src[9] = {s.Jx_flat, s.Jy_flat, s.Jz_flat, s.pxx_flat, s.pxy_flat,
                       s.pxz_flat, s.pyy_flat, s.pyz_flat, s.pzz_flat};
    mom[10 * is] = nullptr;   // rhon: not read
    for (int m = 0; m < 9; ++m, p += nodes) {
      if (cudaMemcpyAsync(p, src[m], nodes * sizeof(T), cudaMemcpyHostToDevice, st) != cudaSuccess)
        rc = fail(SPB_ERR_CUDA, "calculateHatDensities: upload");
      mom[10 * is + 1 + m] = p;
    }
  }
  const T *fsrc[3] = {field->Bxn_flat, field->Byn_flat, field->Bzn_flat};
  const T *Bd[3];
  for (int a = 0; a < 3 && rc == SPB_OK; ++a, p += nodes) {
    if (cudaMemcpyAsync(p, fsrc[a], nodes * sizeof(T), cudaMemcpyHostToDevice, st) != cudaSuccess)
      rc = fail(SPB_ERR_CUDA, "calculateHatDensities: upload");
    Bd[a] = p;
  }
  T *jh[3] = {p, p + nodes, p + 2 * nodes};
  p += 3 * nodes;
  T *rhoc = p, *rhoh = p + cells;
  if (rc == SPB_OK &&
      cudaMemcpyAsync(rhoc, idn->rhoc_flat, cells * sizeof(T), cudaMemcpyHostToDevice, st) !=
          cudaSuccess)
    rc = fail(SPB_ERR_CUDA, "calculateHatDensities: upload");
  if (rc == SPB_OK) rc = hat_densities<T>(&d, mom, Bd, rhoc, jh[0], jh[1], jh[2], rhoh, st);
  T *dst[4] = {&aux->Jxh[0][0][0], &aux->Jyh[0][0][0], &aux->Jzh[0][0][0], &aux->rhoh[0][0][0]};
  const T *srcd[4] = {jh[0], jh[1], jh[2], rhoh};
  const long cnt[4] = {nodes, nodes, nodes, cells};
  for (int a = 0; a < 4 && rc == SPB_OK; ++a)
    if (cudaMemcpyAsync(dst[a], srcd[a], cnt[a] * sizeof(T), cudaMemcpyDeviceToHost, st) !=
        cudaSuccess)
      rc = fail(SPB_ERR_CUDA, "calculateHatDensities: download");
  pool_free(buf, st);
  if (cudaStreamSynchronize(st) != cudaSuccess && rc == SPB_OK)
    rc = fail(SPB_ERR_CUDA, "calculateHatDensities: stream");
  cudaStreamDestroy(st);
  return rc;
}

}  // namespace
}  // namespace spb

extern "C" int spb_hat_densities_f32(const spb_hat_desc *d, const float *const *mom,
                                     const float *const B[3], const float *rhoc, float *jxh,
                                     float *jyh, float *jzh, float *rhoh, void *stream) {
  return spb::hat_densities<float>(d, mom, B, rhoc, jxh, jyh, jzh, rhoh, (cudaStream_t)stream);
}

extern "C" int spb_hat_densities_f64(const spb_hat_desc *d, const double *const *mom,
                                     const double *const B[3], const double *rhoc, double *jxh,
                                     double *jyh, double *jzh, double *rhoh, void *stream) {
  return spb::hat_densities<double>(d, mom, B, rhoc, jxh, jyh, jzh, rhoh, (cudaStream_t)stream);
}

extern "C" int spb_calculateHatDensities(struct interpDens_aux *id_aux, struct interpDensNet *idn,
                                         struct interpDensSpecies *ids, struct EMfield *field,
                                         struct grid *grd, struct parameters *param) {
  return spb::hat_dropin(id_aux, idn, ids, field, grd, param);
}

void calculateHatDensities(struct interpDens_aux *id_aux, struct interpDensNet *idn,
                           struct interpDensSpecies *ids, struct EMfield *field, struct grid *grd,
                           struct parameters *param) {
  spb::hat_dropin(id_aux, idn, ids, field, grd, param);
}
