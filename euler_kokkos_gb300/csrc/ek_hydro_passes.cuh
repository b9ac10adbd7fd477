// FP64 hydro step in passes, each over all its cells or faces.
//
// GB300 issues FP64 at 1/64 of the FP32 rate, so the FP64 step's time is its
// count of FP64 instructions: the passes' 807 B a cell and step (ncu, 96^3) are
// little beside it (1.5 Gcell/s x 807 B = 1.2 TB/s of 6.8).  A tile kernel
// repeats work (primitives of the halo 1.56 x, traces of the ring 1.25 x, the
// planes at a chunk's ends) and its phases wait for one another on few warps.
// Here every value is computed once, by one thread of a flat launch at full
// occupancy, and passed on through memory:
//   1. primitives of the cells and two ghost layers (boundary-mapped loads)
//   2. slopes, sources and the face states of each cell (ring cells: only the
//      state that faces the interior)
//   3. one Riemann problem per face
//   4. update, gravity, the next step's CFL
// along slabs of the last axis, so that the workspace stays bounded (a slab repeats
// the primitives of two layers on each side and the traces of one: 256 x 256 x 64
// 1.47 Gcell/s, 512 x 512 x 16, two slabs, 1.36, 1024 x 1024 x 12, a slab a plane,
// 0.81; the former tile kernel 0.69 to 0.72 on all).  The arithmetic is that of the
// tile kernels, function by function (the exact build stays bitwise equal to the
// reference).
#pragma once

#include "ek_hydro_kernels.cuh"
#include "ek_slabs.h"

namespace EK_NS
{

using ekc::HydroSlab;
constexpr int kPassThreads = 128;

__device__ __forceinline__ long long
pass_index()
{
  return (long long)blockIdx.x * kPassThreads + threadIdx.x;
}
// coordinates of cell c of a box with rows of nx and planes of ny rows
__device__ __forceinline__ void
box_coords(unsigned c, unsigned nx, unsigned ny, int & i, int & j, int & k)
{
  const unsigned r = c / nx;
  i = (int)(c - r * nx);
  k = (int)(r / ny);
  j = (int)(r - (unsigned)k * ny);
}

template <int NV>
__global__ void __launch_bounds__(kPassThreads)
hydro_prims_pass(const double * __restrict__ U, const KParams P, const DevClock * clk, int step, HydroSlab<NV> S)
{
  StepConsts sc;
  if (!step_consts(clk, step, sc))
    return;
  const long long c = pass_index(), n = S.box(4);
  if (c >= n)
    return;
  int i, j, k;
  box_coords((unsigned)c, S.nx + 4, S.ny + 4, i, j, k);
  const SrcCell s = src_cell(P, i, S.j0 + j, S.k0 + k);
  double        u[NV], q[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v)
    u[v] = neg_if(ldg(U + v * P.vstride + s.off), flips(s, v, 0));
  hydro_prims<double, NV>(u, q, hydro_const<double>(P));
#pragma unroll
  for (int v = 0; v < NV; ++v)
    S.q[v * n + c] = q[v];
  chain_next();
}

template <int NV, bool GRAV>
__global__ void __launch_bounds__(kPassThreads)
hydro_trace_pass(const KParams P, const DevClock * clk, int step, HydroSlab<NV> S)
{
  constexpr int DIM = HydroSlab<NV>::DIM;
  StepConsts    sc;
  if (!step_consts(clk, step, sc))
    return;
  const int       nx = S.nx, ny = S.ny, nz = DIM == 3 ? S.nz : 1;
  const long long cells = (long long)nx * ny * nz;
  // interior cells first, then the ring: low and high side of each axis
  long long c = pass_index();
  int       i, j, k, axis = -1;
  bool      high = false; // ring: the state on the high (true) or low face
  if (c < cells)
    box_coords((unsigned)c, nx, ny, i, j, k);
  else
  {
    c -= cells;
    const long long sx = (long long)ny * nz, sy = (long long)nx * nz, sz = (long long)nx * ny;
    if (c < 2 * sx)
    {
      axis = 0;
      high = c < sx;
      box_coords((unsigned)(high ? c : c - sx), 1, ny, i, j, k);
      i = high ? -1 : nx;
    }
    else if ((c -= 2 * sx) < 2 * sy)
    {
      axis = 1;
      high = c < sy;
      box_coords((unsigned)(high ? c : c - sy), nx, 1, i, j, k);
      j = high ? -1 : ny;
    }
    else if (DIM == 3 && (c -= 2 * sy) < 2 * sz)
    {
      axis = 2;
      high = c < sz;
      box_coords((unsigned)(high ? c : c - sz), nx, ny, i, j, k);
      k = high ? -1 : nz;
    }
    else
      return;
  }
  const HydroConst<double> C = hydro_const<double>(P);
  const double             dtd[3] = { sc.dtdx, sc.dtdy, sc.dtdz };
  const bool same_xy = sc.dtdx == sc.dtdy, same_all = same_xy && (DIM == 2 || sc.dtdx == sc.dtdz);
  const long long nq = S.box(4), ns = S.box(2);
  const int       qy = nx + 4, qz = qy * (ny + 4);
  const double *  q = S.q + ((DIM == 3 ? k + 2 : 0) * (long long)(ny + 4) + (j + 2)) * (nx + 4) + (i + 2);
  double          w[NV], d[3][NV], s[NV], f[NV], hg[3];
#pragma unroll
  for (int v = 0; v < NV; ++v)
  {
    const double * p = q + v * nq;
    const double   x = p[0];
    w[v] = x;
    d[0][v] = slope_h<double>(x, p[1], p[-1], C.slope_type);
    d[1][v] = slope_h<double>(x, p[qy], p[-qy], C.slope_type);
    d[2][v] = DIM == 3 ? slope_h<double>(x, p[qz], p[-qz], C.slope_type) : 0.0;
  }
  hydro_sources<double, NV>(w, d[0], d[1], d[2], s, C);
  const bool kick = GRAV && P.grav_hancock; // gravity predictor of the face states
  if (kick)
  {
    double g[3];
    grav_at<double, double, NV>(P, i + P.gw, S.j0 + j + P.gw, DIM == 3 ? S.k0 + k + P.gw : 0, g);
#pragma unroll
    for (int e = 0; e < 3; ++e)
      hg[e] = 0.5 * sc.dt * g[e];
  }
  double *   out = S.s + ((DIM == 3 ? k + 1 : 0) * (long long)(ny + 2) + (j + 1)) * (nx + 2) + (i + 1);
  FaceStates<double, NV> F(w, s, dtd[0], C.smallr);
#pragma unroll
  for (int a = 0; a < DIM; ++a)
  {
    if (a > 0)
      F.turn(dtd[a], a == 1 ? same_xy : same_all);
    if (axis >= 0 && axis != a)
      continue;
#pragma unroll
    for (int h = 0; h < 2; ++h)
    {
      if (axis >= 0 && (h == 1) != high)
        continue;
      F.get(d[a], h == 1, f);
      if (kick)
        grav_kick<double, NV>(f, hg);
#pragma unroll
      for (int v = 0; v < NV; ++v)
        out[((2 * a + h) * NV + v) * ns] = f[v];
    }
  }
  chain_next();
}

// faces of one axis, padded to whole blocks: (nx + 1) ny nz along x and so on
template <int NV>
__host__ __device__ inline long long
face_blocks(const HydroSlab<NV> & S, int axis)
{
  const long long nz = HydroSlab<NV>::DIM == 3 ? S.nz : 1;
  const long long n = (S.nx + (axis == 0)) * (long long)(S.ny + (axis == 1)) * (nz + (axis == 2));
  return (n + kPassThreads - 1) / kPassThreads;
}
template <int NV, int RS>
__global__ void __launch_bounds__(kPassThreads)
hydro_flux_pass(const KParams P, const DevClock * clk, int step, HydroSlab<NV> S)
{
  constexpr int DIM = HydroSlab<NV>::DIM;
  StepConsts    sc;
  if (!step_consts(clk, step, sc))
    return;
  // the block's axis, its thread's face
  int       axis = 0;
  long long b = blockIdx.x;
  while (axis < DIM - 1 && b >= face_blocks(S, axis))
    b -= face_blocks(S, axis++);
  const int       nx = S.nx, ny = S.ny, nz = DIM == 3 ? S.nz : 1;
  const int       ex = nx + (axis == 0), ey = ny + (axis == 1), ez = nz + (axis == 2);
  const long long c = b * kPassThreads + threadIdx.x;
  if (c >= (long long)ex * ey * ez)
    return;
  int i, j, k;
  box_coords((unsigned)c, ex, ey, i, j, k);
  const long long ns = S.box(2), nf = S.box(1);
  const long long r = ((DIM == 3 ? k + 1 : 0) * (long long)(ny + 2) + (j + 1)) * (nx + 2) + (i + 1); // the cell above
  const long long l = r - (axis == 0 ? 1 : (axis == 1 ? nx + 2 : (long long)(nx + 2) * (ny + 2)));
  const double *  lo = S.s + (2 * axis + 1) * NV * ns + l; // high state of the cell below
  const double *  hi = S.s + 2 * axis * NV * ns + r;       // low state of the cell above
  // face frame: the normal velocity in IU (the solver's other velocities keep
  // the places that the swap IU <-> IU + axis gives them)
  auto   var = [&](int v) { return v == IU ? IU + axis : (v == IU + axis ? (int)IU : v); };
  double ql[NV], qr[NV], fl[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v)
  {
    ql[v] = lo[var(v) * ns];
    qr[v] = hi[var(v) * ns];
  }
  hydro_riemann<RS, double, NV>(ql, qr, fl, hydro_const<double>(P));
  const double dtd = axis == 0 ? sc.dtdx : (axis == 1 ? sc.dtdy : sc.dtdz);
  double *     out = S.f + axis * NV * nf + ((DIM == 3 ? k : 0) * (long long)(ny + 1) + j) * (nx + 1) + i;
#pragma unroll
  for (int v = 0; v < NV; ++v)
    out[var(v) * nf] = flux_scaled(fl[v], dtd);
  chain_next();
}

template <int NV, bool GRAV>
__global__ void __launch_bounds__(kPassThreads)
hydro_update_pass(const double * __restrict__ Uin, double * __restrict__ Uout, const KParams P, DevClock * clk,
                  int step, HydroSlab<NV> S)
{
  constexpr int DIM = HydroSlab<NV>::DIM;
  StepConsts    sc;
  if (!step_consts(clk, step, sc))
    return;
  const HydroConst<double> C = hydro_const<double>(P);
  const int                nx = S.nx, ny = S.ny, nz = DIM == 3 ? S.nz : 1;
  const long long          c = pass_index(), nf = S.box(1);
  double                   tmax = -INFINITY;
  if (c < (long long)nx * ny * nz)
  {
    int i, j, k;
    box_coords((unsigned)c, nx, ny, i, j, k);
    const int       gi = i + P.gw, gj = S.j0 + j + P.gw, gk = DIM == 3 ? S.k0 + k + P.gw : 0;
    const long long off = (long long)gk * P.plane + (long long)gj * P.isize + gi;
    const double *  f = S.f + ((DIM == 3 ? k : 0) * (long long)(ny + 1) + j) * (nx + 1) + i;
    const long long next[3] = { 1, nx + 1, (long long)(nx + 1) * (ny + 1) };
    const double    dtd[3] = { sc.dtdx, sc.dtdy, sc.dtdz };
    double          u[NV], rho_old = 0.0;
    // UpdateFunctor2D/3D in their order (HydroRunFunctors2D.h:809-836, HydroRunFunctors3D.h:775-809)
#pragma unroll
    for (int v = 0; v < NV; ++v)
    {
      double x = ldg(Uin + v * P.vstride + off);
      if (v == ID)
        rho_old = x;
#pragma unroll
      for (int a = 0; a < DIM; ++a)
      {
        x = add_flux(x, f[(a * NV + v) * nf], dtd[a]);
        x = sub_flux(x, f[(a * NV + v) * nf + next[a]], dtd[a]);
      }
      u[v] = x;
    }
    double g[3];
    if constexpr (GRAV)
    {
      // gravity source term after the flux update (SolverHydroMuscl.cpp:245-252, 333-338)
      grav_at<double, double, NV>(P, gi, gj, gk, g);
      grav_source<double, NV>(u, rho_old, g, 0.5 * sc.dt, C);
    }
#pragma unroll
    for (int v = 0; v < NV; ++v)
      Uout[v * P.vstride + off] = u[v];
    if constexpr (GRAV)
      tmax = hydro_invdt_grav<double, NV>(u, g, C, P);
    else
      tmax = hydro_invdt<double, NV>(u, C, P);
  }
  chain_next();
  block_max_commit<kPassThreads>(cand_key(tmax), &clk->key[(step + 1) % 3]);
  if (!S.last)
    return;
  if (blockIdx.x == 0 && threadIdx.x == 0)
    step_commit(clk, step, sc.t, sc.dt);
  finalize_step(clk, P, step + 1); // the next step's dt, once its CFL key is complete
}

// Workspace of a slab (slab_cells): 2.6 million hydro 3D cells.  A single plane
// may take more, from 1024 x 1024 (1.3 GB) on.
constexpr long long kPassBytes = 1ll << 30;
template <int NV>
inline HydroSlab<NV>
hydro_slab(const KParams & P, int first, int n, void * work)
{
  HydroSlab<NV> S;
  S.nx = P.nx;
  S.ny = NV == 4 ? n : P.ny;
  S.nz = NV == 4 ? 1 : n;
  S.j0 = NV == 4 ? first : 0;
  S.k0 = NV == 4 ? 0 : first;
  S.last = first + n == (NV == 4 ? P.ny : P.nz);
  S.q = (double *)work;
  S.s = S.q + NV * S.box(4);
  S.f = S.s + 2 * HydroSlab<NV>::DIM * NV * S.box(2);
  return S;
}
template <int NV, int RS, bool GRAV>
cudaError_t
hydro_step_passes(const void * Uin, void * Uout, void * work, const KParams & P, DevClock * clk, int step,
                  cudaStream_t st)
{
  constexpr int DIM = HydroSlab<NV>::DIM;
  const double * in = (const double *)Uin;
  const int      N = NV == 4 ? P.ny : P.nz, n = P.slab;
  auto           blocks = [](long long items) { return (unsigned)((items + kPassThreads - 1) / kPassThreads); };
  for (int first = 0; first < N; first += n)
  {
    const HydroSlab<NV> S = hydro_slab<NV>(P, first, N - first < n ? N - first : n, work);
    const long long     nz = DIM == 3 ? S.nz : 1, cells = (long long)S.nx * S.ny * nz;
    const long long     ring = 2 * (S.ny * nz + S.nx * nz + (DIM == 3 ? (long long)S.nx * S.ny : 0));
    long long           fb = 0;
    for (int a = 0; a < DIM; ++a)
      fb += face_blocks(S, a);
    cudaError_t e = launch_chained(hydro_prims_pass<NV>, blocks(S.box(4)), kPassThreads, 0, st, in, P, clk, step, S);
    if (e == cudaSuccess)
      e = launch_chained(hydro_trace_pass<NV, GRAV>, blocks(cells + ring), kPassThreads, 0, st, P, clk, step, S);
    if (e == cudaSuccess)
      e = launch_chained(hydro_flux_pass<NV, RS>, (unsigned)fb, kPassThreads, 0, st, P, clk, step, S);
    if (e == cudaSuccess)
      e = launch_chained(hydro_update_pass<NV, GRAV>, blocks(cells), kPassThreads, 0, st, in, (double *)Uout, P, clk,
                         step, S);
    if (e != cudaSuccess)
      return e;
  }
  return cudaSuccess;
}

} // namespace EK_NS
