// 2D hydro step by warps that march along y.
//
// A tile kernel with its primitives, face states and fluxes in shared memory
// executes 994 instructions a cell in FP32 where the arithmetic of a cell takes
// about 400: primitives of the halo 1.69 x and traces of the ring 1.33 x (32 x 8
// tile), a shared-memory access with its address for every value that passes
// from one phase to the next, rounds that are partly empty, and three barriers.
// Here a warp owns 28 columns (its 32 lanes are 28 and two halo columns on each
// side) and marches over a run of rows: the x neighbours come by shuffles, the
// rows below stay in registers, and nothing waits for another warp.  A run of n
// rows takes the primitives of n + 4, the traces of n + 2 and the y faces of n + 1
// (678 instructions a cell with runs of 8).  Issue bounds large grids (57 to 73 %
// busy, 20 warps per SM at 96 registers; at 80, 24 warps, 2 % slower), the chain
// of one row, 0.6 us, small ones.  us per step, tile / march: mixed 64^2 12.4 /
// 7.9, 512^2 18.5 / 13.2, 1022 x 518 29.6 / 19.4, 2048^2 182 / 84 (the first and
// last row in the loop, by branches: 8.8, 14.4, 22.2, 91); ensemble of 32
// runs of 64^2 to 256^2 mixed 42 / 28, FP64 852 / 549.
#pragma once

#include "ek_chunk.h"
#include "ek_hydro_kernels.cuh"

namespace EK_NS
{

using ekc::kRowCols;  // columns that a warp updates
using ekc::kRowWarps; // warps of a CTA, on consecutive runs of rows

// What the rows need of a run's parameters, for the ensemble, whose instances'
// parameters are in global memory: its CTAs keep these in shared memory.
struct RowParams
{
  int       nx, ny, gw, isize, bc[4];
  long long vstride;
  double    dx, dy, idxd, idyd;
  float     idx, idy;
  __device__ __forceinline__ void
  set(const KParams & P)
  {
    nx = P.nx, ny = P.ny, gw = P.gw, isize = P.isize, vstride = P.vstride;
    dx = P.dx, dy = P.dy, idxd = P.idxd, idyd = P.idyd, idx = P.idx, idy = P.idy;
    for (int b = 0; b < 4; ++b)
      bc[b] = P.bc[b];
  }
};

// Rows [j0, j0 + n) of the columns [x0, x0 + 28): the step of these cells;
// returns the largest CFL candidate of the lane's cells.  Called by whole warps.
template <class S, class R, int RS, bool GRAV, class PP>
__device__ __forceinline__ R
hydro2d_rows(const S * __restrict__ Uin, S * __restrict__ Uout, const PP & P, const HydroConst<R> & C,
             const StepConsts & sc, int x0, int j0, int n)
{
  constexpr int      NV = 4;
  constexpr unsigned ALL = 0xffffffffu;
  const int          lane = threadIdx.x & 31, i = x0 + lane - 2; // lanes past the ghosts repeat the last (bc_map)
  const bool         mine = lane >= 2 && lane < 30 && i < P.nx;
  const R            dtdx = to_r<R>(sc.dtdx), dtdy = to_r<R>(sc.dtdy), hdt = (R)(0.5 * sc.dt);
  const bool         same_xy = dtdx == dtdy; // square cells: one time-advanced state for all faces
  bool               flip_x = false;
  const int          si = bc_map(P.gw + i, P.nx, P.gw, P.bc[0], P.bc[1], &flip_x);

  // A row is loaded one iteration before its first use, and nothing but the loads
  // stands there (a sign flip would wait for them).
  struct Row
  {
    S    u[NV];
    bool flip;
  };
  auto load = [&](int j, Row & w) {
    w.flip = false;
    const int sj = bc_map(P.gw + j, P.ny, P.gw, P.bc[2], P.bc[3], &w.flip);
    const S * p = Uin + (long long)sj * P.isize + si;
#pragma unroll
    for (int v = 0; v < NV; ++v)
      w.u[v] = ldg(p + v * P.vstride);
  };
  auto prims = [&](const Row & w, R (&q)[NV]) {
    R u[NV] = { (R)w.u[ID], (R)w.u[IP], neg_if((R)w.u[IU], flip_x), neg_if((R)w.u[IV], w.flip) };
    hydro_prims<R, NV>(u, q, C);
  };

  R   tmax = R(-INFINITY);
  R   qa[NV], qb[NV], qc[NV]; // primitives of the rows r - 1, r, r + 1
  Row next;
  {
    Row wa, wb;
    load(j0 - 2, wa);
    load(j0 - 1, wb);
    load(j0, next);
    prims(wa, qa);
    prims(wb, qb);
    prims(next, qc);
  }
  R top[NV], acc[NV] = {}, rho_old = R(0); // state above row r - 1; its update so far
  // one row; the first (-1) and the last (n) only for the states that face the run
  auto row = [&](int r, auto part) {
    constexpr bool first = part.value < 0, last = part.value > 0, inner = !first && !last;
    if constexpr (!last)
      load(j0 + r + 2, next);
    S u0[NV];
    if constexpr (inner)
    {
      const S * in = Uin + (long long)(P.gw + j0 + r) * P.isize + si;
#pragma unroll
      for (int v = 0; v < NV; ++v)
        u0[v] = ldg(in + v * P.vstride);
    }
    R dX[NV], dY[NV], dZ[NV], s[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v)
    {
      const R lo = __shfl_up_sync(ALL, qb[v], 1), hi = __shfl_down_sync(ALL, qb[v], 1);
      dX[v] = slope_h<R>(qb[v], hi, lo, C.slope_type);
      dY[v] = slope_h<R>(qb[v], qc[v], qa[v], C.slope_type);
      dZ[v] = R(0);
    }
    hydro_sources<R, NV>(qb, dX, dY, dZ, s, C);
    bool kick = false; // gravity predictor of the face states
    R    hg[3];
    if constexpr (GRAV)
    {
      kick = P.grav_hancock;
      R g[3];
      grav_at<S, R, NV>(P, P.gw + i, P.gw + j0 + r, 0, g);
#pragma unroll
      for (int e = 0; e < 3; ++e)
        hg[e] = hdt * g[e];
    }
    FaceStates<R, NV> F(qb, s, dtdx, C.smallr);
    R                 fx[NV];
    if constexpr (inner)
    {
      // x flux through the low face of the cell
      R l[NV], h[NV];
      F.get(dX, false, h);
      F.get(dX, true, l);
      if (kick)
      {
        grav_kick<R, NV>(h, hg);
        grav_kick<R, NV>(l, hg);
      }
#pragma unroll
      for (int v = 0; v < NV; ++v)
        l[v] = __shfl_up_sync(ALL, l[v], 1);
      hydro_riemann<RS, R, NV>(l, h, fx, C);
#pragma unroll
      for (int v = 0; v < NV; ++v)
        fx[v] = flux_scaled(fx[v], dtdx);
    }
    F.turn(dtdy, same_xy);
    R fy[NV];
    if constexpr (!first)
    {
      // y flux through the low face, IU and IV swapped around the solver
      R l[NV], h[NV], f[NV];
      F.get(dY, false, f);
      if (kick)
        grav_kick<R, NV>(f, hg);
#pragma unroll
      for (int v = 0; v < NV; ++v)
      {
        const int w = v < IU ? v : IU + IV - v;
        l[v] = top[w];
        h[v] = f[w];
      }
      hydro_riemann<RS, R, NV>(l, h, f, C);
#pragma unroll
      for (int v = 0; v < NV; ++v)
        fy[v] = flux_scaled(f[v < IU ? v : IU + IV - v], dtdy);
    }
    if constexpr (!first)
    {
      // row r - 1 is complete (of r = 0: nothing) (UpdateFunctor2D, HydroRunFunctors2D.h:809-836, in its order)
#pragma unroll
      for (int v = 0; v < NV; ++v)
        acc[v] = sub_flux(acc[v], fy[v], dtdy);
      const int          gj = P.gw + j0 + r - 1;
      [[maybe_unused]] R g[3];
      if constexpr (GRAV)
      {
        // gravity source term after the flux update (SolverHydroMuscl.cpp:245-252)
        grav_at<S, R, NV>(P, P.gw + i, gj, 0, g);
        grav_source<R, NV>(acc, rho_old, g, hdt, C);
      }
      if (mine && r >= 1)
      {
        // the next step's dt is computed on the stored (possibly rounded) state
        S * out = Uout + (long long)gj * P.isize + P.gw + i;
        R   us[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v)
        {
          out[v * P.vstride] = (S)acc[v];
          us[v] = (R)(S)acc[v];
        }
        if constexpr (GRAV)
          tmax = max_cand(tmax, hydro_invdt_grav<R, NV>(us, g, C, P));
        else
          tmax = max_cand(tmax, hydro_invdt<R, NV>(us, C, P));
      }
    }
    if constexpr (inner)
    {
#pragma unroll
      for (int v = 0; v < NV; ++v)
      {
        R x = (R)u0[v];
        if (v == ID)
          rho_old = x;
        x = add_flux(x, fx[v], dtdx);
        x = sub_flux(x, __shfl_down_sync(ALL, fx[v], 1), dtdx);
        acc[v] = add_flux(x, fy[v], dtdy);
      }
    }
    if constexpr (!last)
    {
      F.get(dY, true, top);
      if (kick)
        grav_kick<R, NV>(top, hg);
#pragma unroll
      for (int v = 0; v < NV; ++v)
      {
        qa[v] = qb[v];
        qb[v] = qc[v];
      }
      prims(next, qc);
    }
  };
  row(-1, std::integral_constant<int, -1>());
#pragma unroll 1
  for (int r = 0; r < n; ++r)
    row(r, std::integral_constant<int, 0>());
  row(n, std::integral_constant<int, 1>());
  return tmax;
}

// grid: strips of 28 columns, CTAs of kRowWarps runs of `rows` rows
template <class S, class R, int RS, bool GRAV>
__global__ void __launch_bounds__(32 * kRowWarps, EK_MINB(R, EK_H2_MINB_F32, 2))
hydro2d_rows_step(const S * __restrict__ Uin, S * __restrict__ Uout, KParams P, DevClock * clk, int step, int rows)
{
  StepConsts sc; // computed once for the step by the last block of the kernel before
  if (!step_consts(clk, step, sc))
    return;
  const int j0 = (blockIdx.y * kRowWarps + (threadIdx.x >> 5)) * rows;
  R         tmax = R(-INFINITY);
  if (j0 < P.ny)
    tmax = hydro2d_rows<S, R, RS, GRAV>(Uin, Uout, P, hydro_const<R>(P), sc, blockIdx.x * kRowCols, j0,
                                        min(rows, P.ny - j0));
  chain_next();
  block_max_commit<32 * kRowWarps>(cand_key((double)tmax), &clk->key[(step + 1) % 3]);
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0)
    step_commit(clk, step, sc.t, sc.dt);
  finalize_step(clk, P, step + 1); // the next step's dt, once its CFL key is complete
}

// Ensemble of independent 2D runs (uneven grids, own dt each): one launch is one
// step of every instance, a CTA one tile of the flat work list.  The step number
// is the instance's own (DevClock::next, written by its last block), so a
// captured sequence of steps can be replayed as is, and an instance at its end
// time costs its blocks' first loads.
template <class S, class R>
__global__ void __launch_bounds__(32 * kRowWarps, EK_MINB(R, EK_H2_MINB_F32, 2))
ensemble2d_step(const EnsInstance * __restrict__ insts, const EnsTile * __restrict__ tiles, int rows)
{
  const EnsTile       w = tiles[blockIdx.x];
  const EnsInstance & in = insts[w.inst];
  DevClock * const    clk = in.clk;
  __shared__ RowParams     P;
  __shared__ HydroConst<R> C;
  if (threadIdx.x == 0)
  {
    P.set(in.P);
    C = hydro_const<R>(in.P);
  }
  __syncthreads();
  chain_begin();
  const int  step = clk->next;
  StepConsts sc;
  if (!step_consts(clk, step, sc))
    return;
  const int       j0 = (w.by * kRowWarps + (threadIdx.x >> 5)) * rows;
  R               tmax = R(-INFINITY);
  if (j0 < P.ny)
    tmax = hydro2d_rows<S, R, 3, false>((const S *)in.U[step % 2], (S *)in.U[(step + 1) % 2], P, C, sc,
                                        w.bx * kRowCols, j0, min(rows, P.ny - j0));
  chain_next();
  block_max_commit<32 * kRowWarps>(cand_key((double)tmax), &clk->key[(step + 1) % 3]);
  if (w.bx == 0 && w.by == 0 && threadIdx.x == 0)
    step_commit(clk, step, sc.t, sc.dt);
  finalize_step(clk, in.P, step + 1, nullptr, in.tiles);
}

// FP64 mass and total energy of every instance (blockIdx.y = instance), from the
// buffer of its own last step: an instance at its end time stays in it
template <class S>
__global__ void
ensemble_totals_kernel(const EnsInstance * __restrict__ insts, double * __restrict__ out)
{
  const EnsInstance & in = insts[blockIdx.y];
  const KParams &     P = in.P;
  const S *           U = (const S *)in.U[in.clk->iteration % 2];
  double              m = 0.0, e = 0.0;
  for_interior_rows(P, [&](int i, int j, int) {
    const long long off = (long long)j * P.isize + i;
    m += (double)U[off];
    e += (double)U[P.vstride + off];
  });
  for (int o = 16; o > 0; o >>= 1)
  {
    m += __shfl_xor_sync(0xffffffffu, m, o);
    e += __shfl_xor_sync(0xffffffffu, e, o);
  }
  if ((threadIdx.x & 31) == 0)
  {
    atomicAdd(out + 2 * blockIdx.y, m);
    atomicAdd(out + 2 * blockIdx.y + 1, e);
  }
}

} // namespace EK_NS
