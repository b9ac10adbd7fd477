// FP64 MHD step in passes (2D and 3D), for the reason given in
// ek_hydro_passes.cuh: the FP64 step's time is its count of FP64 instructions,
// so every value is computed once.  The tile kernels repeat the primitives, edge
// fields and traces of each tile's halo and the faces and edges of its rim, and
// wait at barriers with few warps.
//   0. primitives, face fields (ghost layers included) and the step's CFL
//   1. electric field on the cell edges
//   2. compact trace of the cells and one layer around
//   3. one HLLD problem per face and one 2D HLLD emf per edge
//   4. update of the hydro variables and of the face fields
// 0 and 1 over the whole grid, 2 to 4 along slabs of the last axis, so that
// the trace does not grow with the grid.  The arithmetic is that of the tile
// kernels, function by function.
#pragma once

#include "ek_hydro_passes.cuh"
#include "ek_mhd2d_kernels.cuh"

namespace EK_NS
{

using ekc::MhdSlab;
static_assert(MhdSlab<3>::NT == T_N && MhdSlab<2>::NT == V_N, "trace fields");

template <int DIM>
__global__ void __launch_bounds__(kPassThreads)
mhd_prims_pass(const void * __restrict__ U, const KParams P, DevClock * clk, int step, MhdSlab<DIM> S)
{
  chain_begin();
  // a step that must not run (finished, or an earlier one did not run)
  if (clk->sid[step % 3] != step || clk->t[step % 3] >= P.tEnd - 1e-14)
    return;
  const MhdState<double> m = mhd_state<double>(U, P);
  const MhdConst<double> C = mhd_const<double>(P);
  const int              lo = P.gw - 2; // cells [gw - 2, n + gw + 2] of each axis
  const long long        c = pass_index();
  double                 tmax = -INFINITY;
  if (c < (long long)(P.nx + 5) * (P.ny + 5) * (DIM == 3 ? P.nz + 5 : 1))
  {
    int i, j, k;
    box_coords((unsigned)c, P.nx + 5, P.ny + 5, i, j, k);
    i += lo, j += lo, k += DIM == 3 ? lo : 0;
    const SrcCell   s = src_cell(P, i, j, k);
    const long long o = (long long)k * P.plane + (long long)j * P.isize + i;
    double          bl[3], br[3] = { 0.0, 0.0, 0.0 };
#pragma unroll
    for (int f = 0; f < 3; ++f)
    {
      bl[f] = load_face<double>(m, P, s, f);
      S.b[f * P.vstride + o] = bl[f];
    }
    auto below = [&](int g, int n) { return g <= n + P.gw + 1; };
    if (below(i, P.nx) && below(j, P.ny) && (DIM == 2 || below(k, P.nz)))
    {
      // primitives with the fields of the cell's high faces (in 2D the third
      // field has no neighbour; ConvertToPrimitivesFunctor2D_MHD / 3D_MHD)
      br[0] = load_face<double>(m, P, src_cell(P, i + 1, j, k), 0);
      br[1] = load_face<double>(m, P, src_cell(P, i, j + 1, k), 1);
      if (DIM == 3)
        br[2] = load_face<double>(m, P, src_cell(P, i, j, k + 1), 2);
      double u[5], q[8];
      load_hydro<double, double>(m, P, s, u);
      mhd_constoprim<double>(u, bl, br, q, C, [](double (&)[3], double (&)[3]) {});
#pragma unroll
      for (int v = 0; v < 8; ++v)
        S.q[v * P.vstride + o] = q[v];
      auto inside = [&](int g, int n) { return g >= P.gw && g < n + P.gw; };
      if (inside(i, P.nx) && inside(j, P.ny) && (DIM == 2 || inside(k, P.nz)))
      {
        if constexpr (DIM == 2)
          tmax = mhd2d_invdt<double>(q, C, P);
        else
          tmax = mhd_invdt<double>(q, C.gamma0, P.dx, P.dy, P.dz, P.idx, P.idy, P.idz, P.idxd, P.idyd, P.idzd);
      }
    }
  }
  chain_next();
  block_max_commit<kPassThreads>(cand_key(tmax), &clk->key[step % 3]);
  finalize_step(clk, P, step); // dt and its ratios for the other passes
}

// the whole-grid arrays around a cell
template <int DIM>
struct GridAcc
{
  const double * q;
  const double * b;
  const double * e;
  long long      vs, plane;
  int            row;
  __device__ __forceinline__
  GridAcc(const MhdSlab<DIM> & S, const KParams & P, long long o)
    : q(S.q + o), b(S.b + o), e(S.e + o), vs(P.vstride), plane(P.plane), row(P.isize)
  {
  }
  __device__ __forceinline__ double
  Q(int v, int i, int j, int k = 0) const
  {
    return ldg(q + v * vs + (k * plane + j * row + i));
  }
  __device__ __forceinline__ double
  B(int f, int i, int j, int k = 0) const
  {
    return ldg(b + f * vs + (k * plane + j * row + i));
  }
  __device__ __forceinline__ double
  E(int d, int i, int j, int k) const
  {
    return ldg(e + d * vs + (k * plane + j * row + i));
  }
  __device__ __forceinline__ double
  E(int i, int j) const // 2D
  {
    return ldg(e + (j * row + i));
  }
};

// ComputeElecFieldFunctor3D (MHDRunFunctors3D.h:318-356); 8 E in the FP64 FMA
// build, as in the tile kernel
template <int DIM>
__global__ void __launch_bounds__(kPassThreads)
mhd_efield_pass(const KParams P, const DevClock * clk, int step, MhdSlab<DIM> S)
{
  StepConsts sc;
  if (!step_consts(clk, step, sc))
    return;
  const long long c = pass_index(); // cells [gw - 1, n + gw + 1] of each axis
  if (c >= (long long)(P.nx + 3) * (P.ny + 3) * (DIM == 3 ? P.nz + 3 : 1))
    return;
  int i, j, k;
  box_coords((unsigned)c, P.nx + 3, P.ny + 3, i, j, k);
  i += P.gw - 1, j += P.gw - 1, k += DIM == 3 ? P.gw - 1 : 0;
  const long long    o = (long long)k * P.plane + (long long)j * P.isize + i;
  const GridAcc<DIM> A_(S, P, o);
  if constexpr (DIM == 2)
    S.e[o] = corner_ez<double>(A_, 0, 0);
  else
  {
    constexpr double quarter = kFast64<double> ? 1.0 : 0.25, half = kFast64<double> ? 1.0 : 0.5;
    double           uu, vv, ww, A, B, Cc;
    vv = quarter * (A_.Q(IV, 0, -1, -1) + A_.Q(IV, 0, -1, 0) + A_.Q(IV, 0, 0, -1) + A_.Q(IV, 0, 0, 0));
    ww = quarter * (A_.Q(IW, 0, -1, -1) + A_.Q(IW, 0, -1, 0) + A_.Q(IW, 0, 0, -1) + A_.Q(IW, 0, 0, 0));
    B = half * (A_.B(1, 0, 0, -1) + A_.B(1, 0, 0, 0));
    Cc = half * (A_.B(2, 0, -1, 0) + A_.B(2, 0, 0, 0));
    S.e[o] = vv * Cc - ww * B;
    uu = quarter * (A_.Q(IU, -1, 0, -1) + A_.Q(IU, -1, 0, 0) + A_.Q(IU, 0, 0, -1) + A_.Q(IU, 0, 0, 0));
    ww = quarter * (A_.Q(IW, -1, 0, -1) + A_.Q(IW, -1, 0, 0) + A_.Q(IW, 0, 0, -1) + A_.Q(IW, 0, 0, 0));
    A = half * (A_.B(0, 0, 0, -1) + A_.B(0, 0, 0, 0));
    Cc = half * (A_.B(2, -1, 0, 0) + A_.B(2, 0, 0, 0));
    S.e[P.vstride + o] = ww * A - uu * Cc;
    uu = quarter * (A_.Q(IU, -1, -1, 0) + A_.Q(IU, -1, 0, 0) + A_.Q(IU, 0, -1, 0) + A_.Q(IU, 0, 0, 0));
    vv = quarter * (A_.Q(IV, -1, -1, 0) + A_.Q(IV, -1, 0, 0) + A_.Q(IV, 0, -1, 0) + A_.Q(IV, 0, 0, 0));
    A = half * (A_.B(0, 0, -1, 0) + A_.B(0, 0, 0, 0));
    B = half * (A_.B(1, -1, 0, 0) + A_.B(1, 0, 0, 0));
    S.e[2 * P.vstride + o] = uu * B - vv * A;
  }
  chain_next();
}

template <int DIM>
__global__ void __launch_bounds__(kPassThreads, 4)
mhd_trace_pass(const KParams P, const DevClock * clk, int step, MhdSlab<DIM> S)
{
  StepConsts sc;
  if (!step_consts(clk, step, sc))
    return;
  const long long c = pass_index(), n = S.box(2);
  if (c >= n)
    return;
  int i, j, k;
  box_coords((unsigned)c, S.nx + 2, S.ny + 2, i, j, k);
  const int gi = i - 1 + P.gw, gj = S.j0 + j - 1 + P.gw, gk = DIM == 3 ? S.k0 + k - 1 + P.gw : 0;
  const GridAcc<DIM>     A_(S, P, (long long)gk * P.plane + (long long)gj * P.isize + gi);
  const MhdConst<double> C = mhd_const<double>(P);
  if constexpr (DIM == 2)
    trace2d_compact<double>(A_, sc.dtdx, sc.dtdy, C, S.t + c, n);
  else
  {
    double o[T_N];
    trace_state<double>(A_, sc.dtdx, sc.dtdy, sc.dtdz, C, o);
#pragma unroll
    for (int f = 0; f < T_N; ++f)
      S.t[f * n + c] = o[f];
  }
  chain_next();
}

// Blocks of pass 3: the edges (the longer problem) by axis, then the faces,
// each kind padded to whole blocks.  kind 0..2: edges along x, y, z (2D: z
// only), 3..5: faces normal to x, y, z.
template <int DIM>
__host__ __device__ inline void
mhd_kind_extent(const MhdSlab<DIM> & S, int kind, int & ex, int & ey, int & ez)
{
  const bool edge = kind < 3;
  const int  d = kind % 3;
  ex = S.nx + (edge ? d != 0 : d == 0);
  ey = S.ny + (edge ? d != 1 : d == 1);
  ez = DIM == 3 ? S.nz + (edge ? d != 2 : d == 2) : 1;
}
template <int DIM>
__host__ __device__ inline bool
mhd_kind_used(int kind)
{
  return DIM == 3 || kind == 2 || kind == 3 || kind == 4;
}
template <int DIM>
__host__ __device__ inline long long
mhd_kind_blocks(const MhdSlab<DIM> & S, int kind)
{
  int ex, ey, ez;
  mhd_kind_extent(S, kind, ex, ey, ez);
  return mhd_kind_used<DIM>(kind) ? ((long long)ex * ey * ez + kPassThreads - 1) / kPassThreads : 0;
}

template <int DIM, int RS>
__global__ void __launch_bounds__(kPassThreads)
mhd_flux_pass(const KParams P, const DevClock * clk, int step, MhdSlab<DIM> S)
{
  StepConsts sc;
  if (!step_consts(clk, step, sc))
    return;
  int       kind = 0;
  long long blk = blockIdx.x;
  while (blk >= mhd_kind_blocks(S, kind))
    blk -= mhd_kind_blocks(S, kind++);
  int ex, ey, ez, i, j, k;
  mhd_kind_extent(S, kind, ex, ey, ez);
  const long long c = blk * kPassThreads + threadIdx.x;
  if (c >= (long long)ex * ey * ez)
    return;
  box_coords((unsigned)c, ex, ey, i, j, k);
  const MhdConst<double> C = mhd_const<double>(P);
  const double           sr = C.smallr, sp = C.smallp;
  const long long        st = S.trace_stride(); // 64 bits: 46 st passes 2^31 on planes of 4000 x 4000
  const long long        nf = S.box(1), out = S.face(i, j, k);
  const double *         t = S.t + S.tcell(i, j, k);
  const int              back[3] = { 1, S.nx + 2, (S.nx + 2) * (S.ny + 2) };
  if (kind < 3)
  {
    // edge along d at the low corner of the cell; corners RT, RB, LT, LB at -1
    // along (p1, p2), p1, p2 and nowhere (MHDRunFunctors3D.h:2180-2230)
    const int            d = kind, p1 = (d + 1) % 3, p2 = (d + 2) % 3;
    EdgeCorner<double>   RT, RB, LT, LB;
    if constexpr (DIM == 2)
    {
      RT = edge2d_corner<double, 1, 1>(t - back[0] - back[1], st, sr, sp);
      RB = edge2d_corner<double, 1, -1>(t - back[0], st, sr, sp);
      LT = edge2d_corner<double, -1, 1>(t - back[1], st, sr, sp);
      LB = edge2d_corner<double, -1, -1>(t, st, sr, sp);
    }
    else
    {
      RT = edge_corner<double, 1, 1>(t - back[p1] - back[p2], st, d, p1, p2, sr, sp);
      RB = edge_corner<double, 1, -1>(t - back[p1], st, d, p1, p2, sr, sp);
      LT = edge_corner<double, -1, 1>(t - back[p2], st, d, p1, p2, sr, sp);
      LB = edge_corner<double, -1, -1>(t, st, d, p1, p2, sr, sp);
    }
    S.em[(DIM == 3 ? d : 0) * nf + out] = mhd_emf_corners<double>(RT, RB, LT, LB, C.gamma0, C.smallc);
    return;
  }
  // face normal to d between the cell and the one below (MHDRunFunctors3D.h:1839-1874)
  const int d = kind - 3;
  double    ql[8], qr[8], fl[MhdSlab<DIM>::NF];
  if constexpr (DIM == 2)
  {
    face2d_state<double, true>(t - back[d], st, d, ql, sr, sp);
    face2d_state<double, false>(t, st, d, qr, sr, sp);
  }
  else
  {
    face_state_dir<double, true>(t - back[d], st, d, ql, sr, sp);
    face_state_dir<double, false>(t, st, d, qr, sr, sp);
  }
  mhd_riemann<RS, double, MhdSlab<DIM>::NF>(ql, qr, fl, C);
  // out of the face frame (the swap IU <-> IU + d)
#pragma unroll
  for (int v = 0; v < MhdSlab<DIM>::NF; ++v)
  {
    const int w = v == IU ? IU + d : (v == IU + d ? (int)IU : v);
    S.f[(d * MhdSlab<DIM>::NF + w) * nf + out] = fl[v];
  }
  chain_next();
}

template <int DIM>
__global__ void __launch_bounds__(kPassThreads)
mhd_update_pass(const double * __restrict__ Uin, double * __restrict__ Uout, const KParams P, DevClock * clk,
                int step, MhdSlab<DIM> S)
{
  constexpr int NF = MhdSlab<DIM>::NF;
  StepConsts    sc;
  if (!step_consts(clk, step, sc))
    return;
  if (S.last && blockIdx.x == 0 && threadIdx.x == 0)
    step_commit(clk, step, sc.t, sc.dt);
  const long long c = pass_index();
  if (c >= S.box(0))
    return;
  int i, j, k;
  box_coords((unsigned)c, S.nx, S.ny, i, j, k);
  const long long off = (DIM == 3 ? (long long)(S.k0 + k + P.gw) * P.plane : 0) +
                        (long long)(S.j0 + j + P.gw) * P.isize + (i + P.gw);
  const long long nf = S.box(1), at = S.face(i, j, k), st = P.vstride;
  const long long nx1[3] = { 1, S.nx + 1, (long long)(S.nx + 1) * (S.ny + 1) };
  const double    dtd[3] = { sc.dtdx, sc.dtdy, sc.dtdz };
  // UpdateFunctor2D_MHD / 3D_MHD (MHDRunFunctors3D.h:2488-2527)
#pragma unroll
  for (int v = 0; v < 5; ++v)
  {
    double x = ldg(Uin + v * st + off);
#pragma unroll
    for (int a = 0; a < DIM; ++a)
    {
      const double * f = S.f + (a * NF + v) * nf + at;
      x += f[0] * dtd[a];
      x -= f[nx1[a]] * dtd[a];
    }
    Uout[v * st + off] = x;
  }
  // constrained transport (UpdateEmfFunctor2D / 3D, MHDRunFunctors3D.h:2590-2613)
  const double * em = S.em + at;
  double         bx = ldg(Uin + 5 * st + off), by = ldg(Uin + 6 * st + off), bz = ldg(Uin + 7 * st + off);
  if constexpr (DIM == 2)
  {
#pragma unroll
    for (int a = 0; a < 2; ++a)
    {
      const double * f = S.f + (a * NF + 5) * nf + at;
      bz += f[0] * dtd[a];
      bz -= f[nx1[a]] * dtd[a];
    }
    bx += (em[nx1[1]] - em[0]) * sc.dtdy;
    by -= (em[nx1[0]] - em[0]) * sc.dtdx;
  }
  else
  {
    const double *Ex = em, *Ey = em + nf, *Ez = em + 2 * nf;
    bx += (Ez[nx1[1]] - Ez[0]) * sc.dtdy;
    by -= (Ez[nx1[0]] - Ez[0]) * sc.dtdx;
    bx -= (Ey[nx1[2]] - Ey[0]) * sc.dtdz;
    by += (Ex[nx1[2]] - Ex[0]) * sc.dtdz;
    bz += (Ey[nx1[0]] - Ey[0]) * sc.dtdx;
    bz -= (Ex[nx1[1]] - Ex[0]) * sc.dtdy;
  }
  Uout[5 * st + off] = bx;
  Uout[6 * st + off] = by;
  Uout[7 * st + off] = bz;
  chain_next();
}

template <int DIM>
inline MhdSlab<DIM>
mhd_slab(const KParams & P, int first, int n, void * work)
{
  MhdSlab<DIM> S;
  S.nx = P.nx;
  S.ny = DIM == 2 ? n : P.ny;
  S.nz = DIM == 2 ? 1 : n;
  S.j0 = DIM == 2 ? first : 0;
  S.k0 = DIM == 2 ? 0 : first;
  S.last = first + n == (DIM == 2 ? P.ny : P.nz);
  S.q = (double *)work;
  S.b = S.q + 8 * P.vstride;
  S.e = S.b + 3 * P.vstride;
  S.t = S.e + MhdSlab<DIM>::NE * P.vstride;
  S.f = S.t + MhdSlab<DIM>::NT * S.box(2);
  S.em = S.f + DIM * MhdSlab<DIM>::NF * S.box(1);
  return S;
}
// one step: phase 0 (passes 0 and 1), phase 1 (passes 2 to 4)
template <int DIM>
cudaError_t
mhd_passes_t(int phase, const void * Uin, void * Uout, void * work, const KParams & P, DevClock * clk, int step,
             cudaStream_t st)
{
  auto      blocks = [](long long items) { return (unsigned)((items + kPassThreads - 1) / kPassThreads); };
  const int N = DIM == 2 ? P.ny : P.nz, n = P.slab;
  if (phase == 0)
  {
    const MhdSlab<DIM> S = mhd_slab<DIM>(P, 0, n, work);
    auto all = [&](int w) { return (long long)(P.nx + w) * (P.ny + w) * (DIM == 3 ? P.nz + w : 1); };
    cudaError_t e = launch_chained(mhd_prims_pass<DIM>, blocks(all(5)), kPassThreads, 0, st, Uin, P, clk, step, S);
    if (e == cudaSuccess)
      e = launch_chained(mhd_efield_pass<DIM>, blocks(all(3)), kPassThreads, 0, st, P, clk, step, S);
    return e;
  }
  for (int first = 0; first < N; first += n)
  {
    const MhdSlab<DIM> S = mhd_slab<DIM>(P, first, N - first < n ? N - first : n, work);
    long long          fb = 0;
    for (int kind = 0; kind < 6; ++kind)
      fb += mhd_kind_blocks(S, kind);
    auto flux = P.riemann == 1 ? mhd_flux_pass<DIM, 1> : P.riemann == 2 ? mhd_flux_pass<DIM, 2> : mhd_flux_pass<DIM, 4>;
    cudaError_t e = launch_chained(mhd_trace_pass<DIM>, blocks(S.box(2)), kPassThreads, 0, st, P, clk, step, S);
    if (e == cudaSuccess)
      e = launch_chained(flux, (unsigned)fb, kPassThreads, 0, st, P, clk, step, S);
    if (e == cudaSuccess)
      e = launch_chained(mhd_update_pass<DIM>, blocks(S.box(0)), kPassThreads, 0, st, (const double *)Uin, (double *)Uout,
                         P, clk, step, S);
    if (e != cudaSuccess)
      return e;
  }
  return cudaSuccess;
}

// Cells of the last axis per slab of the FP64 step in passes.  0 for the small 2D
// grids, where one tile kernel ends before four or five launches do (us per step,
// passes / tiles): hydro 64^2 28 / 15, 256^2 49 / 42 (both when the rule was made),
// 512^2 118 / 125, 1024^2 431 / 467; MHD 64^2 53 / 45, 128^2 72 / 66 (then), 200 x 136
// (425 tiles of 8 x 8) 89 / 89, 256^2 139 / 201, 1024^2 1861 / 2834.  3D: hydro 24^3 30 /
// 64, 33 x 31 x 99 89 / 211, 96^3 606 / 711, 200 x 180 x 160 3861 / 5490; MHD 16^3 61 /
// 179, 32^3 158 / 292, 64^3 1016 / 1587, 160^3 15237 / 19328.
int
pass_slab(int dim, int mhd, const KParams & P)
{
  if (dim == 2 && (mhd ? (long long)((P.nx + 7) / 8) * ((P.ny + 7) / 8) <= 3ll * P.sms : (long long)P.nx * P.ny < (1ll << 18)))
    return 0;
  // the MHD arrays of the whole grid do not count towards a slab
  const long long whole = mhd ? (long long)pass_bytes(dim, mhd, P, 0) : 0;
  return ekc::slab_cells(dim == 2 ? P.ny : P.nz, kPassBytes,
                         [&](int n) { return (long long)pass_bytes(dim, mhd, P, n) - whole; });
}
// bytes of the workspace for slabs of n cells (MHD, n = 0: of the whole grid's arrays)
size_t
pass_bytes(int dim, int mhd, const KParams & P, int n)
{
  if (!mhd)
    return (size_t)(dim == 2 ? hydro_slab<4>(P, 0, n, nullptr).bytes() : hydro_slab<5>(P, 0, n, nullptr).bytes());
  const size_t whole = sizeof(double) * (11 + (dim == 2 ? MhdSlab<2>::NE : MhdSlab<3>::NE)) * (size_t)P.vstride;
  if (n == 0)
    return whole;
  return whole + (size_t)(dim == 2 ? mhd_slab<2>(P, 0, n, nullptr).slab_bytes() : mhd_slab<3>(P, 0, n, nullptr).slab_bytes());
}
cudaError_t
mhd_passes(int dim, int phase, const void * Uin, void * Uout, void * work, const KParams & P, DevClock * clk, int step,
           cudaStream_t st)
{
  return dim == 2 ? mhd_passes_t<2>(phase, Uin, Uout, work, P, clk, step, st)
                  : mhd_passes_t<3>(phase, Uin, Uout, work, P, clk, step, st);
}
// launches of a step in passes
int
pass_launches(int dim, int mhd, const KParams & P)
{
  const int N = dim == 2 ? P.ny : P.nz, slabs = (N + P.slab - 1) / P.slab;
  return mhd ? 2 + 3 * slabs : 4 * slabs;
}

} // namespace EK_NS
