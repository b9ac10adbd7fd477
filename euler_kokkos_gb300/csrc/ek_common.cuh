// Common device-side definitions for the fused MUSCL-Hancock kernels.
//
// Layout (identical to the reference's Kokkos::LayoutLeft device arrays,
// kokkos_shared.h:24-42): U[var][k][j][i], i fastest, ghost cells included.
// The step kernels never read the ghost cells stored in memory: a ghost
// coordinate is mapped to the interior cell the reference's boundary fill
// would copy from (BoundariesFunctors.h:17-1057), one dimension at a time.
// Because the reference fills the faces in the order x, y, z over the full
// transverse ranges (SolverBase.cpp:488-512), every edge/corner ghost ends up
// as the composition of the per-dimension maps, which is what this mapping
// computes.
#pragma once

#include <cstdint>
#include <cuda.h> // CUtensorMap (the type only; maps are encoded through the runtime's driver entry point)
#include <cuda_runtime.h>

#ifndef EK_NS
#define EK_NS ek_fast
#endif

namespace ekc
{

// variable indexes, enums.h:17-40
enum : int
{
  ID = 0,
  IP = 1,
  IU = 2,
  IV = 3,
  IW = 4,
  IA = 5,
  IB = 6,
  IC = 7
};

enum : int
{
  BC_DIRICHLET = 1, // reflecting
  BC_NEUMANN = 2,   // outflow / copy
  BC_PERIODIC = 3
};

struct KParams
{
  int       nx, ny, nz, gw;
  int       isize, jsize, ksize;
  int       mhd;
  long long plane;   // isize * jsize
  long long vstride; // isize * jsize * ksize: distance between variables
  int       bc[6];
  double    dx, dy, dz;
  double    gamma0, smallr, smallc, smallp, slope_type, cfl, tEnd, cIso;
  int       riemann;
  int       kchunk;       // interior planes per CTA (3D kernels)
  int       kchunk_trace; // trace planes per CTA (3D MHD trace kernel)
  int       sms;          // SMs of the device
  // FP32 copies prepared on the host, so that mixed kernels do no per-thread
  // FP64 arithmetic (one FP64 instruction costs 64 FP32 ones on GB300)
  float     gamma0f, smallrf, smallcf, smallpf, slopef;
  float     idx, idy, idz; // 1/dx, 1/dy, 1/dz
  double    idxd, idyd, idzd; // 1/dx, 1/dy, 1/dz in FP64 (FP64 FMA build's CFL)
  int       mhd_stage;     // MHD update: stage the trace planes in shared memory
  int       slab;          // cells of the last axis per slab (FP64 steps in passes)
  double    entho;           // 1 / (gamma0 - 1)
  float     enthof;
  double    gamma6, smallpp; // riemann_approx constants (HydroParams.cpp:353-356)
  float     gamma6f, smallppf;
  // static gravity (hydro; GravityParams.h:22-37): the field is gfield
  // (dim planes of the state's precision over the full grid) when set,
  // else the uniform vector g
  int          grav;         // source term + gravity CFL
  int          grav_hancock; // Hancock predictor of the face states
  double       g[3];
  float        gf[3];
  double       cfl_dxmin, dxmin; // cfl * min(dx, dy[, dz]) and min(dx, dy[, dz])
  float        cfl_dxminf, idxminf;
  const void * gfield;
};

// Per-step scalars kept on the device so that consecutive steps need no host
// round trip.  Slot s = step % 3 holds the max-reduced inverse time step
// (as an order-preserving integer key) and the time at the start of step.
// dt of a step and its FP64 ratios, computed once per step (step = -1: none)
struct StepConsts
{
  double t, dt, dtdx, dtdy, dtdz;
  int    step, active;
};
// Quotients by a shared denominator: the exact build divides each one, as the
// reference does; the FMA builds take one reciprocal and multiply (FP64: a
// division is a sequence of FMAs on GB300's 1/64-rate FP64 pipe).
#ifdef EK_EXACT_ONLY
constexpr bool kShareRecip = false;
#else
constexpr bool kShareRecip = true;
#endif

struct DevClock
{
  unsigned long long key[3];
  double             t[3];
  int                sid[3];    // step number the slot was written for
  int                iteration; // number of steps taken
  int                error;     // sticky device error flags
  double *           dtlog;     // dt of each step (capacity dtcap)
  int                dtcap;
  double             last_dt;   // dt of the last step taken (read with the clock)
  StepConsts         sc[3];     // per slot, by the last block of the CFL kernel
  unsigned int       fin[3];    // blocks of that kernel done (reset by the last)
  int                next;      // the step whose constants were computed last
};

enum : int
{
  EK_DEVERR_NONFINITE_DT = 1,
  EK_DEVERR_TMA_TIMEOUT = 2, // a tensor copy did not complete within its wait limit
};

// One instance of an ensemble of independent runs and one tile of work.
struct EnsInstance
{
  KParams    P;
  void *     U[2]; // ping-pong states
  DevClock * clk;
  unsigned   tiles; // of the work list
};
struct EnsTile
{
  int inst, bx, by;
};

// Mixed-precision MHD state: 5 FP32 hydro planes, then (256-byte aligned) the
// 3 FP64 face-field planes.
__host__ __device__ inline size_t
mixed_bfield_offset(long long vstride)
{
  return ((size_t)(5 * vstride * 4) + 255) / 256 * 256;
}
__host__ __device__ inline double *
mixed_bfield(void * U, const KParams & P)
{
  return (double *)((char *)U + mixed_bfield_offset(P.vstride));
}
__host__ __device__ inline const double *
mixed_bfield(const void * U, const KParams & P)
{
  return (const double *)((const char *)U + mixed_bfield_offset(P.vstride));
}

// order-preserving map double -> uint64 (total order on non-NaN values)
__host__ __device__ inline unsigned long long
dkey(double x)
{
  unsigned long long b;
#ifdef __CUDA_ARCH__
  b = (unsigned long long)__double_as_longlong(x);
#else
  memcpy(&b, &x, 8);
#endif
  return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}
__host__ __device__ inline double
dkey_inv(unsigned long long k)
{
  unsigned long long b = (k & 0x8000000000000000ull) ? (k & 0x7fffffffffffffffull) : ~k;
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double x;
  memcpy(&x, &b, 8);
  return x;
#endif
}
// key of -DBL_MAX: the identity of the reference's Kokkos::Max reducer
#define EK_KEY_LOWEST 0x0010000000000000ull

} // namespace ekc

namespace EK_NS
{
using namespace ekc;
// Minimum resident CTAs per SM requested from the register allocator for the
// step kernels (FP32 / FP64 instantiations); overridable at build time.
#ifndef EK_H3_MINB_F32
#define EK_H3_MINB_F32 4
#endif
#ifndef EK_H3_MINB_F64
#define EK_H3_MINB_F64 2
#endif
#ifndef EK_MT_MINB_F32
#define EK_MT_MINB_F32 0
#endif
#ifndef EK_MT_MINB_F64
#define EK_MT_MINB_F64 0
#endif
#ifndef EK_MU_MINB_F32
#define EK_MU_MINB_F32 8
#endif
#ifndef EK_MU_MINB_F64
#define EK_MU_MINB_F64 2
#endif
#ifndef EK_M2_MINB_F32
#define EK_M2_MINB_F32 0
#endif
#ifndef EK_M2_MINB_F64
#define EK_M2_MINB_F64 0
#endif
#ifndef EK_H2_MINB_F32
#define EK_H2_MINB_F32 5
#endif
#define EK_MINB(R, F32, F64) (sizeof(R) == 4 ? (F32) : (F64))
// Tile shapes (output cells per CTA in x, y) of the step kernels; the
// defaults are the measured best, euler_kokkos_gb300/tuning.py re-tunes them.
#ifndef EK_H3_TX
#define EK_H3_TX 32
#endif
#ifndef EK_H3_TY
#define EK_H3_TY 8
#endif
#ifndef EK_MT_TX
#define EK_MT_TX 32
#endif
#ifndef EK_MT_TY
#define EK_MT_TY 4
#endif
#ifndef EK_MU_TX
#define EK_MU_TX 16
#endif
#ifndef EK_MU_TY
#define EK_MU_TY 8
#endif
// The FP64 MHD kernels: bound by the FP64 pipe they gain nothing from longer
// rows, and smaller tiles fill the SMs of small grids and balance the others.
// Best times over the planes per CTA (us): update 32 x 8 / 16 x 8: 242 / 242 at
// 32^3, 675 / 536 at 48^3, 1272 / 1282 at 64^3, 2437 / 2440 at 96 x 80 x 70 (256
// threads on a 16 x 8 tile: 211, 527, 1327, 2502); trace 16 x 8 / 8 x 8: 89 / 72
// at 32^3, 398 / 361 at 64^3, 999 / 1003 at 96^3.
#ifndef EK_MU_TX_F64
#define EK_MU_TX_F64 16
#endif
#ifndef EK_MU_TY_F64
#define EK_MU_TY_F64 8
#endif
#ifndef EK_MT_TX_F64
#define EK_MT_TX_F64 8
#endif
#ifndef EK_MT_TY_F64
#define EK_MT_TY_F64 8
#endif
#ifndef EK_M2_TX
#define EK_M2_TX 16
#endif
#ifndef EK_M2_TY
#define EK_M2_TY 8
#endif


// FP64 <-> FP32 conversions on the integer pipes.  The hardware conversion
// instructions run on the FP64 unit, which issues at 1/64 of the FP32 rate on
// this GPU, so the mixed kernels convert the FP64 face fields this way.
// Normal results and zeros take the integer path and equal the hardware
// round-to-nearest-even conversion bit for bit; subnormal, overflowing,
// infinite and NaN values fall back to the hardware instruction.
__device__ __forceinline__ float
d2f_rn(double x)
{
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned           hi = (unsigned)(b >> 32), lo = (unsigned)b;
  const unsigned           e = (hi >> 20) & 0x7ffu;
  if (e - 897u <= 253u)
  {
    const unsigned m = ((hi & 0xfffffu) << 3) | (lo >> 29);
    const unsigned rest = lo & 0x1fffffffu;
    unsigned       f = (hi & 0x80000000u) | ((e - 896u) << 23) | m;
    f += (rest > 0x10000000u || (rest == 0x10000000u && (m & 1u))) ? 1u : 0u;
    return __uint_as_float(f);
  }
  if ((b << 1) == 0ull)
    return __uint_as_float(hi & 0x80000000u);
  return __double2float_rn(x);
}
__device__ __forceinline__ double
f2d(float x)
{
  const unsigned b = __float_as_uint(x);
  const unsigned e = (b >> 23) & 0xffu;
  if (e - 1u < 254u)
    return __hiloint2double((int)((b & 0x80000000u) | ((e + 896u) << 20) | ((b & 0x7fffffu) >> 3)),
                            (int)(b << 29));
  if ((b << 1) == 0u)
    return __hiloint2double((int)(b & 0x80000000u), 0);
  return (double)x;
}
// Approximate FP32 reciprocal, reciprocal square root and square root (one
// special-function-unit instruction each, about 1 ulp).  The mixed form uses
// them where the reference divides several numbers by one denominator or
// divides by a square root; the FP64 forms keep the reference's divisions.
__device__ __forceinline__ float
rcp_a(float x)
{
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float
rsqrt_a(float x)
{
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float
sqrt_a(float x)
{
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Packed FP32 pairs: one instruction computes two lanes (sm_100 and later).
// The mixed form's solvers put the left and right states of a face in the two
// lanes; each lane rounds as the scalar operation does.
__device__ __forceinline__ float2
f2(float a, float b)
{
  return make_float2(a, b);
}
__device__ __forceinline__ float2
f2s(float a)
{
  return make_float2(a, a);
}
__device__ __forceinline__ float2
add2(float2 a, float2 b)
{
  return __fadd2_rn(a, b);
}
__device__ __forceinline__ float2
sub2(float2 a, float2 b)
{
  return __ffma2_rn(b, make_float2(-1.f, -1.f), a); // b * -1 is exact: one rounding, as a - b
}
__device__ __forceinline__ float2
mul2(float2 a, float2 b)
{
  return __fmul2_rn(a, b);
}
__device__ __forceinline__ float2
fma2(float2 a, float2 b, float2 c)
{
  return __ffma2_rn(a, b, c);
}
__device__ __forceinline__ float2
neg2(float2 a)
{
  return make_float2(-a.x, -a.y);
}

// ---------------------------------------------------------------------------
// FP64 arithmetic of the FMA build.  The FP64 kernels are bound by GB300's
// FP64 pipe (ncu: 78-84 % busy with 8 % of the issue slots used), which takes
// one warp instruction per 16 cycles and SM and serves not only additions and
// products but also comparisons, minima, maxima, negations and conversions
// (probe, independent chains: FMA 617 Gop/s, fmax 490, 1/x 115, c/x 70, sqrt
// 70, rsqrt 108).  The helpers below keep what need not be there on the
// integer and special-function pipes.
// ---------------------------------------------------------------------------
template <class R>
constexpr bool kFast64 = sizeof(R) == 8 && kShareRecip;

__device__ __forceinline__ int
hi32(double x)
{
  return __double2hiint(x);
}
__device__ __forceinline__ double
with_hi(int hi, double x)
{
  return __hiloint2double(hi, __double2loint(x));
}
// zero, infinity or NaN (the seed instructions below return no subnormals)
__device__ __forceinline__ bool
seed_special(double y)
{
  return ((hi32(y) + 0x00100000) & 0x7fe00000) == 0;
}
// 1/x: the hardware's 20-bit seed y (rcp.approx.ftz.f64), then the geometric
// series of 1/(1 - e), e = 1 - x y, to second order: e^3 is below 2^-58, so
// the error is that of the last rounding.  Measured over 2^-40..2^40: 1.003 x
// 2^-53 at most, 1.000 for the division; 182 Gop/s, 115 for the division.
// Subnormal x give infinity, |x| above 2^1022 zero.
__device__ __forceinline__ double
rcp64(double x)
{
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  const double r = fma(y, fma(e, e, e), y);
  return seed_special(y) ? y : r;
}
// 1/sqrt(x): the hardware's seed (rsqrt.approx.ftz.f64) and the binomial
// series of (1 - r)^(-1/2), r = 1 - x y^2, to second order.  Error 1.012 x
// 2^-53 at most, as CUDA's rsqrt.
__device__ __forceinline__ double
rsqrt64(double x)
{
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double r = fma(-x, y * y, 1.0);
  const double q = fma(y * r, fma(r, 0.375, 0.5), y);
  return seed_special(y) ? y : q;
}
// sqrt(x) from the same series; error 1.5 x 2^-53 at most (84 Gop/s, 70 for
// the correctly rounded root).  Zero, infinity and subnormals return x.
__device__ __forceinline__ double
sqrt64(double x)
{
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double g = x * y;
  const double r = fma(-g, y, 1.0);
  const double q = fma(g * r, fma(r, 0.375, 0.5), g);
  return seed_special(y) ? ((hi32(y) & 0x000fffff) != 0 ? y : x) : q;
}
// x not in [2^-1021, 2^1022): the results above may be rounded, 0 or infinite
__device__ __forceinline__ bool
out_of_range64(double x)
{
  return (unsigned)(hi32(x) - 0x00200000) >= 0x7fc00000u;
}
__device__ __forceinline__ bool
both_zero64(double a, double b) // a, b >= 0
{
  return (__double_as_longlong(a) | __double_as_longlong(b)) == 0;
}
// sqrt(n / d) for n >= 0, d > 0; by the quotient where n d leaves the range (a
// branch on integer comparisons that ordinary states do not take)
__device__ __forceinline__ double
sqrt_ratio64(double n, double d)
{
  const double x = n * d;
  double       c = n * rsqrt64(x);
  if (out_of_range64(x))
    c = both_zero64(n, n) ? 0.0 : sqrt64(n * rcp64(d));
  return c;
}
// the larger of sqrt(n1 / d1) and sqrt(n2 / d2), the quotients compared by products
__device__ __forceinline__ double
sqrt_larger_ratio64(double n1, double d1, double n2, double d2)
{
  const long long p1 = __double_as_longlong(n1 * d2), p2 = __double_as_longlong(n2 * d1);
  const bool      first = p1 >= p2;
  if (out_of_range64(__longlong_as_double(first ? p1 : p2)))
    return both_zero64(n1, n2) ? 0.0 : sqrt64(fmax(n1 * rcp64(d1), n2 * rcp64(d2)));
  return sqrt_ratio64(first ? n1 : n2, first ? d1 : d2);
}
__device__ __forceinline__ bool
positive64(double x) // x > 0
{
  return (unsigned long long)(__double_as_longlong(x) - 1) < 0x7ff0000000000000ull;
}
__device__ __forceinline__ bool
negative64(double x) // the sign bit
{
  return hi32(x) < 0;
}
// the larger of x (any sign) and f >= 0, f where x is a NaN of either sign (as fmax);
// the smaller of two non-negative values: the integer order of the bit patterns is
// the numbers' order.  x stays where its bits lie between those of f and infinity.
__device__ __forceinline__ double
max_floor64(double x, double f)
{
  const unsigned long long b = (unsigned long long)__double_as_longlong(f);
  return (unsigned long long)__double_as_longlong(x) - b <= 0x7ff0000000000000ull - b ? x : f;
}
__device__ __forceinline__ double
min_pos64(double a, double b)
{
  return __longlong_as_double(min(__double_as_longlong(a), __double_as_longlong(b)));
}
// x with the sign flipped when f
__device__ __forceinline__ double
flip64(double x, bool f)
{
  return with_hi(hi32(x) ^ (f ? (int)0x80000000 : 0), x);
}
// integers in the order of the numbers, and back
__device__ __forceinline__ long long
order64(double x)
{
  const long long b = __double_as_longlong(x);
  return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
__device__ __forceinline__ double
from_order64(long long b)
{
  return __longlong_as_double(b ^ ((b >> 63) & 0x7fffffffffffffffll));
}
// |x| (fabs and unary minus can become FP64 additions)
__device__ __forceinline__ double
abs64(double x)
{
  return with_hi(hi32(x) & 0x7fffffff, x);
}
// x / 2 by the exponent; where that leaves the normal range, by a shift of the
// significand (exact but for the last subnormal bit, which is cut)
__device__ __forceinline__ double
half64(double x)
{
  const long long b = __double_as_longlong(x), m = b & 0x7fffffffffffffffll;
  const long long h = m >= 0x7ff0000000000000ll ? m : (m >= 0x0020000000000000ll ? m - 0x0010000000000000ll : m >> 1);
  return __longlong_as_double(h | (b ^ m));
}
// x / 2^K for x >= 0 by the exponent; zero below 2^(K - 1021)
template <int K>
__device__ __forceinline__ double
scale_pos64(double x)
{
  const int hi = hi32(x);
  const bool tiny = hi < ((K + 1) << 20);
  return __hiloint2double(tiny ? 0 : hi - (K << 20), tiny ? 0 : __double2loint(x));
}
// max(p, d floor) for d > 0: the product only where the high words say that
// p / d may be below 2 floor.  They are logarithms of positive normal p alone: a
// negative p, below any floor (also one of zero), takes the product always, and
// zero, a subnormal, infinity and NaN do.
__device__ __forceinline__ double
floor_ratio64(double p, double d, double floor)
{
  const int hp = hi32(p);
  if ((unsigned)(hp - 0x00100000) >= 0x7fe00000u || hp - hi32(d) < hi32(floor) - 0x3ff00000 + 0x00100000)
    p = max_floor64(p, d * floor);
  return p;
}
// running maximum of CFL candidates: NaN is ignored, as fmax does
__device__ __forceinline__ double
max_cand64(double m, double v)
{
  const long long b = __double_as_longlong(v);
  return b <= 0x7ff0000000000000ll ? __longlong_as_double(max(__double_as_longlong(m), b)) : m;
}
__device__ __forceinline__ float
max_cand(float m, float v)
{
  return fmaxf(m, v);
}
__device__ __forceinline__ double
max_cand(double m, double v)
{
  if constexpr (kShareRecip)
    return max_cand64(m, v);
  else
    return fmax(m, v);
}

// FP64 value in the working precision R
template <class R>
__device__ __forceinline__ R
to_r(double x)
{
  if constexpr (sizeof(R) == 4)
    return d2f_rn(x);
  else
    return x;
}

// Map a (possibly ghost) coordinate g in [0, n+2gw) of one dimension to the
// interior coordinate the boundary fill copies from; *flip is set when the
// reflecting wall flips the sign of the normal components.
__device__ __forceinline__ int
bc_map(int g, int n, int gw, int bc_lo, int bc_hi, bool * flip)
{
  // coordinates past the ghost layers only occur in the padding of partial
  // tiles; clamping keeps every read inside the array
  g = g < 0 ? 0 : (g > n + 2 * gw - 1 ? n + 2 * gw - 1 : g);
  if (g < gw)
  {
    if (bc_lo == BC_DIRICHLET)
    {
      *flip = !*flip;
      return 2 * gw - 1 - g;
    }
    if (bc_lo == BC_NEUMANN)
      return gw;
    return n + g;
  }
  if (g >= n + gw)
  {
    if (bc_hi == BC_DIRICHLET)
    {
      *flip = !*flip;
      return 2 * n + 2 * gw - 1 - g;
    }
    if (bc_hi == BC_NEUMANN)
      return n + gw - 1;
    return g - n;
  }
  return g;
}

// Source offset (in one variable plane) and per-dimension flips of a cell.
struct SrcCell
{
  long long off;
  bool      fx, fy, fz;
};

__device__ __forceinline__ SrcCell
src_cell(const KParams & P, int gi, int gj, int gk)
{
  SrcCell s;
  s.fx = s.fy = s.fz = false;
  int si = bc_map(gi, P.nx, P.gw, P.bc[0], P.bc[1], &s.fx);
  int sj = bc_map(gj, P.ny, P.gw, P.bc[2], P.bc[3], &s.fy);
  int sk = gk;
  if (P.ksize > 1)
    sk = bc_map(gk, P.nz, P.gw, P.bc[4], P.bc[5], &s.fz);
  s.off = (long long)sk * P.plane + (long long)sj * P.isize + si;
  return s;
}

// sign of variable v at a mapped cell: the reflecting fill multiplies the
// normal velocity (and, for MHD, the normal face field) by -1 per wall
__device__ __forceinline__ bool
flips(const SrcCell & s, int v, int mhd)
{
  bool f = false;
  if (v == IU || (mhd && v == IA))
    f ^= s.fx;
  if (v == IV || (mhd && v == IB))
    f ^= s.fy;
  if (v == IW || (mhd && v == IC))
    f ^= s.fz;
  return f;
}

// x or -x; the sign of a double is flipped with an integer XOR so that no
// FP64 instruction is issued (the result equals the FP64 negation bit for bit)
__device__ __forceinline__ double
neg_if(double x, bool f)
{
  return __longlong_as_double(__double_as_longlong(x) ^ (f ? (long long)0x8000000000000000ull : 0ll));
}
__device__ __forceinline__ float
neg_if(float x, bool f)
{
  return f ? -x : x;
}

template <class T>
__device__ __forceinline__ T
ldg(const T * p)
{
  return __ldg(p);
}

// Called by every block of the kernel that completes the CFL key of `step`
// (after its atomicMax): the last block to finish computes the step's dt and
// dt/dx ratios in FP64 once, for the step's kernels to read (step_consts), so
// that no block of those kernels runs the divisions behind a barrier.  The
// clock fields written by other blocks are read through volatile loads.
// repair: the HLLD repair pass's list, if any; when tiles are listed the pass
// completes the key, and computes the constants.  blocks: their number, where it
// is not the grid's.
__device__ __forceinline__ void
finalize_step(DevClock * clk, const KParams & P, int step, const int * repair = nullptr, unsigned blocks = 0)
{
  __shared__ int last;
  __syncthreads();
  const int s = step % 3;
  if (threadIdx.x == 0)
  {
    __threadfence();
    const unsigned nb = blocks ? blocks : gridDim.x * gridDim.y * gridDim.z;
    last = atomicAdd(&clk->fin[s], 1u) == nb - 1;
  }
  __syncthreads();
  if (last && threadIdx.x == 0)
  {
    __threadfence();
    volatile DevClock * v = clk;
    clk->fin[s] = 0;
    if (repair && *(const volatile int *)repair != 0)
      return;
    StepConsts c;
    c.step = step;
    c.active = 0;
    c.t = c.dt = c.dtdx = c.dtdy = c.dtdz = 0.0;
    // dt at the start of a step, SolverBase::compute_dt (SolverBase.cpp:124-154);
    // the step must not run when the simulation is finished (t >= tEnd - 1e-14,
    // SolverBase.cpp:170-176) or an earlier launched step did not run (its slot
    // was never committed)
    if (v->sid[s] == step)
    {
      const double invDt = dkey_inv(v->key[s]);
      double       d = P.cfl / invDt;
      const double tt = v->t[s];
      if (tt + d > P.tEnd)
        d = P.tEnd - tt;
      c.t = tt;
      c.dt = d;
      c.active = !(tt >= P.tEnd - 1e-14);
      c.dtdx = d / P.dx;
      c.dtdy = d / P.dy;
      c.dtdz = d / P.dz;
    }
    clk->sc[s] = c;
    clk->next = step;
  }
}
// The kernels of consecutive steps are launched with programmatic stream
// serialisation (launch_chained): once all blocks of a kernel have come to
// chain_next, or have ended, the blocks of the next one may become resident, and
// wait in chain_begin, before they touch memory, until the kernel has finished
// and its writes are visible.  chain_next stands where a block's work is done
// but for the reductions and the step's bookkeeping: called at the start, the
// waiting blocks took the slots of working ones (MHD 160^3 mixed 1095 -> 1473 us
// a step).  Without the launch attribute both instructions do nothing.
// Per step, unchained / chained: 2D hydro mixed 128^2 9.9 / 7.8 us, 2D MHD mixed
// 128^2 20.9 / 16.4, 3D hydro FP64 24^3 40.5 / 30.3, MHD mixed 32^3 49.9 / 43.7.
__device__ __forceinline__ void
chain_begin()
{
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void
chain_next()
{
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class... KA, class... A>
inline cudaError_t
launch_step_kernel(bool chained, void (*kernel)(KA...), dim3 grid, int threads, size_t smem, cudaStream_t st, A... args)
{
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = dim3((unsigned)threads);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = at;
  c.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&c, kernel, KA(args)...);
}
template <class... KA, class... A>
inline cudaError_t
launch_chained(void (*kernel)(KA...), dim3 grid, int threads, size_t smem, cudaStream_t st, A... args)
{
  return launch_step_kernel(true, kernel, grid, threads, smem, st, args...);
}
// A tile kernel whose time is a tile's (FP64) and that has one to three tiles
// per SM is not chained: the blocks brought in early crowd on the SMs that end
// first.  us per step by tiles per SM, unchained / chained: hydro 8 x 8, 1.1 18.6 /
// 17.6, 1.5 19.0 / 19.8, 1.7 19.7 / 22.3, 2.1 24.2 / 24.4, 2.6 24.4 / 26.8, 3.2 29.6 /
// 29.5; 16 x 16, 1.7 43.1 / 48.5, 2.1 59.6 / 57.2; MHD, 1.1 63.7 / 66.1, 1.7 63.7 /
// 85.8, 2.1 89.5 / 87.8, 2.6 90.1 / 99.9, 2.9 89.3 / 104.
inline bool
chain_tiles(const KParams & P, long long tiles)
{
  return tiles <= P.sms || tiles > 3ll * P.sms;
}

// the constants of `step`; false when the step must not run (or they were
// not computed for it).  Every step kernel begins with it.
__device__ __forceinline__ bool
step_consts(const DevClock * clk, int step, StepConsts & c)
{
  chain_begin();
  c = clk->sc[step % 3];
  return c.step == step && c.active;
}

// Visit the interior cells of a state row by row: a block takes whole rows
// (j, k) with a grid stride and its threads take the cells of a row, so the
// index math needs one 32-bit division per row (a per-cell 64-bit division is
// a long software sequence).  f(i, j, k) gets ghost-inclusive indices.
template <class F>
__device__ __forceinline__ void
for_interior_rows(const KParams & P, F && f)
{
  const int nrows = P.ny * (P.ksize > 1 ? P.nz : 1);
  for (int row = blockIdx.x; row < nrows; row += gridDim.x)
  {
    const int j = row % P.ny + P.gw;
    const int k = P.ksize > 1 ? row / P.ny + P.gw : 0;
    for (int i = threadIdx.x + P.gw; i < P.nx + P.gw; i += blockDim.x)
      f(i, j, k);
  }
}
// blocks for a row-wise pass over the interior
__host__ __device__ inline int
row_blocks(const KParams & P)
{
  const long long nrows = (long long)P.ny * (P.ksize > 1 ? P.nz : 1);
  return (int)(nrows < 8192 ? nrows : 8192);
}

// bookkeeping done once per step by block 0, thread 0
__device__ __forceinline__ void
step_commit(DevClock * clk, int step, double t, double dt)
{
  clk->t[(step + 1) % 3] = t + dt;
  clk->sid[(step + 1) % 3] = step + 1;
  clk->key[(step + 2) % 3] = EK_KEY_LOWEST;
  if (step < clk->dtcap)
    clk->dtlog[step] = dt;
  clk->last_dt = dt;
  clk->iteration = step + 1;
}

// block-wide max of a thread-local key, then one atomicMax per block
template <int NT>
__device__ __forceinline__ void
block_max_commit(unsigned long long local, unsigned long long * dst)
{
  __shared__ unsigned long long red[NT / 32];
  for (int o = 16; o > 0; o >>= 1)
  {
    unsigned long long other = __shfl_xor_sync(0xffffffffu, local, o);
    local = other > local ? other : local;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0)
    red[warp] = local;
  __syncthreads();
  if (warp == 0)
  {
    local = lane < NT / 32 ? red[lane] : 0ull;
    for (int o = 16; o > 0; o >>= 1)
    {
      unsigned long long other = __shfl_xor_sync(0xffffffffu, local, o);
      local = other > local ? other : local;
    }
    if (lane == 0)
      atomicMax(dst, local);
  }
}

// fmax semantics of the reference's reduction: a NaN candidate is ignored
__device__ __forceinline__ unsigned long long
cand_key(double v)
{
  // NaN by its bits (a comparison is an FP64-pipe instruction)
  return (__double_as_longlong(v) & 0x7fffffffffffffffll) > 0x7ff0000000000000ll ? 0ull : dkey(v);
}


// ---------------------------------------------------------------------------
// Tensor-memory-access (TMA) staging: one elected thread starts an
// asynchronous tiled copy global -> shared memory that completes on an
// mbarrier; the consumers wait on the barrier's phase.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned
smem_addr(const void * p)
{
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void
mbar_init(unsigned long long * bar, unsigned count)
{
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
  // make the initialised barrier visible to the tensor-copy (async) proxy
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// order this thread's earlier generic accesses of shared memory before the
// async-proxy writes of a tensor copy issued after it
__device__ __forceinline__ void
fence_proxy_async_smem()
{
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void
mbar_expect_tx(unsigned long long * bar, unsigned bytes)
{
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
// 4D tiled tensor copy of the box at (x, y, z, w) of *map into dst
__device__ __forceinline__ void
tma_load_4d(void * dst, const CUtensorMap * map, int x, int y, int z, int w, unsigned long long * bar)
{
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
               " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_addr(dst)),
               "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(z), "r"(w), "r"(smem_addr(bar))
               : "memory");
}
__device__ __forceinline__ unsigned long long
global_ns()
{
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// wait until phase `parity` of the barrier has completed; false when that
// has not happened within limit_ns (the caller reports the error and leaves)
__device__ __forceinline__ bool
mbar_wait(unsigned long long * bar, unsigned parity, unsigned long long limit_ns)
{
  const unsigned addr = smem_addr(bar);
  unsigned long long t0 = 0;
  for (int n = 0;; ++n)
  {
    unsigned done;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(done)
                 : "r"(addr), "r"(parity)
                 : "memory");
    if (done)
      return true;
    const unsigned long long t = global_ns();
    if (n == 0)
      t0 = t;
    else if (t - t0 > limit_ns)
      return false;
  }
}


// Per-thread asynchronous copies global -> shared memory (element gathers
// whose source addresses follow the boundary mapping); completion is waited
// for by the issuing thread (cp.async.wait_all) before a block barrier.
template <int BYTES>
__device__ __forceinline__ void
cp_async(void * dst, const void * src)
{
  static_assert(BYTES == 4 || BYTES == 8, "cp.async element size");
  if constexpr (BYTES == 4)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void
cp_async_commit()
{
  asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void
cp_async_wait_all()
{
  asm volatile("cp.async.wait_all;" ::: "memory");
}

} // namespace EK_NS
