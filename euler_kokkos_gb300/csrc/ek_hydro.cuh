// Hydro cell/face arithmetic of the unsplit MUSCL-Hancock step, written for
// one cell or one face so the fused kernels can call it on shared-memory
// tiles.  Every expression keeps the evaluation order of the reference so the
// FP64 build compiled without FMA contraction reproduces it bit for bit; the
// cited reference lines define the arithmetic.
#pragma once

#include "ek_common.cuh"

namespace EK_NS
{

template <class R>
struct HydroConst
{
  R gamma0, smallr, smallp, smallc, slope_type, gamma6, smallpp;
  R entho; // 1 / (gamma0 - 1), the value every Riemann solver of the reference computes
};


// slope_unsplit_hydro_3d_scalar, one direction (HydroBaseFunctor3D.h:413-462,
// HydroBaseFunctor2D.h:423-453): minmod (slope_type 1) / MC (slope_type 2)
template <class R>
__device__ __forceinline__ R
slope1(R q, R qp, R qm, R st)
{
  if constexpr (sizeof(R) == 4)
  {
    // the same limiter, FP32 form (signed zeros may differ).  st is 0, 1 or
    // 2, so scaling by it is exact and min(|st dl|, |st dr|) = st min(|dl|,
    // |dr|) (0 for first order).
    // Where dl and dr have one sign, so has dcen, and |dcen| >= min(|dl|,
    // |dr|) after rounding too (rounding is monotonic): with st = 1 (minmod)
    // the centred difference never binds.
    const float dl = q - qm, dr = qp - q;
    float       m = st * fminf(fabsf(dl), fabsf(dr));
    if (st != 1.f)
      m = fminf(m, fabsf(0.5f * (qp - qm)));
    return (dl * dr > 0.f) ? copysignf(m, dl) : 0.f;
  }
  const R dlft = st * (q - qm);
  const R drgt = st * (qp - q);
  const R dcen = R(0.5) * (qp - qm);
  const R dsgn = (dcen >= R(0)) ? R(1) : R(-1);
  const R slop = fmin(fabs(dlft), fabs(drgt));
  R       dlim = slop;
  if ((dlft * drgt) <= R(0))
    dlim = R(0);
  return dsgn * fmin(dlim, fabs(dcen));
}

// Two slopes at once in packed FP32 (slope1's FP32 form, lane by lane).
__device__ __forceinline__ float2
slope2(float2 q, float2 qp, float2 qm, float st)
{
  const float2 dl = sub2(q, qm), dr = sub2(qp, q), pr = mul2(dl, dr);
  float2       m = f2(fminf(fabsf(dl.x), fabsf(dr.x)), fminf(fabsf(dl.y), fabsf(dr.y)));
  if (st != 1.f)
  {
    const float2 dc = mul2(f2s(0.5f), sub2(qp, qm));
    m = mul2(f2s(st), m);
    m = f2(fminf(m.x, fabsf(dc.x)), fminf(m.y, fabsf(dc.y)));
  }
  return f2(pr.x > 0.f ? copysignf(m.x, dl.x) : 0.f, pr.y > 0.f ? copysignf(m.y, dl.y) : 0.f);
}

// Half of slope1's slope, for the FP64 FMA build: every use of a slope takes
// its half.  Two differences on the FP64 pipe (three for MC); the minima, the
// scaling by powers of two and the signs on the integer pipes.  A slope is
// zero where dl and dr differ in sign or either is zero, and, as the
// reference's test dl dr <= 0 has it, where their product underflows; with st =
// 1 (minmod) the centred difference never binds (see the FP32 form above).
__device__ __forceinline__ double
half_slope64(double q, double qp, double qm, double st)
{
  const double dl = q - qm, dr = qp - q;
  const double m = min_pos64(abs64(dl), abs64(dr));
  double       h;
  const int    lim = hi32(st); // 1.0 or 2.0 by the high word: a comparison would be an FP64 instruction
  if (lim == 0x3ff00000)
    h = scale_pos64<1>(m);
  else if (lim == 0x40000000)
    h = min_pos64(m, scale_pos64<2>(abs64(qp - qm)));
  else
    h = 0.0;
  // the sign of dl, or zero
  const int      sl = hi32(dl), sr = hi32(dr);
  const unsigned e2 = (unsigned)(sl & 0x7fffffff) + (unsigned)(sr & 0x7fffffff); // log2 |dl dr| + 2046, x 2^20
  const bool     zero = (sl ^ sr) < 0 || e2 < (970u << 20);
  return __hiloint2double((zero ? 0 : hi32(h)) | (sl & (int)0x80000000), zero ? 0 : __double2loint(h));
}
// the slope, or its half in the FP64 FMA build (kFast64)
template <class R>
__device__ __forceinline__ R
slope_h(R q, R qp, R qm, R st)
{
  if constexpr (kFast64<R>)
    return half_slope64(q, qp, qm, st);
  else
    return slope1<R>(q, qp, qm, st);
}

// Slopes of all variables.  The mixed form's 3D kernel, bound by issue, takes (rho,
// p) and (u, v) as packed pairs here, in the sources and in the face states
// (256^3 680 -> 665 us); the 2D march gains nothing from it.
template <class R, int NV>
__device__ __forceinline__ void
slopes_h(const R (&q)[NV], const R (&qp)[NV], const R (&qm)[NV], R st, R (&d)[NV])
{
  if constexpr (sizeof(R) == 4 && NV == 5)
  {
#pragma unroll
    for (int v = 0; v < 4; v += 2)
    {
      const float2 s = slope2(f2(q[v], q[v + 1]), f2(qp[v], qp[v + 1]), f2(qm[v], qm[v + 1]), st);
      d[v] = s.x;
      d[v + 1] = s.y;
    }
    d[4] = slope_h<R>(q[4], qp[4], qm[4], st);
  }
  else
  {
#pragma unroll
    for (int v = 0; v < NV; ++v)
      d[v] = slope_h<R>(q[v], qp[v], qm[v], st);
  }
}

// computePrimitives (HydroBaseFunctor2D.h:78-102, HydroBaseFunctor3D.h:80-106).
// In the mixed form (R = float) the internal energy is recomputed in FP64
// when E/rho and the kinetic energy cancel to fewer than ~7 significant bits.
template <class R, int NV>
__device__ __forceinline__ void
hydro_prims(const R (&u)[NV], R (&q)[NV], const HydroConst<R> & C)
{
  if constexpr (kFast64<R>)
  {
    // FP64 FMA build: p = (gamma - 1) (E - rho v^2 / 2), 12 FP64-pipe operations in 3D
    const R d = max_floor64(u[ID], C.smallr), id = rcp64(d);
    q[ID] = d;
    q[IU] = u[IU] * id;
    q[IV] = u[IV] * id;
    R k = q[IU] * q[IU] + q[IV] * q[IV];
    if constexpr (NV == 5)
    {
      q[IW] = u[IW] * id;
      k += q[IW] * q[IW];
    }
    q[IP] = floor_ratio64((C.gamma0 - R(1)) * fma(R(-0.5) * d, k, u[IP]), d, C.smallp);
    return;
  }
  const R d = fmax(u[ID], C.smallr);
  // one reciprocal of the density for the four quotients (FP32: approximate;
  // FP64 exact build: four divisions)
  R id = R(0);
  if constexpr (sizeof(R) == 4)
    id = rcp_a(d);
  auto over_d = [&](R x) {
    if constexpr (sizeof(R) == 4)
      return x * id;
    else
      return x / d;
  };
  const R ux = over_d(u[IU]);
  const R uy = over_d(u[IV]);
  R       eken, uz = R(0);
  if constexpr (NV == 4)
    eken = R(0.5) * (ux * ux + uy * uy);
  else
  {
    uz = over_d(u[IW]);
    eken = R(0.5) * (ux * ux + uy * uy + uz * uz);
  }
  const R ed = over_d(u[IP]);
  R       e = ed - eken;
  if constexpr (sizeof(R) == 4)
  {
    if (e < R(1.0 / 128.0) * ed)
    {
      // FP64 island: cancellation between total and kinetic energy
      const double dd = (double)d;
      const double vx = (double)u[IU] / dd, vy = (double)u[IV] / dd;
      double       ek = vx * vx + vy * vy;
      if constexpr (NV == 5)
      {
        const double vz = (double)u[IW] / dd;
        ek += vz * vz;
      }
      e = (R)((double)u[IP] / dd - 0.5 * ek);
    }
  }
  const R p = fmax((C.gamma0 - R(1)) * d * e, d * C.smallp);
  q[ID] = d;
  q[IP] = p;
  q[IU] = ux;
  q[IV] = uy;
  if constexpr (NV == 5)
    q[IW] = uz;
}

// sound speed as computePrimitives computes it: sqrt(gamma0 * p / d)
template <class R>
__device__ __forceinline__ R
hydro_sound(R d, R p, const HydroConst<R> & C)
{
  if constexpr (sizeof(R) == 4)
    return sqrt_a(C.gamma0 * p * rcp_a(d));
  else if constexpr (kFast64<R>)
    return sqrt_ratio64(C.gamma0 * p, d);
  else
    return sqrt(C.gamma0 * (p) / d);
}

// Per-cell source terms of trace_unsplit_{2d,3d}_along_dir
// (HydroBaseFunctor2D.h:250-253, HydroBaseFunctor3D.h:321-325).  They do not
// depend on the face, so they are computed once per cell.
template <class R, int NV>
__device__ __forceinline__ void
hydro_sources(const R (&q)[NV], const R (&dx)[NV], const R (&dy)[NV], const R (&dz)[NV], R (&s)[NV],
              const HydroConst<R> & C)
{
  const R r = q[ID], p = q[IP], u = q[IU], v = q[IV];
  if constexpr (kFast64<R>)
  {
    // FP64 FMA build, from half slopes (so half the sources): one FMA chain each
    const R ir = rcp64(r), gp = C.gamma0 * p;
    R       div = dx[IU] + dy[IV];
    if constexpr (NV == 5)
      div += dz[IW];
    auto adv = [&](int f, R x) { // x - v . grad f
      x = fma(-v, dy[f], fma(-u, dx[f], x));
      if constexpr (NV == 5)
        x = fma(-q[IW], dz[f], x);
      return x;
    };
    s[ID] = adv(ID, -div * r);
    s[IP] = adv(IP, -div * gp);
    s[IU] = adv(IU, -dx[IP] * ir);
    s[IV] = adv(IV, -dy[IP] * ir);
    if constexpr (NV == 5)
      s[IW] = adv(IW, -dz[IP] * ir);
    return;
  }
  if constexpr (sizeof(R) == 4 && NV == 5)
  {
    // packed pairs (slopes_h)
    const float  w = q[IW], ir = rcp_a(r), div = dx[IU] + dy[IV] + dz[IW];
    const float2 mu = f2s(-u), mv = f2s(-v), mw = f2s(-w);
    const float2 rp = fma2(mw, f2(dz[ID], dz[IP]), fma2(mv, f2(dy[ID], dy[IP]), mul2(mu, f2(dx[ID], dx[IP]))));
    const float2 uv = fma2(mw, f2(dz[IU], dz[IV]), fma2(mv, f2(dy[IU], dy[IV]), mul2(mu, f2(dx[IU], dx[IV]))));
    const float2 a = fma2(f2s(-div), f2(r, C.gamma0 * p), rp), b = fma2(f2s(-ir), f2(dx[IP], dy[IP]), uv);
    s[ID] = a.x, s[IP] = a.y, s[IU] = b.x, s[IV] = b.y;
    s[IW] = -u * dx[IW] - v * dy[IW] - w * dz[IW] - dz[IP] * ir;
    return;
  }
  R ir = R(0);
  if constexpr (sizeof(R) == 4)
    ir = rcp_a(r);
  auto over_r = [&](R x) {
    if constexpr (sizeof(R) == 4)
      return x * ir;
    else
      return x / r;
  };
  if constexpr (NV == 4)
  {
    s[ID] = -u * dx[ID] - v * dy[ID] - (dx[IU] + dy[IV]) * r;
    s[IP] = -u * dx[IP] - v * dy[IP] - (dx[IU] + dy[IV]) * C.gamma0 * p;
    s[IU] = -u * dx[IU] - v * dy[IU] - over_r(dx[IP]);
    s[IV] = -u * dx[IV] - v * dy[IV] - over_r(dy[IP]);
  }
  else
  {
    const R w = q[IW];
    s[ID] = -u * dx[ID] - v * dy[ID] - w * dz[ID] - (dx[IU] + dy[IV] + dz[IW]) * r;
    s[IP] = -u * dx[IP] - v * dy[IP] - w * dz[IP] - (dx[IU] + dy[IV] + dz[IW]) * C.gamma0 * p;
    s[IU] = -u * dx[IU] - v * dy[IU] - w * dz[IU] - over_r(dx[IP]);
    s[IV] = -u * dx[IV] - v * dy[IV] - w * dz[IV] - over_r(dy[IP]);
    s[IW] = -u * dx[IW] - v * dy[IW] - w * dz[IW] - over_r(dz[IP]);
  }
}

// face state of trace_unsplit_*_along_dir: q -/+ dq/2 + s*dtdx/2, rho floored
// (HydroBaseFunctor3D.h:327-365); sgn = -1 for the MIN face, +1 for MAX
template <class R, int NV>
__device__ __forceinline__ void
hydro_face(const R (&q)[NV], const R (&d)[NV], const R (&s)[NV], R dtd, bool plus, R (&f)[NV],
           R smallr)
{
  if constexpr (sizeof(R) == 4)
  {
    // mixed form: two fused multiply-adds per variable, in 3D per pair (slopes_h)
    const R       hdtd = R(0.5) * dtd, hd = plus ? R(0.5) : R(-0.5);
    constexpr int first = NV == 5 ? 4 : 0;
    if constexpr (NV == 5)
    {
#pragma unroll
      for (int v = 0; v < 4; v += 2)
      {
        const float2 x = fma2(f2s(hd), f2(d[v], d[v + 1]), fma2(f2(s[v], s[v + 1]), f2s(hdtd), f2(q[v], q[v + 1])));
        f[v] = x.x;
        f[v + 1] = x.y;
      }
    }
#pragma unroll
    for (int v = first; v < NV; ++v)
      f[v] = fma(hd, d[v], fma(s[v], hdtd, q[v]));
  }
  else
  {
#pragma unroll
    for (int v = 0; v < NV; ++v)
    {
      if (plus)
        f[v] = q[v] + R(0.5) * d[v] + s[v] * dtd * R(0.5);
      else
        f[v] = q[v] - R(0.5) * d[v] + s[v] * dtd * R(0.5);
    }
  }
  f[ID] = fmax(smallr, f[ID]);
}

// The face states of one cell.  In the FP64 FMA build slopes and sources are
// halves and the time-advanced state q + s dt/dx is computed once for all
// directions whose dt/dx is the same.
template <class R, int NV>
struct FaceStates
{
  const R (&q)[NV], (&s)[NV];
  R dtd, smallr;
  R b[kFast64<R> ? NV : 1];
  __device__ __forceinline__
  FaceStates(const R (&q_)[NV], const R (&s_)[NV], R dtd_, R smallr_)
    : q(q_), s(s_), smallr(smallr_)
  {
    set(dtd_);
  }
  __device__ __forceinline__ void
  set(R dtd_)
  {
    dtd = dtd_;
    if constexpr (kFast64<R>)
    {
#pragma unroll
      for (int v = 0; v < NV; ++v)
        b[v] = fma(s[v], dtd, q[v]);
    }
  }
  // the next direction; same: its dt/dx is the present one
  __device__ __forceinline__ void
  turn(R dtd_, bool same)
  {
    if (!kFast64<R> || !same)
      set(dtd_);
  }
  __device__ __forceinline__ void
  get(const R (&d)[NV], bool plus, R (&f)[NV]) const
  {
    if constexpr (kFast64<R>)
    {
#pragma unroll
      for (int v = 0; v < NV; ++v)
        f[v] = plus ? b[v] + d[v] : b[v] - d[v];
      f[ID] = max_floor64(f[ID], smallr);
    }
    else
      hydro_face<R, NV>(q, d, s, dtd, plus, f, smallr);
  }
};

// Face fluxes are kept scaled by dt/dx, as the reference stores them; the FP64
// FMA build keeps them unscaled and scales in the update's FMAs.
template <class R>
__device__ __forceinline__ R
flux_scaled(R f, R dtd)
{
  if constexpr (sizeof(R) == 4)
    return __fmul_rn(f, dtd); // rounded: both cells of a face take the same value, whichever code adds it
  else
    return kFast64<R> ? f : f * dtd;
}
template <class R>
__device__ __forceinline__ R
add_flux(R x, R f, R dtd)
{
  return kFast64<R> ? fma(f, dtd, x) : x + f;
}
template <class R>
__device__ __forceinline__ R
sub_flux(R x, R f, R dtd)
{
  return kFast64<R> ? fma(-f, dtd, x) : x - f;
}

// riemann_hllc (RiemannSolvers.h:445-568) in the FP64 FMA build: the same star
// state with about 51 FP64-pipe operations per 3D face.  The larger sound speed is one reciprocal square
// root (densities are positive: p_l / rho_l >= p_r / rho_r where p_l rho_r >=
// p_r rho_l).  With w = (p_l - p_r - rc_r (u_l - u_r)) / (rc_l + rc_r), u* = u_l
// + w and p* = p_l - rc_l w; rc = rho |S - u| is also the star density's
// numerator.  The four-way choice is by sign bits and selects (integer pipes).
// With the half slopes and the FMA updates: FP64 2D step 74.3 -> 52.1 us at
// 256^2, two-shock 3D step 2224 -> 1287 us at 33 x 31 x 99.
template <int NV>
__device__ __forceinline__ void
hllc64(const double (&ql)[NV], const double (&qr)[NV], double (&flux)[NV], const HydroConst<double> & C)
{
  const double rl = max_floor64(ql[ID], C.smallr), rr = max_floor64(qr[ID], C.smallr);
  const double pl = floor_ratio64(ql[IP], rl, C.smallp), pr = floor_ratio64(qr[IP], rr, C.smallp);
  const double ul = ql[IU], ur = qr[IU];
  double       kl = ul * ul + ql[IV] * ql[IV], kr = ur * ur + qr[IV] * qr[IV];
  if constexpr (NV == 5)
  {
    kl += ql[IW] * ql[IW];
    kr += qr[IW] * qr[IW];
  }
  const double el = fma(pl, C.entho, scale_pos64<1>(rl) * kl), er = fma(pr, C.entho, scale_pos64<1>(rr) * kr);

  const double cmax = max_floor64(sqrt_larger_ratio64(C.gamma0 * pl, rl, C.gamma0 * pr, rr), C.smallc);

  const double du = ul - ur;
  const bool   lslow = negative64(du); // ul < ur
  const double SL = (lslow ? ul : ur) - cmax, SR = (lslow ? ur : ul) + cmax;
  const double al = ul - SL, ar = SR - ur;
  const double rcl = rl * al, rcr = rr * ar;
  const double w = fma(-rcr, du, pl - pr) * rcp64(rcr + rcl);
  const double us = ul + w, ps = fma(-rcl, w, pl);

  // the star state on the side of the contact (left when u* > 0), or the left
  // state's own side when its wave is the one sampled: without a sound speed the
  // star state of an expansion is 0 / 0
  const bool   left = positive64(us) || positive64(SL);
  const double Sk = left ? SL : SR, uk = left ? ul : ur, ek = left ? el : er, pk = left ? pl : pr;
  const double is = rcp64(Sk - us);
  const double rs = (left ? flip64(rcl, true) : rcr) * is;
  const double es = fma(ps, us, fma(-pk, uk, (left ? flip64(al, true) : ar) * ek)) * is;
  const bool   out = left ? positive64(SL) : !positive64(SR); // supersonic: the side's own state
  const double ro = out ? (left ? rl : rr) : rs, uo = out ? uk : us, po = out ? pk : ps, eo = out ? ek : es;

  const double m = ro * uo;
  const bool   ml = positive64(m);
  flux[ID] = m;
  flux[IU] = fma(m, uo, po);
  flux[IP] = (eo + po) * uo;
  flux[IV] = m * (ml ? ql[IV] : qr[IV]);
  if constexpr (NV == 5)
    flux[IW] = m * (ml ? ql[IW] : qr[IW]);
}

// riemann_hllc (RiemannSolvers.h:445-568).  States are in the face frame
// (normal velocity in IU); NV = 4 (2D) or 5 (3D).
template <class R, int NV>
__device__ __forceinline__ void
hllc(const R (&ql)[NV], const R (&qr)[NV], R (&flux)[NV], const HydroConst<R> & C)
{
  if constexpr (kFast64<R>)
  {
    hllc64<NV>(ql, qr, flux, C);
    return;
  }
  const R entho = C.entho;
  R       rl, pl, ul, etotl, rr, pr, ur, etotr, cmax; // cmax: the larger sound speed
  if constexpr (sizeof(R) == 4)
  {
    // mixed form: the two states in the lanes of packed FP32 pairs
    const float2 r = f2(fmaxf(ql[ID], C.smallr), fmaxf(qr[ID], C.smallr));
    const float2 ps = mul2(r, f2s(C.smallp));
    const float2 p = f2(fmaxf(ql[IP], ps.x), fmaxf(qr[IP], ps.y));
    const float2 u = f2(ql[IU], qr[IU]), v = f2(ql[IV], qr[IV]);
    float2       k2 = fma2(v, v, mul2(u, u));
    if constexpr (NV == 5)
      k2 = fma2(f2(ql[IW], qr[IW]), f2(ql[IW], qr[IW]), k2);
    const float2 etot = fma2(p, f2s(entho), mul2(mul2(f2s(0.5f), r), k2));
    const float2 c2 = mul2(mul2(f2s(C.gamma0), p), f2(rcp_a(r.x), rcp_a(r.y)));
    const float  sc2 = C.smallc * C.smallc;
    rl = r.x, pl = p.x, ul = u.x, etotl = etot.x;
    rr = r.y, pr = p.y, ur = u.y, etotr = etot.y;
    cmax = sqrt_a(fmaxf(fmaxf(c2.x, c2.y), sc2));
  }
  else
  {
    rl = fmax(ql[ID], C.smallr);
    pl = fmax(ql[IP], rl * C.smallp);
    ul = ql[IU];
    R ecinl = R(0.5) * rl * ul * ul;
    ecinl += R(0.5) * rl * ql[IV] * ql[IV];
    if constexpr (NV == 5)
      ecinl += R(0.5) * rl * ql[IW] * ql[IW];
    etotl = pl * entho + ecinl;

    rr = fmax(qr[ID], C.smallr);
    pr = fmax(qr[IP], rr * C.smallp);
    ur = qr[IU];
    R ecinr = R(0.5) * rr * ur * ur;
    ecinr += R(0.5) * rr * qr[IV] * qr[IV];
    if constexpr (NV == 5)
      ecinr += R(0.5) * rr * qr[IW] * qr[IW];
    etotr = pr * entho + ecinr;

    cmax = fmax(sqrt(fmax(C.gamma0 * pl / rl, C.smallc * C.smallc)),
                sqrt(fmax(C.gamma0 * pr / rr, C.smallc * C.smallc)));
  }
  const R ptotl = pl, ptotr = pr;

  const R SL = fmin(ul, ur) - cmax;
  const R SR = fmax(ul, ur) + cmax;

  const R rcl = rl * (ul - SL);
  const R rcr = rr * (SR - ur);

  R ustar, ptotstar;
  if constexpr (sizeof(R) == 4)
  {
    const float irc = rcp_a(rcr + rcl);
    ustar = (rcr * ur + rcl * ul + (ptotl - ptotr)) * irc;
    ptotstar = (rcr * ptotl + rcl * ptotr + rcl * rcr * (ul - ur)) * irc;
  }
  else
  {
    ustar = (rcr * ur + rcl * ul + (ptotl - ptotr)) / (rcr + rcl);
    ptotstar = (rcr * ptotl + rcl * ptotr + rcl * rcr * (ul - ur)) / (rcr + rcl);
  }

  R ro, uo, ptoto, etoto;
  if constexpr (sizeof(R) == 4)
  {
    // FP32: the reference's four-way choice without branches -- the star
    // state is formed once, on the side of the contact (left when ustar > 0)
    const bool  left = ustar > 0.f;
    const float Sk = left ? SL : SR, rk = left ? rl : rr, uk = left ? ul : ur;
    const float ek = left ? etotl : etotr, pk = left ? ptotl : ptotr;
    const float is = rcp_a(Sk - ustar);
    const float rs = rk * (Sk - uk) * is;
    const float es = ((Sk - uk) * ek - pk * uk + ptotstar * ustar) * is;
    const bool  cL = SL > 0.f;                       // left state
    const bool  cR = !cL && !left && !(SR > 0.f);    // right state
    ro = cL ? rl : (cR ? rr : rs);
    uo = cL ? ul : (cR ? ur : ustar);
    ptoto = cL ? ptotl : (cR ? ptotr : ptotstar);
    etoto = cL ? etotl : (cR ? etotr : es);
  }
  else if (SL > R(0))
  {
    ro = rl;
    uo = ul;
    ptoto = ptotl;
    etoto = etotl;
  }
  else if (ustar > R(0))
  {
    uo = ustar;
    ptoto = ptotstar;
    ro = rl * (SL - ul) / (SL - ustar);
    etoto = ((SL - ul) * etotl - ptotl * ul + ptotstar * ustar) / (SL - ustar);
  }
  else if (SR > R(0))
  {
    uo = ustar;
    ptoto = ptotstar;
    ro = rr * (SR - ur) / (SR - ustar);
    etoto = ((SR - ur) * etotr - ptotr * ur + ptotstar * ustar) / (SR - ustar);
  }
  else
  {
    ro = rr;
    uo = ur;
    ptoto = ptotr;
    etoto = etotr;
  }
  flux[ID] = ro * uo;
  flux[IU] = ro * uo * uo + ptoto;
  flux[IP] = (etoto + ptoto) * uo;
  flux[IV] = flux[ID] * ((flux[ID] > R(0)) ? ql[IV] : qr[IV]);
  if constexpr (NV == 5)
    flux[IW] = flux[ID] * ((flux[ID] > R(0)) ? ql[IW] : qr[IW]);
}

// cmpflx (RiemannSolvers.h:20-53): flux of a Godunov state
template <class R, int NV>
__device__ __forceinline__ void
cmpflx(const R (&qg)[NV], R (&flux)[NV], const HydroConst<R> & C)
{
  flux[ID] = qg[ID] * qg[IU];
  flux[IU] = flux[ID] * qg[IU] + qg[IP];
  flux[IV] = flux[ID] * qg[IV];
  if constexpr (NV == 5)
    flux[IW] = flux[ID] * qg[IW];
  const R entho = C.entho;
  R       ekin = R(0.5) * qg[ID] * (qg[IU] * qg[IU] + qg[IV] * qg[IV]);
  if constexpr (NV == 5)
    ekin += R(0.5) * qg[ID] * (qg[IW] * qg[IW]);
  const R etot = qg[IP] * entho + ekin;
  flux[IP] = qg[IU] * (etot + qg[IP]);
}

// riemann_approx (RiemannSolvers.h:60-200) in the FP64 FMA build: a Newton
// iteration takes four reciprocals and reciprocal square roots (about 45
// FP64-pipe operations) instead of eight divisions and two square roots: with
// x = c (1 + gamma6 (p - p_k) / p_k), w = x rsqrt(x) and the shock velocity's
// quotient by w is a product with rsqrt(x).
template <int NV>
__device__ __forceinline__ void
riemann_approx64(const double (&ql)[NV], const double (&qr)[NV], double (&flux)[NV], const HydroConst<double> & C)
{
  const double rl = max_floor64(ql[ID], C.smallr), ul = ql[IU], pl = floor_ratio64(ql[IP], rl, C.smallp);
  const double rr = max_floor64(qr[ID], C.smallr), ur = qr[IU], pr = floor_ratio64(qr[IP], rr, C.smallp);
  const double cl = C.gamma0 * pl * rl, cr = C.gamma0 * pr * rr;
  // c gamma6 / p = gamma0 gamma6 rho
  const double kl = C.gamma0 * C.gamma6 * rl, kr = C.gamma0 * C.gamma6 * rr;
  const double du = ul - ur;
  double       wl = sqrt64(cl), wr = sqrt64(cr);
  double       p = max_floor64(fma(wl * wr, du, fma(wr, pl, wl * pr)) * rcp64(wl + wr), 0.0);
  double       yl, yr;
  for (int iter = 0;; ++iter)
  {
    const double dl = p - pl, dr = p - pr;
    const double xl = fma(kl, dl, cl), xr = fma(kr, dr, cr);
    yl = rsqrt64(xl);
    yr = rsqrt64(xr);
    wl = xl * yl;
    wr = xr * yr;
    if (iter == 10)
      break;
    // q = 2 w^3 / (w^2 + c)
    const double gl = xl * wl * rcp64(xl + cl), gr = xr * wr * rcp64(xr + cr);
    const double dv = fma(-dr, yr, fma(-dl, yl, du)); // u_l* - u_r*
    double       delp = (gr + gr) * gl * rcp64(gr + gl) * dv;
    delp = negative64(delp + p) ? flip64(p, true) : delp;
    p += delp;
    // |delp / (p + smallpp)| > 1e-6
    if (__double_as_longlong(abs64(delp)) <= __double_as_longlong(abs64((p + C.smallpp) * 1e-6)))
    {
      const double x2l = fma(kl, p - pl, cl), x2r = fma(kr, p - pr, cr);
      yl = rsqrt64(x2l);
      yr = rsqrt64(x2r);
      wl = x2l * yl;
      wr = x2r * yr;
      break;
    }
  }
  const double us = 0.5 * (ul + ur + fma(pl - p, yl, -((pr - p) * yr)));
  const bool   left = !negative64(us);
  const double ro = left ? rl : rr, po = left ? pl : pr, wo = left ? wl : wr, yo = left ? yl : yr;
  const double uo = flip64(left ? ul : ur, !left), ss = flip64(us, !left); // sgnm u
  const double co = max_floor64(sqrt_ratio64(abs64(C.gamma0 * po), ro), C.smallc);
  // rho / (1 + rho (p_o - p*) / w^2)
  const double rs = max_floor64(ro * rcp64(fma(ro * (po - p), yo * yo, 1.0)), C.smallr);
  const double cs = max_floor64(sqrt_ratio64(abs64(C.gamma0 * p), rs), C.smallc);
  double       spout = co - uo, spin = cs - ss;
  if (p >= po)
    spin = spout = fma(wo, rcp64(ro), -uo); // shock
  const double sum = spout + spin;
  const double scr = fmax(spout - spin, C.smallc + fabs(sum));
  double       frac = fma(0.5 * sum, rcp64(scr), 0.5);
  frac = frac != frac ? 0.0 : (frac >= 1.0 ? 1.0 : (frac <= 0.0 ? 0.0 : frac));
  double qg[NV];
  qg[ID] = fma(frac, rs - ro, ro);
  qg[IU] = fma(frac, us - (left ? ul : ur), left ? ul : ur);
  qg[IP] = fma(frac, p - po, po);
  if (negative64(spout))
    qg[ID] = ro, qg[IU] = left ? ul : ur, qg[IP] = po;
  if (positive64(spin))
    qg[ID] = rs, qg[IU] = us, qg[IP] = p;
  qg[IV] = left ? ql[IV] : qr[IV];
  if constexpr (NV == 5)
    qg[IW] = left ? ql[IW] : qr[IW];
  cmpflx<double, NV>(qg, flux, C);
}

// riemann_approx (RiemannSolvers.h:60-200): two-shock iterative solver,
// at most 10 Newton iterations on p*
template <class R, int NV>
__device__ __forceinline__ void
riemann_approx(const R (&ql)[NV], const R (&qr)[NV], R (&flux)[NV], const HydroConst<R> & C)
{
  if constexpr (kFast64<R>)
  {
    riemann_approx64<NV>(ql, qr, flux, C);
    return;
  }
  const R gamma0 = C.gamma0, gamma6 = C.gamma6, smallr = C.smallr, smallc = C.smallc, smallp = C.smallp;
  const R rl = fmax(ql[ID], smallr), ul = ql[IU], pl = fmax(ql[IP], rl * smallp);
  const R rr = fmax(qr[ID], smallr), ur = qr[IU], pr = fmax(qr[IP], rr * smallp);
  const R cl = gamma0 * pl * rl;
  const R cr = gamma0 * pr * rr;
  R       wl = sqrt(cl);
  R       wr = sqrt(cr);
  R       pstar = fmax(((wr * pl + wl * pr) + wl * wr * (ul - ur)) / (wl + wr), R(0));
  R       pold = pstar;
  R       conv = R(1);
  for (int iter = 0; (iter < 10) && (conv > R(1e-6)); ++iter)
  {
    const R wwl = sqrt(cl * (R(1) + gamma6 * (pold - pl) / pl));
    const R wwr = sqrt(cr * (R(1) + gamma6 * (pold - pr) / pr));
    const R qql = R(2) * wwl * wwl * wwl / (wwl * wwl + cl);
    const R qqr = R(2) * wwr * wwr * wwr / (wwr * wwr + cr);
    const R usl = ul - (pold - pl) / wwl;
    const R usr = ur + (pold - pr) / wwr;
    const R delp = fmax(qqr * qql / (qqr + qql) * (usl - usr), -pold);
    pold = pold + delp;
    conv = fabs(delp / (pold + C.smallpp));
  }
  pstar = pold;
  wl = sqrt(cl * (R(1) + gamma6 * (pstar - pl) / pl));
  wr = sqrt(cr * (R(1) + gamma6 * (pstar - pr) / pr));
  const R ustar = R(0.5) * (ul + (pl - pstar) / wl + ur - (pr - pstar) / wr);
  const R sgnm = copysign(R(1), ustar);
  R       ro, uo, po, wo;
  if (sgnm > R(0))
    ro = rl, uo = ul, po = pl, wo = wl;
  else
    ro = rr, uo = ur, po = pr, wo = wr;
  const R co = fmax(smallc, sqrt(fabs(gamma0 * po / ro)));
  const R rstar = fmax(R(ro / (R(1) + ro * (po - pstar) / (wo * wo))), smallr);
  const R cstar = fmax(smallc, sqrt(fabs(gamma0 * pstar / rstar)));
  R       spout = co - sgnm * uo;
  R       spin = cstar - sgnm * ustar;
  const R ushock = wo / ro - sgnm * uo;
  if (pstar >= po)
  {
    spin = ushock;
    spout = ushock;
  }
  const R scr = fmax(spout - spin, smallc + fabs(spout + spin));
  R       frac = R(0.5) * (R(1) + (spout + spin) / scr);
  if (frac != frac)
    frac = R(0);
  else
    frac = frac >= R(1) ? R(1) : frac <= R(0) ? R(0) : frac;
  R qg[NV];
  qg[ID] = frac * rstar + (R(1) - frac) * ro;
  qg[IU] = frac * ustar + (R(1) - frac) * uo;
  qg[IP] = frac * pstar + (R(1) - frac) * po;
  if (spout < R(0))
    qg[ID] = ro, qg[IU] = uo, qg[IP] = po;
  if (spin > R(0))
    qg[ID] = rstar, qg[IU] = ustar, qg[IP] = pstar;
  qg[IV] = sgnm > R(0) ? ql[IV] : qr[IV];
  if constexpr (NV == 5)
    qg[IW] = sgnm > R(0) ? ql[IW] : qr[IW];
  cmpflx<R, NV>(qg, flux, C);
}

// conservative state and flux of a primitive state, as riemann_llf and
// riemann_hll build them (RiemannSolvers.h:262-320, 384-420)
template <class R, int NV>
__device__ __forceinline__ void
hydro_uf(const R (&q)[NV], R (&u)[NV], R (&f)[NV], R entho)
{
  u[ID] = q[ID];
  u[IP] = q[IP] * entho + R(0.5) * q[ID] * q[IU] * q[IU];
  u[IP] += R(0.5) * q[ID] * q[IV] * q[IV];
  if constexpr (NV == 5)
    u[IP] += R(0.5) * q[ID] * q[IW] * q[IW];
  u[IU] = q[ID] * q[IU];
  u[IV] = q[ID] * q[IV];
  if constexpr (NV == 5)
    u[IW] = q[ID] * q[IW];
  f[ID] = u[ID] * q[IU];
  f[IP] = q[IU] * (u[IP] + q[IP]);
  f[IU] = q[IP] + u[IU] * q[IU];
  f[IV] = f[ID] * q[IV];
  if constexpr (NV == 5)
    f[IW] = f[ID] * q[IW];
}

// riemann_llf (RiemannSolvers.h:218-330)
template <class R, int NV>
__device__ __forceinline__ void
riemann_llf(const R (&ql)[NV], const R (&qr)[NV], R (&flux)[NV], const HydroConst<R> & C)
{
  const R entho = C.entho;
  const R rl = fmax(ql[ID], C.smallr), ul = ql[IU], pl = fmax(ql[IP], rl * C.smallp);
  const R rr = fmax(qr[ID], C.smallr), ur = qr[IU], pr = fmax(qr[IP], rr * C.smallp);
  const R cl = kFast64<R> ? sqrt_ratio64(C.gamma0 * pl, rl) : sqrt(C.gamma0 * pl / rl);
  const R cr = kFast64<R> ? sqrt_ratio64(C.gamma0 * pr, rr) : sqrt(C.gamma0 * pr / rr);
  const R cmax = fmax(fabs(ul) + cl, fabs(ur) + cr);
  R       uleft[NV], uright[NV], fleft[NV], fright[NV];
  hydro_uf<R, NV>(ql, uleft, fleft, entho);
  hydro_uf<R, NV>(qr, uright, fright, entho);
#pragma unroll
  for (int v = 0; v < NV; ++v)
    flux[v] = R(0.5) * (fleft[v] + fright[v] - cmax * (uright[v] - uleft[v]));
}

// riemann_hll (RiemannSolvers.h:344-432); used for 2D only, as the
// reference's 3D dispatch has no HLL branch
template <class R, int NV>
__device__ __forceinline__ void
riemann_hll(const R (&ql)[NV], const R (&qr)[NV], R (&flux)[NV], const HydroConst<R> & C)
{
  const R entho = C.entho;
  const R rl = fmax(ql[ID], C.smallr), ul = ql[IU], pl = fmax(ql[IP], rl * C.smallp);
  const R rr = fmax(qr[ID], C.smallr), ur = qr[IU], pr = fmax(qr[IP], rr * C.smallp);
  const R cl = kFast64<R> ? sqrt_ratio64(C.gamma0 * pl, rl) : sqrt(C.gamma0 * pl / rl);
  const R cr = kFast64<R> ? sqrt_ratio64(C.gamma0 * pr, rr) : sqrt(C.gamma0 * pr / rr);
  const R SL = fmin(fmin(ul, ur) - fmax(cl, cr), R(0));
  const R SR = fmax(fmax(ul, ur) + fmax(cl, cr), R(0));
  R       uleft[NV], uright[NV], fleft[NV], fright[NV];
  hydro_uf<R, NV>(ql, uleft, fleft, entho);
  hydro_uf<R, NV>(qr, uright, fright, entho);
#pragma unroll
  for (int v = 0; v < NV; ++v)
    flux[v] = (SR * fleft[v] - SL * fright[v] + SR * SL * (uright[v] - uleft[v])) / (SR - SL);
}

// riemann_hydro (RiemannSolvers.h:573-640) with the solver fixed at compile
// time: RS = the reference's riemannSolverType (0 approx, 1 llf, 2 hll, 3 hllc)
template <int RS, class R, int NV>
__device__ __forceinline__ void
hydro_riemann(const R (&ql)[NV], const R (&qr)[NV], R (&flux)[NV], const HydroConst<R> & C)
{
  if constexpr (RS == 0)
    riemann_approx<R, NV>(ql, qr, flux, C);
  else if constexpr (RS == 1)
    riemann_llf<R, NV>(ql, qr, flux, C);
  else if constexpr (RS == 2)
    riemann_hll<R, NV>(ql, qr, flux, C);
  else
    hllc<R, NV>(ql, qr, flux, C);
}

// per-cell CFL candidate of ComputeDtFunctor{2D,3D}
// (HydroRunFunctors2D.h:56-84, HydroRunFunctors3D.h:49-84), in the working
// precision: FP64 keeps the reference's expression; the mixed form uses the
// FP32 inverse cell sizes.  Threads keep a NaN-ignoring max (fmax, as the
// reference's reduction) and convert to the FP64 key once.
template <class R, int NV, class PP>
__device__ __forceinline__ R
hydro_invdt(const R (&u)[NV], const HydroConst<R> & C, const PP & P)
{
  R q[NV];
  hydro_prims<R, NV>(u, q, C);
  const R c = hydro_sound<R>(q[ID], q[IP], C);
  const R vx = c + fabs(q[IU]);
  const R vy = c + fabs(q[IV]);
  if constexpr (sizeof(R) == 8 && !kFast64<R>)
  {
    if constexpr (NV == 4)
      return vx / P.dx + vy / P.dy;
    else
    {
      const R vz = c + fabs(q[IW]);
      return vx / P.dx + vy / P.dy + vz / P.dz;
    }
  }
  else if constexpr (sizeof(R) == 8)
  {
    // FP64 FMA build: the inverse cell sizes prepared on the host
    if constexpr (NV == 4)
      return vx * P.idxd + vy * P.idyd;
    else
    {
      const R vz = c + fabs(q[IW]);
      return vx * P.idxd + vy * P.idyd + vz * P.idzd;
    }
  }
  else
  {
    if constexpr (NV == 4)
      return vx * P.idx + vy * P.idy;
    else
    {
      const R vz = c + fabs(q[IW]);
      return vx * P.idx + vy * P.idy + vz * P.idz;
    }
  }
}

// ---------------------------------------------------------------------------
// Static gravity (SolverHydroMuscl with [gravity] enabled)
// ---------------------------------------------------------------------------

// gravity vector of cell (i, j, k) in raw array indexes (ghosts included;
// the field is read as stored, not mapped through the boundary conditions).
// Indexes past the array (cells of partial tiles, whose results are
// discarded) are clamped.
template <class S, class R, int NV>
__device__ __forceinline__ void
grav_at(const KParams & P, int i, int j, int k, R (&g)[3])
{
  if (P.gfield)
  {
    i = min(max(i, 0), P.isize - 1);
    j = min(max(j, 0), P.jsize - 1);
    k = min(max(k, 0), P.ksize - 1);
    const S *       G = (const S *)P.gfield;
    const long long off = (long long)k * P.plane + (long long)j * P.isize + i;
    g[0] = (R)ldg(G + off);
    g[1] = (R)ldg(G + P.vstride + off);
    g[2] = NV == 5 ? (R)ldg(G + 2 * P.vstride + off) : R(0);
  }
  else if constexpr (sizeof(R) == 8)
  {
    g[0] = P.g[0], g[1] = P.g[1], g[2] = P.g[2];
  }
  else
  {
    g[0] = P.gf[0], g[1] = P.gf[1], g[2] = P.gf[2];
  }
}

// Hancock gravity predictor of one face state: q += (dt/2) g of the cell the
// state was traced from, on the velocity components in the cell's own frame
// (before any IU/IV/IW swap; HydroRunFunctors2D.h:656-665,
// HydroRunFunctors3D.h:489-500).  hg = (0.5 dt) g.
template <class R, int NV>
__device__ __forceinline__ void
grav_kick(R (&q)[NV], const R (&hg)[3])
{
  q[IU] += hg[0];
  q[IV] += hg[1];
  if constexpr (NV == 5)
    q[IW] += hg[2];
}

// GravitySourceTermFunctor2D/3D (HydroRunFunctors2D.h:1555-1630,
// HydroRunFunctors3D.h:1903-1980) on the updated state u of one cell:
// momentum += (dt/2) g (rho_old + rho_new), energy += the kinetic energy
// change; the 2D form floors rho_new at smallr.  FP64 keeps the reference's
// expression (ekin_new - ekin_old); FP32 uses the equal form
// sum du (m + du/2) / rho_new, which has no cancellation.
template <class R, int NV>
__device__ __forceinline__ void
grav_source(R (&u)[NV], R rho_old, const R (&g)[3], R hdt, const HydroConst<R> & C)
{
  const R rn = NV == 4 ? fmax(C.smallr, u[ID]) : u[ID];
  if constexpr (sizeof(R) == 8)
  {
    R ru = u[IU], rv = u[IV];
    if constexpr (NV == 4)
    {
      const R ek0 = R(0.5) * (ru * ru + rv * rv) / rn;
      ru += hdt * g[0] * (rho_old + rn);
      rv += hdt * g[1] * (rho_old + rn);
      u[IU] = ru;
      u[IV] = rv;
      const R ek1 = R(0.5) * (ru * ru + rv * rv) / rn;
      u[IP] += (ek1 - ek0);
    }
    else
    {
      R       rw = u[IW];
      const R ek0 = R(0.5) * (ru * ru + rv * rv + rw * rw) / rn;
      ru += hdt * g[0] * (rho_old + rn);
      rv += hdt * g[1] * (rho_old + rn);
      rw += hdt * g[2] * (rho_old + rn);
      u[IU] = ru;
      u[IV] = rv;
      u[IW] = rw;
      const R ek1 = R(0.5) * (ru * ru + rv * rv + rw * rw) / rn;
      u[IP] += (ek1 - ek0);
    }
  }
  else
  {
    const R rs = rho_old + rn;
    R       de = R(0);
#pragma unroll
    for (int e = 0; e < NV - 2; ++e)
    {
      const R du = hdt * g[e] * rs;
      de += du * (u[IU + e] + R(0.5) * du);
      u[IU + e] += du;
    }
    u[IP] += de * rcp_a(rn);
  }
}

// per-cell CFL candidate of ComputeDtGravityFunctor2D/3D
// (HydroRunFunctors2D.h:125-170, HydroRunFunctors3D.h:133-184):
// g dt^2 / (2 dx) + u dt / dx <= cfl, u = sum(|v_i| + c), g = sum(|g_i|),
// dx = min(dx, dy[, dz]).  FP64 keeps the reference's expression; FP32 writes
// the correction factor kk / (sqrt(1 + 2 kk) - 1) as (sqrt(1 + 2 kk) + 1) / 2,
// equal without the cancellation.
template <class R, int NV>
__device__ __forceinline__ R
hydro_invdt_grav(const R (&u)[NV], const R (&g)[3], const HydroConst<R> & C, const KParams & P)
{
  R q[NV];
  hydro_prims<R, NV>(u, q, C);
  const R c = hydro_sound<R>(q[ID], q[IP], C);
  R       velocity = c + fabs(q[IU]);
  velocity += c + fabs(q[IV]);
  R kk = fabs(g[0]) + fabs(g[1]);
  if constexpr (NV == 5)
  {
    velocity += c + fabs(q[IW]);
    kk = kk + fabs(g[2]);
  }
  if constexpr (sizeof(R) == 8)
  {
    kk *= P.cfl_dxmin / (velocity * velocity);
    kk = fmax(kk, 1e-4);
    velocity *= kk / (sqrt(1.0 + 2.0 * kk) - 1.0);
    return velocity / P.dxmin;
  }
  else
  {
    kk = fmax(kk * P.cfl_dxminf * rcp_a(velocity * velocity), 1e-4f);
    return velocity * (R(0.5) * (sqrt_a(R(1) + R(2) * kk) + R(1))) * P.idxminf;
  }
}

} // namespace EK_NS
