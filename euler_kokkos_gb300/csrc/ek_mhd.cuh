// CT-MHD cell/face/edge arithmetic (3D), one cell, face or edge at a time.
// Expressions keep the reference's evaluation order (cited per function), so
// the FP64 build without FMA contraction reproduces the reference bit for bit.
#pragma once

#include <type_traits>

#include "ek_common.cuh"
#include "ek_slabs.h"

namespace EK_NS
{

template <class R>
struct MhdConst
{
  R gamma0, smallr, smallp, smallc, slope_type;
  R entho; // 1 / (gamma0 - 1), the value every Riemann solver of the reference computes
};

// rho c_fast^2 from gamma p, B^2 and Bn^2 in the FP64 FMA build: with all terms
// multiplied by rho no reciprocal of the density is needed before the outer
// root, which is one sqrt_ratio64 for the largest of several speeds.  The
// discriminant, (B^2 - gamma p)^2 / 4 + gamma p Bt^2 by its parts, is not
// negative.
// beyond 2^-500 to 2^500, where the squares leave the range: scaled by 2^600 or
// 2^-600 (out of line, so that the callers' registers are not its)
__device__ __noinline__ double
fast_num64_scaled(double s, double gp, double bn2)
{
  const bool   small = hi32(s) < 0x3ff00000;
  const double f = small ? 0x1p600 : 0x1p-600, t = s * f;
  return (t + sqrt64(max_floor64(fma(t, t, -((gp * f) * (bn2 * f))), 0.0))) * (small ? 0x1p-600 : 0x1p600);
}
__device__ __forceinline__ double
fast_num64(double gp, double b2, double bn2)
{
  const double s = scale_pos64<1>(b2 + gp);
  if ((unsigned)(hi32(s) - 0x20b00000) >= 0x3e800000u)
    return fast_num64_scaled(s, gp, bn2);
  return s + sqrt64(max_floor64(fma(s, s, -(gp * bn2)), 0.0));
}

// find_speed_fast<dir> (mhd_utils.h:89-117)
template <class R, int DIR>
__device__ __forceinline__ R
mhd_speed_fast(const R (&q)[8], R gamma0)
{
  const R d = q[ID], p = q[IP], a = q[IA], b = q[IB], c = q[IC];
  const R b2 = a * a + b * b + c * c;
  const R bn = DIR == 0 ? a : (DIR == 1 ? b : c);
  if constexpr (kFast64<R>)
    return sqrt_ratio64(fast_num64(gamma0 * p, b2, bn * bn), d);
  else if constexpr (kShareRecip)
  {
    const R id = R(1) / d;
    const R c2 = gamma0 * p * id;
    const R d2 = R(0.5) * (b2 * id + c2);
    return sqrt(d2 + sqrt(d2 * d2 - c2 * bn * bn * id));
  }
  const R c2 = gamma0 * p / d;
  const R d2 = R(0.5) * (b2 / d + c2);
  return sqrt(d2 + sqrt(d2 * d2 - c2 * bn * bn / d));
}

// find_speed_info<THREE_D> summed as ComputeDtFunctor3D_MHD does
// (mhd_utils.h:319-366, MHDRunFunctors3D.h:58-76).  FP64: the reference's
// expression; mixed: the candidate is formed in FP32 with 1/dx (the
// max-reduction and dt stay FP64).
template <class R>
__device__ __forceinline__ R
mhd_invdt(const R (&q)[8], R gamma0, double dx, double dy, double dz, float idx, float idy, float idz,
          double idxd, double idyd, double idzd)
{
  const R d = q[ID], p = q[IP], a = q[IA], b = q[IB], c = q[IC];
  const R b2 = a * a + b * b + c * c;
  if constexpr (sizeof(R) == 4)
  {
    const float id = rcp_a(d);
    const float c2 = gamma0 * p * id;
    const float d2 = 0.5f * (b2 * id + c2);
    const float dd = d2 * d2, cr = c2 * id;
    const float cfx = sqrt_a(d2 + sqrt_a(dd - cr * a * a));
    const float cfy = sqrt_a(d2 + sqrt_a(dd - cr * b * b));
    const float cfz = sqrt_a(d2 + sqrt_a(dd - cr * c * c));
    return (cfx + fabsf(q[IU])) * idx + (cfy + fabsf(q[IV])) * idy + (cfz + fabsf(q[IW])) * idz;
  }
  if constexpr (kFast64<R>)
  {
    // FP64 FMA build: host-prepared 1/dx
    const R gp = gamma0 * p;
    const R cfx = sqrt_ratio64(fast_num64(gp, b2, a * a), d);
    const R cfy = sqrt_ratio64(fast_num64(gp, b2, b * b), d);
    const R cfz = sqrt_ratio64(fast_num64(gp, b2, c * c), d);
    return (cfx + fabs(q[IU])) * idxd + (cfy + fabs(q[IV])) * idyd + (cfz + fabs(q[IW])) * idzd;
  }
  const R c2 = gamma0 * p / d;
  const R d2 = R(0.5) * (b2 / d + c2);
  const R cfx = sqrt(d2 + sqrt(d2 * d2 - c2 * a * a / d));
  const R cfy = sqrt(d2 + sqrt(d2 * d2 - c2 * b * b / d));
  const R cfz = sqrt(d2 + sqrt(d2 * d2 - c2 * c * c / d));
  const R vx = cfx + fabs(q[IU]);
  const R vy = cfy + fabs(q[IV]);
  const R vz = cfz + fabs(q[IW]);
  return vx / dx + vy / dy + vz / dz;
}

// constoprim_mhd (MHDBaseFunctor3D.h:194-242).  u: hydro variables of the
// cell, bl/br: face fields of the cell and of its +1 neighbours.  In the
// mixed form (R = float) the internal energy is recomputed in FP64 from the
// FP64 face fields (bl64/br64, only read then) when total and
// magnetic+kinetic energy cancel (low beta / high Mach).
template <class R, class FB>
__device__ __forceinline__ void
mhd_constoprim(const R (&u)[5], const R (&bl)[3], const R (&br)[3], R (&q)[8], const MhdConst<R> & C,
               FB && fp64_faces)
{
  if constexpr (kFast64<R>)
  {
    // FP64 FMA build: p = (gamma - 1) (E - B^2 / 2 - rho v^2 / 2)
    const R d = max_floor64(u[ID], C.smallr), id = rcp64(d);
    q[ID] = d;
    q[IU] = u[IU] * id;
    q[IV] = u[IV] * id;
    q[IW] = u[IW] * id;
    q[IA] = half64(bl[0] + br[0]);
    q[IB] = half64(bl[1] + br[1]);
    q[IC] = half64(bl[2] + br[2]);
    const R k2 = q[IU] * q[IU] + q[IV] * q[IV] + q[IW] * q[IW];
    const R b2 = q[IA] * q[IA] + q[IB] * q[IB] + q[IC] * q[IC];
    q[IP] = floor_ratio64((C.gamma0 - R(1)) * fma(R(-0.5) * d, k2, fma(R(-0.5), b2, u[IP])), d, C.smallp);
    return;
  }
  q[ID] = fmax(u[ID], C.smallr);
  R id = R(0);
  if constexpr (sizeof(R) == 4)
  {
    id = rcp_a(q[ID]);
    q[IU] = u[IU] * id;
    q[IV] = u[IV] * id;
    q[IW] = u[IW] * id;
  }
  else
  {
    q[IU] = u[IU] / q[ID];
    q[IV] = u[IV] / q[ID];
    q[IW] = u[IW] / q[ID];
  }
  q[IA] = R(0.5) * (bl[0] + br[0]);
  q[IB] = R(0.5) * (bl[1] + br[1]);
  q[IC] = R(0.5) * (bl[2] + br[2]);
  const R eken = R(0.5) * (q[IU] * q[IU] + q[IV] * q[IV] + q[IW] * q[IW]);
  const R emag = R(0.5) * (q[IA] * q[IA] + q[IB] * q[IB] + q[IC] * q[IC]);
  R       eint;
  if constexpr (sizeof(R) == 4)
    eint = (u[IP] - emag) * id - eken;
  else
    eint = (u[IP] - emag) / q[ID] - eken;
  if constexpr (sizeof(R) == 4)
  {
    // FP64 island: E - emag - rho*eken cancels (low beta or high Mach)
    if (fabs(eint * q[ID]) < R(1.0 / 128.0) * fabs(u[IP]))
    {
      double bl64[3], br64[3];
      fp64_faces(bl64, br64);
      const double ba = 0.5 * (bl64[0] + br64[0]), bb = 0.5 * (bl64[1] + br64[1]),
                   bc = 0.5 * (bl64[2] + br64[2]);
      const double em = 0.5 * (ba * ba + bb * bb + bc * bc);
      const double d = (double)q[ID];
      const double vx = (double)u[IU] / d, vy = (double)u[IV] / d, vz = (double)u[IW] / d;
      eint = (R)(((double)u[IP] - em) / d - 0.5 * (vx * vx + vy * vy + vz * vz));
    }
  }
  q[IP] = fmax((C.gamma0 - R(1.0)) * q[ID] * eint, q[ID] * C.smallp);
}

// riemann_hlld in FP32 for the mixed form: the reference's solver with each
// shared denominator inverted once (rcp_a), |B_n| / sqrt(rho*) as a
// reciprocal square root, and the left and right states in the two lanes of
// packed FP32 pairs; the same branches, and the faces it cannot decide left
// to FP64 (below).

// The star-state denominators of HLLD, estar = rho (S - u)(S - ustar) - Bn^2,
// cancel as the state approaches the degenerate one (transverse field near
// zero, fast speed near the Alfven speed).  In FP32 their quotients
// (v*, B*, w*, C*) then lose all accuracy and a face flux can blow up the
// solution; FP64 keeps them accurate, as the reference's FP64 build shows.
// Below this fraction of Bn^2 the face is recomputed in FP64: FP32 rounding
// leaves estar an absolute error of a few 1e-7 Bn^2, so above the threshold the
// quotients keep a relative accuracy of about 1e-2 or better.  (A threshold of
// 2^-7 flags a few per cent of the Orszag-Tang faces, where the transverse
// field crosses zero; 2^-14 flags none of them.)
constexpr float kHlldStarTol = 1.0f / 16384.0f;

// false: a star-state denominator of this face is ill-conditioned in FP32
// (|estar| < kHlldStarTol Bn^2), or the reference's degenerate-state test
// |estar / Bn^2 - 1| <= 1e-8 cannot be decided in FP32; the face is then
// solved in FP64 (flux is not written)
template <int NF>
__device__ __forceinline__ bool
mhd_hlld_f32(const float (&ql)[8], const float (&qr)[8], float (&flux)[NF], float gamma0, float entho)
{
  // left state in lane x, right state in lane y
  const float  a = 0.5f * (ql[IA] + qr[IA]);
  const float  sgnm = (a >= 0.f) ? 1.f : -1.f;
  const float  a2 = a * a;
  const float2 A = f2s(a), A2 = f2s(a2), H = f2s(0.5f);
  const float2 r = f2(ql[ID], qr[ID]), p = f2(ql[IP], qr[IP]), u = f2(ql[IU], qr[IU]);
  const float2 v = f2(ql[IV], qr[IV]), w = f2(ql[IW], qr[IW]), b = f2(ql[IB], qr[IB]), c = f2(ql[IC], qr[IC]);
  const float2 bt2 = fma2(c, c, mul2(b, b)), bsq = add2(bt2, A2);
  const float2 ecin = mul2(mul2(H, fma2(w, w, fma2(v, v, mul2(u, u)))), r);
  const float2 emag = mul2(H, bsq);
  const float2 etot = add2(fma2(p, f2s(entho), ecin), emag);
  const float2 ptot = add2(p, emag);
  const float2 vdotb = fma2(w, c, fma2(v, b, mul2(u, A)));

  // the larger fast magnetosonic speed (find_speed_fast, the normal field a), the
  // discriminant as (B^2 - gamma p)^2 / 4 + gamma p Bt^2, which does not cancel.
  // All terms divided by the density first: squares of pressures, or a pressure
  // times a density, leave FP32's range where the speeds are ordinary
  const float2 id = f2(rcp_a(r.x), rcp_a(r.y)), g = mul2(mul2(f2s(gamma0), p), id);
  const float2 h = mul2(H, fma2(bsq, id, g)), hm = sub2(h, g);
  const float2 dq = fma2(g, mul2(bt2, id), mul2(hm, hm)), n = add2(h, f2(sqrt_a(dq.x), sqrt_a(dq.y)));
  const float  cmax = sqrt_a(fmaxf(n.x, n.y));
  const float  sl = fminf(u.x, u.y) - cmax;
  const float  sr = fmaxf(u.x, u.y) + cmax;
  const float2 S = f2(sl, sr);
  const float2 su = sub2(S, u);  // S - u
  const float2 rsu = mul2(r, su); // rho (S - u): -rcl, rcr
  // u* = u_l + w, p* = p_l - rcl w
  const float  w0 = (ptot.x - ptot.y - rsu.y * (u.x - u.y)) * rcp_a(rsu.y - rsu.x);
  const float  ustar = u.x + w0, ptotstar = fmaf(rsu.x, w0, ptot.x);
  const float2 US = f2s(ustar);
  const float2 sus = sub2(S, US);
  // the star-state denominators; the face goes to FP64 when one is
  // ill-conditioned, or within 1e-6 of the reference's degenerate-state test
  // |estar / Bn^2 - 1| <= 1e-8 (which FP32 cannot decide).  So that test is
  // false for every face solved here, and its branch is not needed below.
  const float2 estar = fma2(rsu, sus, neg2(A2));
  auto         ill = [&](float e) { return fabsf(e) < kHlldStarTol * a2 || fabsf(e - a2) <= 1e-6f * a2; };
  if (ill(estar.x) || ill(estar.y))
    return false;

  const float2 is = f2(rcp_a(sus.x), rcp_a(sus.y));
  const float2 rstar = mul2(rsu, is);
  const float2 e = fma2(rsu, su, neg2(A2)); // rho (S - u)^2 - Bn^2
  const float2 ie = f2(rcp_a(estar.x), rcp_a(estar.y));
  const float2 t = mul2(mul2(A, sub2(US, u)), ie);
  const float2 vstar = fma2(b, neg2(t), v);
  const float2 bstar = mul2(mul2(b, e), ie);
  const float2 wstar = fma2(c, neg2(t), w);
  const float2 cstar = mul2(mul2(c, e), ie);
  const float2 vdotbstar = fma2(wstar, cstar, fma2(vstar, bstar, mul2(US, A)));
  const float2 etotstar =
    mul2(add2(fma2(su, etot, neg2(mul2(ptot, u))), fma2(A, sub2(vdotb, vdotbstar), f2s(ptotstar * ustar))), is);
  const float  sqrrstarl = sqrt_a(rstar.x), sqrrstarr = sqrt_a(rstar.y);
  const float  sal = ustar - fabsf(a) * rsqrt_a(rstar.x);
  const float  sar = ustar + fabsf(a) * rsqrt_a(rstar.y);

  const float rl = r.x, ul = u.x, vl = v.x, wl = w.x, bl = b.x, cl = c.x;
  const float rr = r.y, ur = u.y, vr = v.y, wr = w.y, br = b.y, cr = c.y;
  const float ptotl = ptot.x, ptotr = ptot.y, etotl = etot.x, etotr = etot.y, vdotbl = vdotb.x, vdotbr = vdotb.y;
  const float rstarl = rstar.x, rstarr = rstar.y;
  const float vstarl = vstar.x, vstarr = vstar.y, wstarl = wstar.x, wstarr = wstar.y;
  const float bstarl = bstar.x, bstarr = bstar.y, cstarl = cstar.x, cstarr = cstar.y;
  const float vdotbstarl = vdotbstar.x, vdotbstarr = vdotbstar.y, etotstarl = etotstar.x, etotstarr = etotstar.y;

  float ro, uo, vo, wo, bo, co, ptoto, etoto, vdotbo;
  if (sl > 0.f)
  {
    ro = rl, uo = ul, vo = vl, wo = wl, bo = bl, co = cl;
    ptoto = ptotl, etoto = etotl, vdotbo = vdotbl;
  }
  else if (sal > 0.f)
  {
    ro = rstarl, uo = ustar, vo = vstarl, wo = wstarl, bo = bstarl, co = cstarl;
    ptoto = ptotstar, etoto = etotstarl, vdotbo = vdotbstarl;
  }
  else if (sr > 0.f && !(ustar > 0.f) && !(sar > 0.f))
  {
    ro = rstarr, uo = ustar, vo = vstarr, wo = wstarr, bo = bstarr, co = cstarr;
    ptoto = ptotstar, etoto = etotstarr, vdotbo = vdotbstarr;
  }
  else if (!(sr > 0.f) && !(ustar > 0.f) && !(sar > 0.f))
  {
    ro = rr, uo = ur, vo = vr, wo = wr, bo = br, co = cr;
    ptoto = ptotr, etoto = etotr, vdotbo = vdotbr;
  }
  else
  {
    const float iss = rcp_a(sqrrstarl + sqrrstarr);
    const float vss = (sqrrstarl * vstarl + sqrrstarr * vstarr + sgnm * (bstarr - bstarl)) * iss;
    const float wss = (sqrrstarl * wstarl + sqrrstarr * wstarr + sgnm * (cstarr - cstarl)) * iss;
    const float bss = (sqrrstarl * bstarr + sqrrstarr * bstarl + sgnm * sqrrstarl * sqrrstarr * (vstarr - vstarl)) * iss;
    const float css = (sqrrstarl * cstarr + sqrrstarr * cstarl + sgnm * sqrrstarl * sqrrstarr * (wstarr - wstarl)) * iss;
    const float vdotbss = ustar * a + vss * bss + wss * css;
    vo = vss, wo = wss, bo = bss, co = css;
    uo = ustar, ptoto = ptotstar, vdotbo = vdotbss;
    if (ustar > 0.f)
    {
      ro = rstarl;
      etoto = etotstarl - sgnm * sqrrstarl * (vdotbstarl - vdotbss);
    }
    else
    {
      ro = rstarr;
      etoto = etotstarr + sgnm * sqrrstarr * (vdotbstarr - vdotbss);
    }
  }
  flux[ID] = ro * uo;
  flux[IP] = (etoto + ptoto) * uo - a * vdotbo;
  flux[IU] = ro * uo * uo - a2 + ptoto;
  flux[IV] = ro * uo * vo - a * bo;
  flux[IW] = ro * uo * wo - a * co;
  if constexpr (NF > 5)
    flux[5] = co * uo - a * wo;
  return true;
}

// riemann_hlld (RiemannSolvers_MHD.h:130-364) in the FP64 FMA build: the same
// states with about 180 FP64-pipe operations per face.  Both fast speeds share
// one outer root (fast_num64); u* and p* follow from one quotient w; the
// degenerate-state test |estar / Bn^2 - 1| <= 1e-8 is taken without the
// division; roots and quotients by rsqrt64 / rcp64; regions, minima and signs on
// the integer pipes.  With the emf and trace below: FP64 2D step 189 -> 122 us at
// 200 x 136, 3D step 4170 -> 2830 us at 32^3.
template <int NF>
__device__ __forceinline__ void
mhd_hlld64(const double (&ql)[8], const double (&qr)[8], double (&flux)[NF], double gamma0, double entho)
{
  const double a = half64(ql[IA] + qr[IA]), a2 = a * a;
  struct Side
  {
    double pt, et, vb, n; // total pressure and energy, v.B, rho c_fast^2
  };
  auto side = [&](const double (&q)[8]) {
    Side         s;
    const double b2 = fma(q[IC], q[IC], fma(q[IB], q[IB], a2)), em = scale_pos64<1>(b2);
    const double k2 = fma(q[IW], q[IW], fma(q[IV], q[IV], q[IU] * q[IU]));
    s.pt = q[IP] + em;
    s.et = fma(q[IP], entho, fma(scale_pos64<1>(q[ID]), k2, em));
    s.vb = fma(q[IW], q[IC], fma(q[IV], q[IB], q[IU] * a));
    s.n = fast_num64(gamma0 * q[IP], b2, a2);
    return s;
  };
  const Side   L = side(ql), R = side(qr);
  const double ul = ql[IU], ur = qr[IU];
  const double cmax = sqrt_larger_ratio64(L.n, ql[ID], R.n, qr[ID]);
  const double du = ul - ur;
  const bool   lslow = negative64(du);
  const double sl = (lslow ? ul : ur) - cmax, sr = (lslow ? ur : ul) + cmax;
  const double al = ul - sl, ar = sr - ur;
  const double rcl = ql[ID] * al, rcr = qr[ID] * ar;
  const double w = fma(-rcr, du, L.pt - R.pt) * rcp64(rcr + rcl);
  const double us = ul + w, ps = fma(-rcl, w, L.pt);
  const double usa = us * a, psus = ps * us;

  struct Star
  {
    double r, v, w, b, c, vb, et, sq, al; // sq = sqrt(rho*), al = |Bn| / sqrt(rho*)
  };
  // dS = S - u, rd = rho dS, du = u* - u
  auto star = [&](const double (&q)[8], const Side & s, double S, double dS, double rd, double du) {
    Star         t;
    const double sus = S - us, is = rcp64(sus);
    t.r = rd * is;
    const double es = fma(rd, sus, -a2), e = fma(rd, dS, -a2), ie = rcp64(es);
    const bool   deg = positive64(a2) &&
                     __double_as_longlong(abs64(es - a2)) <= __double_as_longlong(1e-8 * a2);
    const double h = deg ? 0.0 : a * du * ie, f = deg ? 1.0 : e * ie;
    t.v = fma(-q[IB], h, q[IV]);
    t.w = fma(-q[IC], h, q[IW]);
    t.b = q[IB] * f;
    t.c = q[IC] * f;
    t.vb = fma(t.w, t.c, fma(t.v, t.b, usa));
    t.et = fma(a, s.vb - t.vb, fma(-s.pt, q[IU], fma(dS, s.et, psus))) * is;
    const double y = rsqrt64(t.r);
    t.sq = t.r * y;
    t.al = abs64(a) * y;
    return t;
  };
  const Star   Ls = star(ql, L, sl, flip64(al, true), flip64(rcl, true), w), Rs = star(qr, R, sr, ar, rcr, us - ur);
  const double sal = us - Ls.al, sar = us + Rs.al;
  const bool   left = positive64(sl), lstar = !left && positive64(sal);
  const bool   rside = !left && !lstar && !positive64(us) && !positive64(sar);
  double       ro, uo, vo, wo, bo, co, po, eo, vbo;
  if (left || (rside && !positive64(sr)))
  {
    ro = left ? ql[ID] : qr[ID], uo = left ? ul : ur, vo = left ? ql[IV] : qr[IV], wo = left ? ql[IW] : qr[IW];
    bo = left ? ql[IB] : qr[IB], co = left ? ql[IC] : qr[IC];
    po = left ? L.pt : R.pt, eo = left ? L.et : R.et, vbo = left ? L.vb : R.vb;
  }
  else if (lstar || rside)
  {
    ro = lstar ? Ls.r : Rs.r, uo = us, vo = lstar ? Ls.v : Rs.v, wo = lstar ? Ls.w : Rs.w;
    bo = lstar ? Ls.b : Rs.b, co = lstar ? Ls.c : Rs.c;
    po = ps, eo = lstar ? Ls.et : Rs.et, vbo = lstar ? Ls.vb : Rs.vb;
  }
  else
  {
    const bool   neg = negative64(a), cl = positive64(us); // sgn(Bn) < 0; left of the contact
    const double is = rcp64(Ls.sq + Rs.sq), sq2 = Ls.sq * Rs.sq;
    vo = (fma(Ls.sq, Ls.v, Rs.sq * Rs.v) + flip64(Rs.b - Ls.b, neg)) * is;
    wo = (fma(Ls.sq, Ls.w, Rs.sq * Rs.w) + flip64(Rs.c - Ls.c, neg)) * is;
    bo = fma(sq2, flip64(Rs.v - Ls.v, neg), fma(Ls.sq, Rs.b, Rs.sq * Ls.b)) * is;
    co = fma(sq2, flip64(Rs.w - Ls.w, neg), fma(Ls.sq, Rs.c, Rs.sq * Ls.c)) * is;
    vbo = fma(wo, co, fma(vo, bo, usa));
    uo = us, po = ps;
    ro = cl ? Ls.r : Rs.r;
    eo = fma(flip64(cl ? Ls.sq : Rs.sq, neg == cl), vbo - (cl ? Ls.vb : Rs.vb), cl ? Ls.et : Rs.et);
  }
  const double m = ro * uo;
  flux[ID] = m;
  flux[IP] = fma(eo + po, uo, -(a * vbo));
  flux[IU] = fma(m, uo, po - a2);
  flux[IV] = fma(m, vo, -(a * bo));
  flux[IW] = fma(m, wo, -(a * co));
  if constexpr (NF > 5)
    flux[5] = fma(co, uo, -(a * wo));
}

// riemann_hlld (RiemannSolvers_MHD.h:130-364), states in the face frame.
// The 3D update uses the five hydro components of the flux (NF = 5); the 2D
// update also uses the Bz component, returned in flux[5] when NF = 6.
// Returns false when the FP32 solver leaves the face to its FP64 island (an
// ill-conditioned star state, see mhd_hlld_f32): the caller then solves it
// with mhd_hlld<double> from the same states.
template <class R, int NF = 5>
__device__ __forceinline__ bool
mhd_hlld(R (&ql)[8], R (&qr)[8], R (&flux)[NF], R gamma0, R entho)
{
  if constexpr (sizeof(R) == 4)
    return mhd_hlld_f32<NF>(ql, qr, flux, gamma0, entho);
  else if constexpr (kFast64<R>)
  {
    mhd_hlld64<NF>(ql, qr, flux, gamma0, entho);
    return true;
  }
  else
  {
  const R a = R(0.5) * (ql[IA] + qr[IA]);
  const R sgnm = (a >= R(0)) ? R(1) : R(-1);
  ql[IA] = a;
  qr[IA] = a;
  const R rl = ql[ID], pl = ql[IP], ul = ql[IU], vl = ql[IV], wl = ql[IW], bl = ql[IB], cl = ql[IC];
  const R ecinl = R(0.5) * (ul * ul + vl * vl + wl * wl) * rl;
  const R emagl = R(0.5) * (a * a + bl * bl + cl * cl);
  const R etotl = pl * entho + ecinl + emagl;
  const R ptotl = pl + emagl;
  const R vdotbl = ul * a + vl * bl + wl * cl;
  const R rr = qr[ID], pr = qr[IP], ur = qr[IU], vr = qr[IV], wr = qr[IW], br = qr[IB], cr = qr[IC];
  const R ecinr = R(0.5) * (ur * ur + vr * vr + wr * wr) * rr;
  const R emagr = R(0.5) * (a * a + br * br + cr * cr);
  const R etotr = pr * entho + ecinr + emagr;
  const R ptotr = pr + emagr;
  const R vdotbr = ur * a + vr * br + wr * cr;

  const R cmax = fmax(mhd_speed_fast<R, 0>(ql, gamma0), mhd_speed_fast<R, 0>(qr, gamma0));
  const R sl = fmin(ul, ur) - cmax;
  const R sr = fmax(ul, ur) + cmax;
  const R rcl = rl * (ul - sl);
  const R rcr = rr * (sr - ur);
  const R ustar = (rcr * ur + rcl * ul + (ptotl - ptotr)) / (rcr + rcl);
  const R ptotstar = (rcr * ptotl + rcl * ptotr + rcl * rcr * (ul - ur)) / (rcr + rcl);

  R estar;
  auto degenerate = [&](R e) { return a * a > R(0) && fabs(e / (a * a) - R(1)) <= R(1e-8); };
  const R rstarl = rl * (sl - ul) / (sl - ustar);
  estar = rl * (sl - ul) * (sl - ustar) - a * a;
  const R el = rl * (sl - ul) * (sl - ul) - a * a;
  R       vstarl, wstarl, bstarl, cstarl;
  if (degenerate(estar))
  {
    vstarl = vl;
    bstarl = bl;
    wstarl = wl;
    cstarl = cl;
  }
  else
  {
    vstarl = vl - a * bl * (ustar - ul) / estar;
    bstarl = bl * el / estar;
    wstarl = wl - a * cl * (ustar - ul) / estar;
    cstarl = cl * el / estar;
  }
  const R vdotbstarl = ustar * a + vstarl * bstarl + wstarl * cstarl;
  const R etotstarl =
    ((sl - ul) * etotl - ptotl * ul + ptotstar * ustar + a * (vdotbl - vdotbstarl)) / (sl - ustar);
  const R sqrrstarl = sqrt(rstarl);
  const R calfvenl = fabs(a) / sqrrstarl;
  const R sal = ustar - calfvenl;

  const R rstarr = rr * (sr - ur) / (sr - ustar);
  estar = rr * (sr - ur) * (sr - ustar) - a * a;
  const R er = rr * (sr - ur) * (sr - ur) - a * a;
  R       vstarr, wstarr, bstarr, cstarr;
  if (degenerate(estar))
  {
    vstarr = vr;
    bstarr = br;
    wstarr = wr;
    cstarr = cr;
  }
  else
  {
    vstarr = vr - a * br * (ustar - ur) / estar;
    bstarr = br * er / estar;
    wstarr = wr - a * cr * (ustar - ur) / estar;
    cstarr = cr * er / estar;
  }
  const R vdotbstarr = ustar * a + vstarr * bstarr + wstarr * cstarr;
  const R etotstarr =
    ((sr - ur) * etotr - ptotr * ur + ptotstar * ustar + a * (vdotbr - vdotbstarr)) / (sr - ustar);
  const R sqrrstarr = sqrt(rstarr);
  const R calfvenr = fabs(a) / sqrrstarr;
  const R sar = ustar + calfvenr;

  R ro, uo, vo, wo, bo, co, ptoto, etoto, vdotbo;
  if (sl > R(0))
  {
    ro = rl, uo = ul, vo = vl, wo = wl, bo = bl, co = cl;
    ptoto = ptotl, etoto = etotl, vdotbo = vdotbl;
  }
  else if (sal > R(0))
  {
    ro = rstarl, uo = ustar, vo = vstarl, wo = wstarl, bo = bstarl, co = cstarl;
    ptoto = ptotstar, etoto = etotstarl, vdotbo = vdotbstarl;
  }
  else if (sr > R(0) && !(ustar > R(0)) && !(sar > R(0)))
  {
    ro = rstarr, uo = ustar, vo = vstarr, wo = wstarr, bo = bstarr, co = cstarr;
    ptoto = ptotstar, etoto = etotstarr, vdotbo = vdotbstarr;
  }
  else if (!(sr > R(0)) && !(ustar > R(0)) && !(sar > R(0)))
  {
    ro = rr, uo = ur, vo = vr, wo = wr, bo = br, co = cr;
    ptoto = ptotr, etoto = etotr, vdotbo = vdotbr;
  }
  else
  {
    // double-star region (only evaluated when sampled)
    const R vstarstar =
      (sqrrstarl * vstarl + sqrrstarr * vstarr + sgnm * (bstarr - bstarl)) / (sqrrstarl + sqrrstarr);
    const R wstarstar =
      (sqrrstarl * wstarl + sqrrstarr * wstarr + sgnm * (cstarr - cstarl)) / (sqrrstarl + sqrrstarr);
    const R bstarstar =
      (sqrrstarl * bstarr + sqrrstarr * bstarl + sgnm * sqrrstarl * sqrrstarr * (vstarr - vstarl)) /
      (sqrrstarl + sqrrstarr);
    const R cstarstar =
      (sqrrstarl * cstarr + sqrrstarr * cstarl + sgnm * sqrrstarl * sqrrstarr * (wstarr - wstarl)) /
      (sqrrstarl + sqrrstarr);
    const R vdotbstarstar = ustar * a + vstarstar * bstarstar + wstarstar * cstarstar;
    vo = vstarstar, wo = wstarstar, bo = bstarstar, co = cstarstar;
    uo = ustar, ptoto = ptotstar, vdotbo = vdotbstarstar;
    if (ustar > R(0))
    {
      ro = rstarl;
      etoto = etotstarl - sgnm * sqrrstarl * (vdotbstarl - vdotbstarstar);
    }
    else
    {
      ro = rstarr;
      etoto = etotstarr + sgnm * sqrrstarr * (vdotbstarr - vdotbstarstar);
    }
  }
  flux[ID] = ro * uo;
  flux[IP] = (etoto + ptoto) * uo - a * vdotbo;
  flux[IU] = ro * uo * uo - a * a + ptoto;
  flux[IV] = ro * uo * vo - a * bo;
  flux[IW] = ro * uo * wo - a * co;
  if constexpr (NF > 5)
    flux[5] = co * uo - a * wo;
  return true;
  }
}

// riemann_mhd (RiemannSolvers_MHD.h:368-389) with the solver fixed at compile
// time: RS = the reference's riemannSolverType (1 llf, 2 hll, 4 hlld)
template <int RS, class R, int NF>
__device__ __forceinline__ bool
mhd_riemann(R (&ql)[8], R (&qr)[8], R (&flux)[NF], const MhdConst<R> & C);

// find_mhd_flux (mhd_utils.h:170-231, cIso = 0): conservative state and
// flux of a face-frame primitive state; components ID, IP, IU, IV, IW and,
// for NF = 6, IC in slot 5
template <class R, int NF>
__device__ __forceinline__ void
find_mhd_flux(const R (&q)[8], R (&cv)[NF], R (&ff)[NF], R gamma0)
{
  const R entho = R(1.0) / (gamma0 - R(1.0));
  const R d = q[ID], p = q[IP], u = q[IU], v = q[IV], w = q[IW], a = q[IA], b = q[IB], c = q[IC];
  const R ecin = R(0.5) * (u * u + v * v + w * w) * d;
  const R emag = R(0.5) * (a * a + b * b + c * c);
  const R etot = p * entho + ecin + emag;
  const R ptot = p + emag;
  cv[ID] = d, cv[IP] = etot, cv[IU] = d * u, cv[IV] = d * v, cv[IW] = d * w;
  ff[ID] = d * u;
  ff[IP] = (etot + ptot) * u - a * (a * u + b * v + c * w);
  ff[IU] = d * u * u - a * a + ptot;
  ff[IV] = d * u * v - a * b;
  ff[IW] = d * u * w - a * c;
  if constexpr (NF > 5)
  {
    cv[5] = c;
    ff[5] = c * u - a * w;
  }
}

// riemann_hll for MHD (RiemannSolvers_MHD.h:27-62)
template <class R, int NF>
__device__ __forceinline__ void
mhd_hll(R (&ql)[8], R (&qr)[8], R (&flux)[NF], R gamma0)
{
  const R bx_mean = R(0.5) * (ql[IA] + qr[IA]);
  ql[IA] = bx_mean;
  qr[IA] = bx_mean;
  R uleft[NF], fleft[NF], uright[NF], fright[NF];
  find_mhd_flux<R, NF>(ql, uleft, fleft, gamma0);
  find_mhd_flux<R, NF>(qr, uright, fright, gamma0);
  const R cfleft = mhd_speed_fast<R, 0>(ql, gamma0);
  const R cfright = mhd_speed_fast<R, 0>(qr, gamma0);
  const R vleft = ql[IU], vright = qr[IU];
  const R sl = fmin(fmin(vleft, vright) - fmax(cfleft, cfright), R(0.0));
  const R sr = fmax(fmax(vleft, vright) + fmax(cfleft, cfright), R(0.0));
#pragma unroll
  for (int v = 0; v < NF; ++v)
    flux[v] = (sr * fleft[v] - sl * fright[v] + sr * sl * (uright[v] - uleft[v])) / (sr - sl);
}

// riemann_llf for MHD (RiemannSolvers_MHD.h:77-104); the information speed
// is find_speed_info of the normal direction (mhd_utils.h:379-403)
template <class R, int NF>
__device__ __forceinline__ void
mhd_llf(R (&ql)[8], R (&qr)[8], R (&flux)[NF], R gamma0)
{
  const R bx_mean = R(0.5) * (ql[IA] + qr[IA]);
  ql[IA] = bx_mean;
  qr[IA] = bx_mean;
  R uleft[NF], fleft[NF], uright[NF], fright[NF];
  find_mhd_flux<R, NF>(ql, uleft, fleft, gamma0);
  find_mhd_flux<R, NF>(qr, uright, fright, gamma0);
#pragma unroll
  for (int v = 0; v < NF; ++v)
    flux[v] = (fleft[v] + fright[v]) / R(2);
  const R cleft = mhd_speed_fast<R, 0>(ql, gamma0) + fabs(ql[IU]);
  const R cright = mhd_speed_fast<R, 0>(qr, gamma0) + fabs(qr[IU]);
  const R vel_info = fmax(cleft, cright);
#pragma unroll
  for (int v = 0; v < NF; ++v)
    flux[v] -= vel_info * (uright[v] - uleft[v]) / R(2);
}

// false: the FP32 HLLD left this face to its FP64 island (mhd_riemann_f64)
template <int RS, class R, int NF>
__device__ __forceinline__ bool
mhd_riemann(R (&ql)[8], R (&qr)[8], R (&flux)[NF], const MhdConst<R> & C)
{
  if constexpr (RS == 1)
    mhd_llf<R, NF>(ql, qr, flux, C.gamma0);
  else if constexpr (RS == 2)
    mhd_hll<R, NF>(ql, qr, flux, C.gamma0);
  else
    return mhd_hlld<R, NF>(ql, qr, flux, C.gamma0, C.entho);
  return true;
}

// The FP64 island of the FP32 HLLD: the face solved in FP64 from the same
// FP32 face states (exact conversions).  Only the repair kernels call it, for
// the faces the FP32 solver declined; the step kernels hold no FP64 HLLD code,
// which would raise their register count (a 64-register 2D step kernel went
// to 126) or spill inside their hot loops.  Out of line, states and flux by
// value.
struct HlldFlux32
{
  float f[6];
};
template <int NF>
__device__ __noinline__ HlldFlux32
mhd_hlld_f64_island(float4 l0, float4 l1, float4 r0, float4 r1, float gamma0)
{
  double l[8] = { f2d(l0.x), f2d(l0.y), f2d(l0.z), f2d(l0.w), f2d(l1.x), f2d(l1.y), f2d(l1.z), f2d(l1.w) };
  double r[8] = { f2d(r0.x), f2d(r0.y), f2d(r0.z), f2d(r0.w), f2d(r1.x), f2d(r1.y), f2d(r1.z), f2d(r1.w) };
  double f[NF];
  mhd_hlld<double, NF>(l, r, f, f2d(gamma0), 1.0 / (f2d(gamma0) - 1.0));
  HlldFlux32 out;
#pragma unroll
  for (int i = 0; i < 6; ++i)
    out.f[i] = i < NF ? d2f_rn(f[i < NF ? i : 0]) : 0.f;
  return out;
}
template <int NF>
__device__ __forceinline__ void
mhd_hlld_f64_from_f32(const float (&ql)[8], const float (&qr)[8], float (&flux)[NF], float gamma0)
{
  const HlldFlux32 o = mhd_hlld_f64_island<NF>(make_float4(ql[0], ql[1], ql[2], ql[3]), make_float4(ql[4], ql[5], ql[6], ql[7]),
                                               make_float4(qr[0], qr[1], qr[2], qr[3]), make_float4(qr[4], qr[5], qr[6], qr[7]),
                                               gamma0);
#pragma unroll
  for (int i = 0; i < NF; ++i)
    flux[i] = o.f[i];
}

template <class R>
__device__ __forceinline__ R
fmax4(R a0, R a1, R a2, R a3)
{
  R r = a0;
  r = (a1 > r) ? a1 : r;
  r = (a2 > r) ? a2 : r;
  r = (a3 > r) ? a3 : r;
  return r;
}
template <class R>
__device__ __forceinline__ R
fmin4(R a0, R a1, R a2, R a3)
{
  R r = a0;
  r = (a1 < r) ? a1 : r;
  r = (a2 < r) ? a2 : r;
  r = (a3 < r) ? a3 : r;
  return r;
}
template <class R>
__device__ __forceinline__ R
fmax5(R a0, R a1, R a2, R a3, R a4)
{
  R r = a0;
  r = (a1 > r) ? a1 : r;
  r = (a2 > r) ? a2 : r;
  r = (a3 > r) ? a3 : r;
  r = (a4 > r) ? a4 : r;
  return r;
}

// The parallel-plane state of one edge corner as mag_riemann2d_hlld reads
// it: density, pressure, two parallel velocities, two parallel fields and the
// orthogonal field (compute_emf, RiemannSolvers_MHD.h:648-860).
template <class R>
struct EdgeQ
{
  R r, p, u, v, a, b, c;
};

// mag_riemann2d_hlld in FP32 for the mixed form, in the algebra of the FP64 FMA
// build's (below), with the left and right corners of a row in the lanes of
// packed pairs (rows LL, RL and LR, RR; a is the same along a row, b along a
// column).  The discriminant of the fast speed is taken as (B^2 - gamma p)^2 / 4
// + gamma p Bt^2, which does not cancel.  26 special-function instructions, and of
// the five cases only the one sampled.  Issue bounds the
// kernels that call it (62 to 68 % busy): with the HLLD fluxes' algebra above,
// update kernel at 256^3 2605 -> 2524 us, 2D step at 2048^2 495 -> 483 us.  Speeds
// are formed from quotients by the density (a step at 256^3 3.84 -> 3.85 ms, at
// 2048^2 503 -> 506 us against squares of pressures and products with densities,
// which overflow and underflow where speeds do not).
__device__ __forceinline__ float
mag_riemann2d_hlld_f32(const EdgeQ<float> & LL, const EdgeQ<float> & RL, const EdgeQ<float> & LR,
                       const EdgeQ<float> & RR, float gamma0, float smallc)
{
  const float  a0 = LL.a, a1 = LR.a, a02 = a0 * a0, a12 = a1 * a1;
  const float2 b = f2(LL.b, RL.b), bb = mul2(b, b);
  struct Row
  {
    float2 r, u, v, pt, ir;
  };
  float cx = 0.f, cy = 0.f; // squares of the largest fast speeds along x and y
  auto  row = [&](const EdgeQ<float> & l, const EdgeQ<float> & r, float a2) {
    Row w;
    w.r = f2(l.r, r.r), w.u = f2(l.u, r.u), w.v = f2(l.v, r.v);
    const float2 p = f2(l.p, r.p), c = f2(l.c, r.c), c2 = mul2(c, c);
    const float2 btx = add2(c2, bb), bty = add2(c2, f2s(a2)), b2 = add2(btx, f2s(a2)); // transverse to x, to y; B^2
    // over the density first, as in mhd_hlld_f32
    const float2 ir = f2(rcp_a(w.r.x), rcp_a(w.r.y)), g = mul2(mul2(f2s(gamma0), p), ir);
    w.ir = ir;
    const float2 h = mul2(f2s(0.5f), fma2(b2, ir, g)), m = sub2(h, g), mm = mul2(m, m), gr = mul2(g, ir);
    const float2 dx = fma2(gr, btx, mm), dy = fma2(gr, bty, mm);
    const float2 fx = add2(h, f2(sqrt_a(dx.x), sqrt_a(dx.y))), fy = add2(h, f2(sqrt_a(dy.x), sqrt_a(dy.y)));
    cx = fmaxf(cx, fmaxf(fx.x, fx.y));
    cy = fmaxf(cy, fmaxf(fy.x, fy.y));
    w.pt = fma2(f2s(0.5f), b2, p);
    return w;
  };
  const Row   B = row(LL, RL, a02), T = row(LR, RR, a12);
  const float cmx = sqrt_a(cx), cmy = sqrt_a(cy);
  const float SL = fminf(fminf(B.u.x, B.u.y), fminf(T.u.x, T.u.y)) - cmx;
  const float SR = fmaxf(fmaxf(B.u.x, B.u.y), fmaxf(T.u.x, T.u.y)) + cmx;
  const float SB = fminf(fminf(B.v.x, B.v.y), fminf(T.v.x, T.v.y)) - cmy;
  const float ST = fmaxf(fmaxf(B.v.x, B.v.y), fmaxf(T.v.x, T.v.y)) + cmy;

  // distances of the corner velocities from the outer waves (positive)
  const float2 sgn = f2(1.f, -1.f), S = f2(-SL, SR);
  const float2 xB = fma2(B.u, sgn, S), xT = fma2(T.u, sgn, S);
  const float2 yB = add2(B.v, f2s(-SB)), yT = fma2(T.v, f2s(-1.f), f2s(ST));
  const float2 wB = mul2(B.r, xB), wT = mul2(T.r, xT), ps = add2(B.pt, T.pt), pd = sub2(B.pt, T.pt);
  const float2 un = fma2(wB, B.u, mul2(wT, T.u)), ud = add2(wB, wT);
  const float  us = (un.x + un.y + (ps.x - ps.y)) * rcp_a(ud.x + ud.y);
  const float2 zB = mul2(B.r, yB), zT = mul2(T.r, yT);
  const float2 vn = fma2(zB, B.v, mul2(zT, T.v)), vd = add2(zB, zT);
  const float  vs = (vn.x + vn.y + (pd.x + pd.y)) * rcp_a(vd.x + vd.y);
  const float2 iX = f2(rcp_a(us - SL), rcp_a(SR - us));
  const float  iB = rcp_a(vs - SB), iT = rcp_a(ST - vs);
  const float2 fxB = mul2(xB, iX), fxT = mul2(xT, iX), fyB = mul2(yB, f2s(iB)), fyT = mul2(yT, f2s(iT));

  // The larger Alfven speed of two corners: sqrt(max(n1 / d1, n2 / d2)), the
  // quotients compared by products, with n and d over the smallest density: n is a
  // speed's square, not a field's (a field of 1e-19 is an ordinary foot of a
  // magnetised region, its square is not among FP32's normal numbers) and d at least
  // about one.  Where n d is below 1e-36 the speed, under 1e-18, is taken as n 1e18.
  const float s = fmaxf(fmaxf(B.ir.x, B.ir.y), fmaxf(T.ir.x, T.ir.y));
  auto larger = [smallc](float n1, float d1, float n2, float d2) {
    const bool  first = n1 * d2 >= n2 * d1;
    const float n = first ? n1 : n2, d = first ? d1 : d2;
    return fmaxf(n * rsqrt_a(fmaxf(n * d, 1e-36f)), smallc);
  };
  const float2 sX = mul2(iX, f2s(s)), bs = mul2(mul2(b, f2s(s)), b);
  const float  sB = iB * s, sT = iT * s, as0 = a0 * s * a0, as1 = a1 * s * a1;
  const float2 dxB = mul2(wB, sX), dxT = mul2(wT, sX), dyB = mul2(zB, f2s(sB)), dyT = mul2(zT, f2s(sT));
  const float  cL = larger(as1 * fmaxf(fyT.x, 1.f), dxT.x, as0 * fmaxf(fyB.x, 1.f), dxB.x);
  const float  cR = larger(as1 * fmaxf(fyT.y, 1.f), dxT.y, as0 * fmaxf(fyB.y, 1.f), dxB.y);
  const float  cB = larger(bs.x * fmaxf(fxB.x, 1.f), dyB.x, bs.y * fmaxf(fxB.y, 1.f), dyB.y);
  const float  cT = larger(bs.x * fmaxf(fxT.x, 1.f), dyT.x, bs.y * fmaxf(fxT.y, 1.f), dyT.y);
  const float  SAL = fminf(us - cL, 0.f), SAR = fmaxf(us + cR, 0.f);
  const float  SAB = fminf(vs - cB, 0.f), SAT = fmaxf(vs + cT, 0.f);

  const bool SLp = !signbit(SL), SRp = !signbit(SR), SBp = !signbit(SB), STp = !signbit(ST);
  if (SBp || !STp)
  {
    // supersonic along y: the x fan of the corners on that side
    const float2 u = SBp ? B.u : T.u, v = SBp ? B.v : T.v, fx = SBp ? fxB : fxT;
    const float  a = SBp ? a0 : a1;
    if (SLp || !SRp)
      return SLp ? u.x * b.x - v.x * a : u.y * b.y - v.y * a;
    const float El = us * (b.x * fx.x) - v.x * a, Er = us * (b.y * fx.y) - v.y * a;
    return (SAR * El - SAL * Er + SAR * SAL * (b.y - b.x)) * rcp_a(SAR - SAL);
  }
  if (SLp || !SRp)
  {
    const float uB = SLp ? B.u.x : B.u.y, uT = SLp ? T.u.x : T.u.y, fB = SLp ? fyB.x : fyB.y, fT = SLp ? fyT.x : fyT.y;
    const float bs = SLp ? b.x : b.y;
    const float Eb = uB * bs - vs * (a0 * fB), Et = uT * bs - vs * (a1 * fT);
    return (SAT * Eb - SAB * Et - SAT * SAB * (a1 - a0)) * rcp_a(SAT - SAB);
  }
  const float2 AB = mul2(f2s(a0), fyB), AT = mul2(f2s(a1), fyT), BB = mul2(b, fxB), BT = mul2(b, fxT);
  const float2 EB = fma2(f2s(us), BB, mul2(f2s(-vs), AB)), ET = fma2(f2s(us), BT, mul2(f2s(-vs), AT));
  const float2 e = fma2(f2s(SAB), ET, mul2(f2s(-SAT), EB)), dA = sub2(AT, AB);
  const float  dB = SAT * (BT.y - BT.x) - SAB * (BB.y - BB.x);
  const float  m = SAL * e.y - SAR * e.x - SAT * SAB * (SAR * dA.y - SAL * dA.x) + SAR * SAL * dB;
  return m * (rcp_a(SAR - SAL) * rcp_a(SAT - SAB));
}

// mag_riemann2d_hlld (RiemannSolvers_MHD.h:395-627) in the FP64 FMA build: the
// same emf with about 300 FP64-pipe operations per edge.  a is the same at
// the two corners of a row (LL, RL and LR, RR), b at the two of a column.  With
// fx = (S - u) / (S - u*), fy likewise, rho*, A* and B* are products, and the two
// Alfven speeds of a corner, |a| / sqrt(rho fx) and |A*| / sqrt(rho fx fy), are
// the root of a^2 max(1, fy) / (rho fx): the larger of two corners' quotients is
// chosen by products, so a side takes one reciprocal root instead of four.  Of
// the five cases only the one sampled is computed.
__device__ __forceinline__ double
mag_riemann2d_hlld64(const EdgeQ<double> & LL, const EdgeQ<double> & RL, const EdgeQ<double> & LR,
                     const EdgeQ<double> & RR, double gamma0, double smallc)
{
  const double a0 = LL.a, a1 = LR.a, b0 = LL.b, b1 = RL.b;
  const double a02 = a0 * a0, a12 = a1 * a1, b02 = b0 * b0, b12 = b1 * b1;
  // total pressure; squares of the fast speeds along x and y
  long long cx = 0, cy = 0;
  auto      corner = [&](const EdgeQ<double> & q, double a2, double b2) {
    const double s = fma(q.c, q.c, a2 + b2), g = gamma0 * q.p, ir = rcp64(q.r);
    cx = max(cx, __double_as_longlong(fast_num64(g, s, a2) * ir));
    cy = max(cy, __double_as_longlong(fast_num64(g, s, b2) * ir));
    return q.p + scale_pos64<1>(s);
  };
  const double PLL = corner(LL, a02, b02), PRL = corner(RL, a02, b12);
  const double PLR = corner(LR, a12, b02), PRR = corner(RR, a12, b12);
  const double cmx = sqrt64(__longlong_as_double(cx)), cmy = sqrt64(__longlong_as_double(cy));
  auto         lowest = [](double p, double q, double r, double s) {
    return from_order64(min(min(order64(p), order64(q)), min(order64(r), order64(s))));
  };
  auto highest = [](double p, double q, double r, double s) {
    return from_order64(max(max(order64(p), order64(q)), max(order64(r), order64(s))));
  };
  const double SL = lowest(LL.u, LR.u, RL.u, RR.u) - cmx, SR = highest(LL.u, LR.u, RL.u, RR.u) + cmx;
  const double SB = lowest(LL.v, LR.v, RL.v, RR.v) - cmy, ST = highest(LL.v, LR.v, RL.v, RR.v) + cmy;

  // distances of the corner velocities from the outer waves (positive)
  const double xLL = LL.u - SL, xLR = LR.u - SL, xRL = SR - RL.u, xRR = SR - RR.u;
  const double yLL = LL.v - SB, yRL = RL.v - SB, yLR = ST - LR.v, yRR = ST - RR.v;
  const double D1 = PLL - PRR, D2 = PLR - PRL;
  double       us, vs;
  {
    const double p = LL.r * xLL, q = LR.r * xLR, r = RL.r * xRL, s = RR.r * xRR;
    us = fma(p, LL.u, fma(q, LR.u, fma(r, RL.u, fma(s, RR.u, D1 + D2)))) * rcp64((p + q) + (r + s));
  }
  {
    const double p = LL.r * yLL, q = LR.r * yLR, r = RL.r * yRL, s = RR.r * yRR;
    vs = fma(p, LL.v, fma(q, LR.v, fma(r, RL.v, fma(s, RR.v, D1 - D2)))) * rcp64((p + q) + (r + s));
  }
  const double iL = rcp64(us - SL), iR = rcp64(SR - us), iB = rcp64(vs - SB), iT = rcp64(ST - vs);
  const double fxLL = xLL * iL, fxLR = xLR * iL, fxRL = xRL * iR, fxRR = xRR * iR;
  const double fyLL = yLL * iB, fyRL = yRL * iB, fyLR = yLR * iT, fyRR = yRR * iT;

  // the larger Alfven speed of two corners: sqrt(max(n1 m1 / d1, n2 m2 / d2)), m >= 1
  auto alfven = [&](double n1, double m1, double d1, double n2, double m2, double d2) {
    n1 *= max_floor64(m1, 1.0);
    n2 *= max_floor64(m2, 1.0);
    return max_floor64(sqrt_larger_ratio64(n1, d1, n2, d2), smallc);
  };
  const double cL = alfven(a12, fyLR, LR.r * fxLR, a02, fyLL, LL.r * fxLL);
  const double cR = alfven(a12, fyRR, RR.r * fxRR, a02, fyRL, RL.r * fxRL);
  const double cB = alfven(b02, fxLL, LL.r * fyLL, b12, fxRL, RL.r * fyRL);
  const double cT = alfven(b02, fxLR, LR.r * fyLR, b12, fxRR, RR.r * fyRR);
  auto         below = [](double x) { return negative64(x) ? x : 0.0; };
  auto         above = [](double x) { return negative64(x) ? 0.0 : x; };
  const double SAL = below(us - cL), SAR = above(us + cR), SAB = below(vs - cB), SAT = above(vs + cT);

  const bool SLp = !negative64(SL), SRp = !negative64(SR), SBp = !negative64(SB), STp = !negative64(ST);
  if (SBp || !STp)
  {
    // supersonic along y: the x fan of the corners on that side
    const EdgeQ<double> &l = SBp ? LL : LR, &r = SBp ? RL : RR;
    const double         b_l = l.b, b_r = r.b;
    if (SLp || !SRp)
      return SLp ? l.u * l.b - l.v * l.a : r.u * r.b - r.v * r.a;
    const double El = us * (b_l * (SBp ? fxLL : fxLR)) - l.v * l.a, Er = us * (b_r * (SBp ? fxRL : fxRR)) - r.v * r.a;
    return (SAR * El - SAL * Er + SAR * SAL * (b_r - b_l)) * rcp64(SAR - SAL);
  }
  if (SLp || !SRp)
  {
    const EdgeQ<double> &b = SLp ? LL : RL, &t = SLp ? LR : RR;
    const double         Eb = b.u * b.b - vs * (b.a * (SLp ? fyLL : fyRL)), Et = t.u * t.b - vs * (t.a * (SLp ? fyLR : fyRR));
    return (SAT * Eb - SAB * Et - SAT * SAB * (t.a - b.a)) * rcp64(SAT - SAB);
  }
  const double ALL = a0 * fyLL, ARL = a0 * fyRL, ALR = a1 * fyLR, ARR = a1 * fyRR;
  const double BLL = b0 * fxLL, BLR = b0 * fxLR, BRL = b1 * fxRL, BRR = b1 * fxRR;
  const double ELL = us * BLL - vs * ALL, ERL = us * BRL - vs * ARL;
  const double ELR = us * BLR - vs * ALR, ERR = us * BRR - vs * ARR;
  const double e1 = SAB * ERR - SAT * ERL, e2 = SAB * ELR - SAT * ELL;
  const double dA = SAR * (ARR - ARL) - SAL * (ALR - ALL), dB = SAT * (BRR - BLR) - SAB * (BRL - BLL);
  const double e = fma(SAR * SAL, dB, fma(-(SAT * SAB), dA, SAL * e1 - SAR * e2));
  return e * (rcp64(SAR - SAL) * rcp64(SAT - SAB));
}

// mag_riemann2d_hlld (RiemannSolvers_MHD.h:395-627); corners LL, RL, LR, RR
template <class R>
__device__ __forceinline__ R
mag_riemann2d_hlld(const EdgeQ<R> & LL, const EdgeQ<R> & RL, const EdgeQ<R> & LR,
                   const EdgeQ<R> & RR, R ELL, R ERL, R ELR, R ERR, R gamma0, R smallc)
{
  if constexpr (sizeof(R) == 4)
    return mag_riemann2d_hlld_f32(LL, RL, LR, RR, gamma0, smallc);
  else if constexpr (kFast64<R>)
    return mag_riemann2d_hlld64(LL, RL, LR, RR, gamma0, smallc);
  else
  {
  // fast speed of a corner state along x or y
  auto fast = [gamma0](const EdgeQ<R> & q, bool ydir) {
    const R b2 = q.a * q.a + q.b * q.b + q.c * q.c;
    const R bn = ydir ? q.b : q.a;
    const R c2 = gamma0 * q.p / q.r;
    const R d2 = R(0.5) * (b2 / q.r + c2);
    return sqrt(d2 + sqrt(d2 * d2 - c2 * bn * bn / q.r));
  };
  const R rLL = LL.r, pLL = LL.p, uLL = LL.u, vLL = LL.v, aLL = LL.a, bLL = LL.b, cLL = LL.c;
  const R rLR = LR.r, pLR = LR.p, uLR = LR.u, vLR = LR.v, aLR = LR.a, bLR = LR.b, cLR = LR.c;
  const R rRL = RL.r, pRL = RL.p, uRL = RL.u, vRL = RL.v, aRL = RL.a, bRL = RL.b, cRL = RL.c;
  const R rRR = RR.r, pRR = RR.p, uRR = RR.u, vRR = RR.v, aRR = RR.a, bRR = RR.b, cRR = RR.c;

  const R cFastLLx = fast(LL, false), cFastLRx = fast(LR, false);
  const R cFastRLx = fast(RL, false), cFastRRx = fast(RR, false);
  const R cFastLLy = fast(LL, true), cFastLRy = fast(LR, true);
  const R cFastRLy = fast(RL, true), cFastRRy = fast(RR, true);

  const R cmx = fmax4(cFastLLx, cFastLRx, cFastRLx, cFastRRx), cmy = fmax4(cFastLLy, cFastLRy, cFastRLy, cFastRRy);
  const R SL = fmin4(uLL, uLR, uRL, uRR) - cmx;
  const R SR = fmax4(uLL, uLR, uRL, uRR) + cmx;
  const R SB = fmin4(vLL, vLR, vRL, vRR) - cmy;
  const R ST = fmax4(vLL, vLR, vRL, vRR) + cmy;

  const R PtotLL = pLL + R(0.5) * (aLL * aLL + bLL * bLL + cLL * cLL);
  const R PtotLR = pLR + R(0.5) * (aLR * aLR + bLR * bLR + cLR * cLR);
  const R PtotRL = pRL + R(0.5) * (aRL * aRL + bRL * bRL + cRL * cRL);
  const R PtotRR = pRR + R(0.5) * (aRR * aRR + bRR * bRR + cRR * cRR);

  const R rcLLx = rLL * (uLL - SL);
  const R rcRLx = rRL * (SR - uRL);
  const R rcLRx = rLR * (uLR - SL);
  const R rcRRx = rRR * (SR - uRR);
  const R rcLLy = rLL * (vLL - SB);
  const R rcLRy = rLR * (ST - vLR);
  const R rcRLy = rRL * (vRL - SB);
  const R rcRRy = rRR * (ST - vRR);

  const R ustar =
    (rcLLx * uLL + rcLRx * uLR + rcRLx * uRL + rcRRx * uRR + (PtotLL - PtotRL + PtotLR - PtotRR)) /
    (rcLLx + rcLRx + rcRLx + rcRRx);
  const R vstar =
    (rcLLy * vLL + rcLRy * vLR + rcRLy * vRL + rcRRy * vRR + (PtotLL - PtotLR + PtotRL - PtotRR)) /
    (rcLLy + rcLRy + rcRLy + rcRRy);

  const R dSLu = SL - ustar, dSRu = SR - ustar, dSBv = SB - vstar, dSTv = ST - vstar;
  auto q_SLu = [&](R x) { return x / dSLu; };
  auto q_SRu = [&](R x) { return x / dSRu; };
  auto q_SBv = [&](R x) { return x / dSBv; };
  auto q_STv = [&](R x) { return x / dSTv; };
  const R rstarLLx = q_SLu(rLL * (SL - uLL));
  const R BstarLL = q_SLu(bLL * (SL - uLL));
  const R rstarLLy = q_SBv(rLL * (SB - vLL));
  const R AstarLL = q_SBv(aLL * (SB - vLL));
  const R rstarLL = q_SBv(q_SLu(rLL * (SL - uLL)) * (SB - vLL));
  const R EstarLLx = ustar * BstarLL - vLL * aLL;
  const R EstarLLy = uLL * bLL - vstar * AstarLL;
  const R EstarLL = ustar * BstarLL - vstar * AstarLL;

  const R rstarLRx = q_SLu(rLR * (SL - uLR));
  const R BstarLR = q_SLu(bLR * (SL - uLR));
  const R rstarLRy = q_STv(rLR * (ST - vLR));
  const R AstarLR = q_STv(aLR * (ST - vLR));
  const R rstarLR = q_STv(q_SLu(rLR * (SL - uLR)) * (ST - vLR));
  const R EstarLRx = ustar * BstarLR - vLR * aLR;
  const R EstarLRy = uLR * bLR - vstar * AstarLR;
  const R EstarLR = ustar * BstarLR - vstar * AstarLR;

  const R rstarRLx = q_SRu(rRL * (SR - uRL));
  const R BstarRL = q_SRu(bRL * (SR - uRL));
  const R rstarRLy = q_SBv(rRL * (SB - vRL));
  const R AstarRL = q_SBv(aRL * (SB - vRL));
  const R rstarRL = q_SBv(q_SRu(rRL * (SR - uRL)) * (SB - vRL));
  const R EstarRLx = ustar * BstarRL - vRL * aRL;
  const R EstarRLy = uRL * bRL - vstar * AstarRL;
  const R EstarRL = ustar * BstarRL - vstar * AstarRL;

  const R rstarRRx = q_SRu(rRR * (SR - uRR));
  const R BstarRR = q_SRu(bRR * (SR - uRR));
  const R rstarRRy = q_STv(rRR * (ST - vRR));
  const R AstarRR = q_STv(aRR * (ST - vRR));
  const R rstarRR = q_STv(q_SRu(rRR * (SR - uRR)) * (ST - vRR));
  const R EstarRRx = ustar * BstarRR - vRR * aRR;
  const R EstarRRy = uRR * bRR - vstar * AstarRR;
  const R EstarRR = ustar * BstarRR - vstar * AstarRR;

  auto b_over_sqrt = [](R b, R r) { return fabs(b) / sqrt(r); };
  const R calfvenL = fmax5(b_over_sqrt(aLR, rstarLRx), b_over_sqrt(AstarLR, rstarLR),
                           b_over_sqrt(aLL, rstarLLx), b_over_sqrt(AstarLL, rstarLL), smallc);
  const R calfvenR = fmax5(b_over_sqrt(aRR, rstarRRx), b_over_sqrt(AstarRR, rstarRR),
                           b_over_sqrt(aRL, rstarRLx), b_over_sqrt(AstarRL, rstarRL), smallc);
  const R calfvenB = fmax5(b_over_sqrt(bLL, rstarLLy), b_over_sqrt(BstarLL, rstarLL),
                           b_over_sqrt(bRL, rstarRLy), b_over_sqrt(BstarRL, rstarRL), smallc);
  const R calfvenT = fmax5(b_over_sqrt(bLR, rstarLRy), b_over_sqrt(BstarLR, rstarLR),
                           b_over_sqrt(bRR, rstarRRy), b_over_sqrt(BstarRR, rstarRR), smallc);

  const R SAL = fmin(ustar - calfvenL, R(0));
  const R SAR = fmax(ustar + calfvenR, R(0));
  const R SAB = fmin(vstar - calfvenB, R(0));
  const R SAT = fmax(vstar + calfvenT, R(0));
  const R dA = SAR - SAL, dB = SAT - SAB;
  auto q_A = [&](R x) { return x / dA; };
  auto q_B = [&](R x) { return x / dB; };

  const R AstarT = q_A(SAR * AstarRR - SAL * AstarLR);
  const R AstarB = q_A(SAR * AstarRL - SAL * AstarLL);
  const R BstarR = q_B(SAT * BstarRR - SAB * BstarRL);
  const R BstarL = q_B(SAT * BstarLR - SAB * BstarLL);

  R       E = 0, tmpE = 0;
  const int SB_pos = (int)(1 + copysign(R(1), SB)) / 2, SB_neg = 1 - SB_pos;
  const int ST_pos = (int)(1 + copysign(R(1), ST)) / 2, ST_neg = 1 - ST_pos;
  const int SL_pos = (int)(1 + copysign(R(1), SL)) / 2, SL_neg = 1 - SL_pos;
  const int SR_pos = (int)(1 + copysign(R(1), SR)) / 2, SR_neg = 1 - SR_pos;

  tmpE = q_B(q_A(SAL * SAB * EstarRR - SAL * SAT * EstarRL - SAR * SAB * EstarLR + SAR * SAT * EstarLL)) -
         q_B(SAT * SAB) * (AstarT - AstarB) + q_A(SAR * SAL) * (BstarR - BstarL);
  E += (R)(SB_neg * ST_pos * SL_neg * SR_pos) * tmpE;

  tmpE = q_A(SAR * EstarLLx - SAL * EstarRLx + SAR * SAL * (bRL - bLL));
  tmpE = (R)SL_pos * ELL + (R)(SL_neg * SR_neg) * ERL + (R)(SL_neg * SR_pos) * tmpE;
  E += (R)SB_pos * tmpE;

  tmpE = q_A(SAR * EstarLRx - SAL * EstarRRx + SAR * SAL * (bRR - bLR));
  tmpE = (R)SL_pos * ELR + (R)(SL_neg * SR_neg) * ERR + (R)(SL_neg * SR_pos) * tmpE;
  E += (R)(SB_neg * ST_neg) * tmpE;

  tmpE = q_B(SAT * EstarLLy - SAB * EstarLRy - SAT * SAB * (aLR - aLL));
  E += (R)(SB_neg * ST_pos * SL_pos) * tmpE;

  tmpE = q_B(SAT * EstarRLy - SAB * EstarRRy - SAT * SAB * (aRR - aRL));
  E += (R)(SB_neg * ST_pos * SL_neg * SR_neg) * tmpE;
  return E;
  }
}

// compute_emf<emfDir> (RiemannSolvers_MHD.h:648-871) on the four corner
// states of an edge.  Each corner carries the components compute_emf reads
// for the edge direction: the velocities and face fields along the two
// transverse directions (u, a along the first, v, b along the second) and the
// field along the edge (c).
template <class R>
struct EdgeCorner
{
  R r, p, u, v, a, b, c;
};

template <class R>
__device__ __forceinline__ R
mhd_emf_corners(const EdgeCorner<R> & RT, const EdgeCorner<R> & RB, const EdgeCorner<R> & LT,
                const EdgeCorner<R> & LB, R gamma0, R smallc)
{
  EdgeQ<R> LL, RL, LR, RR;
  LL.r = RT.r, RL.r = LT.r, LR.r = RB.r, RR.r = LB.r;
  LL.p = RT.p, RL.p = LT.p, LR.p = RB.p, RR.p = LB.p;
  LL.u = RT.u, RL.u = LT.u, LR.u = RB.u, RR.u = LB.u;
  LL.v = RT.v, RL.v = LT.v, LR.v = RB.v, RR.v = LB.v;
  auto half = [](R x) {
    if constexpr (kFast64<R>)
      return half64(x);
    else
      return R(0.5) * x;
  };
  LL.a = RL.a = half(RT.a + LT.a);
  LR.a = RR.a = half(RB.a + LB.a);
  LL.b = LR.b = half(RT.b + RB.b);
  RL.b = RR.b = half(LT.b + LB.b);
  LL.c = RT.c, RL.c = LT.c, LR.c = RB.c, RR.c = LB.c;
  const R ELL = LL.u * LL.b - LL.v * LL.a;
  const R ERL = RL.u * RL.b - RL.v * RL.a;
  const R ELR = LR.u * LR.b - LR.v * LR.a;
  const R ERR = RR.u * RR.b - RR.v * RR.a;
  return mag_riemann2d_hlld<R>(LL, RL, LR, RR, ELL, ERL, ELR, ERR, gamma0, smallc);
}

// -------------------------------------------------------------------------
// Compact trace.  trace_unsplit_mhd_3d_simpler (MHDBaseFunctor3D.h:690-1114)
// produces 6 face states and 12 edge states per cell, all of them simple
// combinations of 47 per-cell numbers: the time-advanced cell-centred state
// and face fields, and the half slopes.  The trace kernel stores those 47
// numbers; the flux/emf kernel rebuilds any face or edge state from them with
// the reference's own expressions, so the result is bit-identical.
// -------------------------------------------------------------------------
enum : int
{
  T_R = 0, T_P, T_U, T_V, T_W, T_A, T_B, T_C,            // advanced cell state
  T_AL, T_AR, T_BL, T_BR, T_CL, T_CR,                    // advanced face fields
  T_DRX, T_DPX, T_DUX, T_DVX, T_DWX, T_DBX, T_DCX,       // half slopes along x
  T_DRY, T_DPY, T_DUY, T_DVY, T_DWY, T_DAY, T_DCY,       // along y
  T_DRZ, T_DPZ, T_DUZ, T_DVZ, T_DWZ, T_DAZ, T_DBZ,       // along z
  T_DALY, T_DALZ, T_DBLX, T_DBLZ, T_DCLX, T_DCLY,        // face-field half slopes
  T_DARY, T_DARZ, T_DBRX, T_DBRZ, T_DCRX, T_DCRY,
  T_N
};

template <class R>
__device__ __forceinline__ void
floor_state(R (&q)[8], R smallr, R smallp)
{
  if constexpr (kFast64<R>)
  {
    q[ID] = max_floor64(q[ID], smallr);
    q[IP] = max_floor64(q[IP], smallp);
    return;
  }
  q[ID] = fmax(smallr, q[ID]);
  q[IP] = fmax(smallp, q[IP]);
}

// Trace field indices as functions of a direction (0 x, 1 y, 2 z), so one
// code path serves the faces and edges of every direction:
//   hydro half slope of variable f (T_R..T_W) along e
//   half slope of the cell-centred field f along e (f != e)
//   face value of field f on the left (0) / right (1) face
//   half slope of that face value along e (e != f)
__device__ __forceinline__ int
t_hslope(int e, int f)
{
  return T_DRX + 7 * e + f;
}
__device__ __forceinline__ int
t_bslope(int e, int f)
{
  return T_DRX + 7 * e + 5 + (f < e ? f : f - 1);
}
__device__ __forceinline__ int
t_bface(int f, int right)
{
  return T_AL + 2 * f + right;
}
__device__ __forceinline__ int
t_bfslope(int f, int right, int e)
{
  return T_DALY + 6 * right + 2 * f + (e < f ? e : e - 1);
}

// Accessors of a cell's trace fields: A(f) is field f.
// StrideAcc: field-major storage with stride st (the staged shared-memory
// planes, the slabs of the FP64 passes).  QuadAcc: the HBM trace, 16-byte quads of fields per cell (see
// trace_cell); the gathers below read compile-time field indices, so only the
// quads a face or edge state needs are loaded (the others are never used and
// their loads are removed), one vector load per quad.
template <class R, class I>
struct StrideAcc
{
  const R * t;
  I         st;
  __device__ __forceinline__ R
  operator()(int f) const
  {
    return t[ekc::field_offset(f, st)];
  }
};
constexpr int kTraceLanes = 32; // cells per block of the HBM trace
template <class R>
using TVec = typename std::conditional<sizeof(R) == 4, float4, double2>::type;
template <class R>
constexpr int kTVecN = 16 / (int)sizeof(R); // fields per quad
template <class R>
constexpr int kTQuads = (T_N + kTVecN<R> - 1) / kTVecN<R>; // quads per cell
template <class R>
struct QuadAcc
{
  TVec<R> v[kTQuads<R>];
  __device__ __forceinline__ explicit QuadAcc(const R * t)
  {
#pragma unroll
    for (int q = 0; q < kTQuads<R>; ++q)
      v[q] = __ldg(reinterpret_cast<const TVec<R> *>(t + q * kTraceLanes * kTVecN<R>));
  }
  __device__ __forceinline__ R
  operator()(int f) const
  {
    const TVec<R> & x = v[f / kTVecN<R>];
    if constexpr (sizeof(R) == 4)
    {
      const int c = f % 4;
      return c == 0 ? x.x : (c == 1 ? x.y : (c == 2 ? x.z : x.w));
    }
    else
      return f % 2 == 0 ? x.x : x.y;
  }
};

// Face state of a cell on its face normal to d (PLUS: the right face, the
// left state of that face), in the face frame the flux functor hands to the
// Riemann solver: normal velocity in IU and normal field in IA, with the
// reference's component swaps for y (IU<->IV, IA<->IB) and z (IU<->IW,
// IA<->IC) faces (trace_unsplit_mhd_3d_simpler, MHDBaseFunctor3D.h:905-955;
// MHDRunFunctors3D.h:1839-1874).
template <class R, bool PLUS, class ACC>
__device__ __forceinline__ void
face_state_acc(const ACC & T, int d, R (&q)[8], R smallr, R smallp)
{
  auto h = [&](int f) {
    const R c = T(f), s = T(t_hslope(d, f));
    return PLUS ? c + s : c - s;
  };
  auto tb = [&](int f) {
    const R c = T(T_A + f), s = T(t_bslope(d, f));
    return PLUS ? c + s : c - s;
  };
  q[ID] = h(T_R);
  q[IP] = h(T_P);
  q[IU] = h(T_U + d);
  q[IV] = h(d == 1 ? T_U : T_V);
  q[IW] = h(d == 2 ? T_U : T_W);
  q[IA] = T(t_bface(d, PLUS ? 1 : 0));
  q[IB] = tb(d == 1 ? 0 : 1);
  q[IC] = tb(d == 2 ? 0 : 2);
  floor_state(q, smallr, smallp);
}
template <class R, bool PLUS, class I>
__device__ __forceinline__ void
face_state_dir(const R * t, I st, int d, R (&q)[8], R smallr, R smallp)
{
  face_state_acc<R, PLUS>(StrideAcc<R, I>{ t, st }, d, q, smallr, smallp);
}

// One corner of an edge along d (MHDBaseFunctor3D.h:957-1113).  The
// transverse directions are p1 = (d+1)%3 and p2 = (d+2)%3, the order in which
// compute_emf<emfDir> reads them; S1/S2 are the sides (+1 right, -1 left) of
// the corner along p1/p2.  Each sum keeps the reference's operands, so the
// result is bit-identical to the per-direction expressions.
template <class R, int S1, int S2, class ACC>
__device__ __forceinline__ EdgeCorner<R>
edge_corner_acc(const ACC & T, int d, int p1, int p2, R smallr, R smallp)
{
  auto sg1 = [](R x) { return S1 > 0 ? x : -x; };
  auto sg2 = [](R x) { return S2 > 0 ? x : -x; };
  auto hyd = [&](int f) { return T(f) + (sg1(T(t_hslope(p1, f))) + sg2(T(t_hslope(p2, f)))); };
  EdgeCorner<R> e;
  if constexpr (kFast64<R>)
  {
    e.r = max_floor64(hyd(T_R), smallr);
    e.p = max_floor64(hyd(T_P), smallp);
  }
  else
  {
    e.r = fmax(smallr, hyd(T_R));
    e.p = fmax(smallp, hyd(T_P));
  }
  e.u = hyd(T_U + p1);
  e.v = hyd(T_U + p2);
  e.a = T(t_bface(p1, S1 > 0)) + sg2(T(t_bfslope(p1, S1 > 0, p2)));
  e.b = T(t_bface(p2, S2 > 0)) + sg1(T(t_bfslope(p2, S2 > 0, p1)));
  e.c = T(T_A + d) + (sg1(T(t_bslope(p1, d))) + sg2(T(t_bslope(p2, d))));
  return e;
}
template <class R, int S1, int S2, class I>
__device__ __forceinline__ EdgeCorner<R>
edge_corner(const R * t, I st, int d, int p1, int p2, R smallr, R smallp)
{
  return edge_corner_acc<R, S1, S2>(StrideAcc<R, I>{ t, st }, d, p1, p2, smallr, smallp);
}

} // namespace EK_NS
