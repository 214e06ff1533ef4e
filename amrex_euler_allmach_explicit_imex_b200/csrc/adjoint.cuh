// Reverse-mode derivatives of one face of the explicit step (adjoint.cu).
//
// A face flux F(l, r) of euler_fv_one_step and its transposed Jacobian: given
// the cotangent of the flux, the cotangents of the two face states.  Branches
// (limiter cases, Riemann fallbacks, upwind side, std::min/max) are taken on
// the values the forward step takes them on, so the result is the derivative
// of the branch the forward took.  States and fluxes are in the face frame:
// density, normal velocity, tangential velocity, pressure.  Formulas and
// branch order follow the reference lines cited at each function (paths
// relative to amrex/apps/euler_compare/src/euler_compare/).
#pragma once

#include <math.h>

#include "ecg.h"

namespace ecg_adj {

struct State {
  double rho, un, ut, p;
};
// A flux or conserved state in the face frame, or a cotangent of one.
struct Flux {
  double rho, mn, mt, E;
};

// limited_slope (core/state_primitives.hpp:57-91) of the one-sided differences
// a (behind) and b (ahead), with its partial derivatives.
struct Slope {
  double s, da, db;
};
__device__ __forceinline__ Slope limited(double a, double b, int lim)
{
  if (a * b <= 0.0) return Slope{0.0, 0.0, 0.0};
  if (lim == ECG_LIMITER_MC) {
    const double c = 0.5 * (a + b);
    Slope t = fabs(2.0 * a) < fabs(c) ? Slope{2.0 * a, 2.0, 0.0} : Slope{c, 0.5, 0.5};
    return fabs(t.s) < fabs(2.0 * b) ? t : Slope{2.0 * b, 0.0, 2.0};
  }
  if (lim == ECG_LIMITER_VANLEER) {
    const double d = a + b;
    if (fabs(d) <= 1.0e-14) return Slope{0.0, 0.0, 0.0};
    const double id = 1.0 / d, s = 2.0 * a * b * id;
    return Slope{s, (2.0 * b - s) * id, (2.0 * a - s) * id};
  }
  return fabs(a) < fabs(b) ? Slope{a, 1.0, 0.0} : Slope{b, 0.0, 1.0};
}

// Sound speed sqrt(g p / rho) and its partial derivatives (none at c = 0).
struct Sound {
  double c, drho, dp;
};
__device__ __forceinline__ Sound sound(double rho, double p, double g)
{
  const double ir = 1.0 / rho;
  const double c = sqrt(g * p * ir);
  const double h = c > 0.0 ? 0.5 * ir / c : 0.0;
  return Sound{c, -(c * c) * h, g * h};
}

// Adds to the cotangent `d` of a state q those of its physical flux
// (physical_flux, reconstruction_fluxes.hpp:66-74) and conserved values
// (to_conserved, state_primitives.hpp:113-117): f and u.
__device__ __forceinline__ void reverse_flux(const State& q, double inv_gm1, const Flux& f, const Flux& u, State& d)
{
  const double k = 0.5 * (q.un * q.un + q.ut * q.ut);
  const double E = q.p * inv_gm1 + q.rho * k;
  const double dE = u.E + f.E * q.un;
  d.rho += f.rho * q.un + f.mn * (q.un * q.un) + f.mt * (q.un * q.ut) + u.rho + u.mn * q.un + u.mt * q.ut + dE * k;
  d.un += f.rho * q.rho + f.mn * (2.0 * q.rho * q.un) + f.mt * (q.rho * q.ut) + f.E * (E + q.p) + u.mn * q.rho +
          dE * (q.rho * q.un);
  d.ut += f.mt * (q.rho * q.un) + u.mt * q.rho + dE * (q.rho * q.ut);
  d.p += f.mn + f.E * q.un + dE * inv_gm1;
}

// rusanov_flux, reconstruction_fluxes.hpp:82-92
__device__ __forceinline__ void reverse_rusanov(const State& l, const State& r, const Sound& sl, const Sound& sr,
                                                double inv_gm1, const Flux& w, State& dl, State& dr)
{
  const double vl = fabs(l.un) + sl.c, vr = fabs(r.un) + sr.c;
  const bool right = vl < vr;  // std::max
  const double h = 0.5 * (right ? vr : vl);
  const double El = l.p * inv_gm1 + 0.5 * l.rho * (l.un * l.un + l.ut * l.ut);
  const double Er = r.p * inv_gm1 + 0.5 * r.rho * (r.un * r.un + r.ut * r.ut);
  const double ds = -0.5 * (w.rho * (r.rho - l.rho) + w.mn * (r.rho * r.un - l.rho * l.un) +
                            w.mt * (r.rho * r.ut - l.rho * l.ut) + w.E * (Er - El));
  const Flux f{0.5 * w.rho, 0.5 * w.mn, 0.5 * w.mt, 0.5 * w.E};
  reverse_flux(l, inv_gm1, f, Flux{h * w.rho, h * w.mn, h * w.mt, h * w.E}, dl);
  reverse_flux(r, inv_gm1, f, Flux{-h * w.rho, -h * w.mn, -h * w.mt, -h * w.E}, dr);
  if (right) {
    dr.un += r.un < 0.0 ? -ds : ds;
    dr.rho += ds * sr.drho;
    dr.p += ds * sr.dp;
  } else {
    dl.un += l.un < 0.0 ? -ds : ds;
    dl.rho += ds * sl.drho;
    dl.p += ds * sl.dp;
  }
}

// hllc_flux, reconstruction_fluxes.hpp:151-210
__device__ __forceinline__ void reverse_hllc(const State& l, const State& r, const Sound& cl, const Sound& cr,
                                             double inv_gm1, const Flux& w, State& dl, State& dr)
{
  const bool sl_right = r.un - cr.c < l.un - cl.c, sr_right = l.un + cl.c < r.un + cr.c;  // std::min, std::max
  const double sl = sl_right ? r.un - cr.c : l.un - cl.c, sr = sr_right ? r.un + cr.c : l.un + cl.c;
  const bool sup_l = sl >= 0.0, sup_r = sr <= 0.0;
  const double al = l.rho * (sl - l.un), ar = r.rho * (sr - r.un);
  const double den = al - ar;
  bool degenerate = !(sl < sr);
  if (!degenerate && (sup_l || sup_r)) {
    if (sup_l) reverse_flux(l, inv_gm1, w, Flux{0.0, 0.0, 0.0, 0.0}, dl);
    else reverse_flux(r, inv_gm1, w, Flux{0.0, 0.0, 0.0, 0.0}, dr);
    return;
  }
  const double iden = 1.0 / den;
  const double sm = (r.p - l.p + al * l.un - ar * r.un) * iden;
  degenerate = degenerate || fabs(den) <= 1.0e-12 || fabs(sl - sm) <= 1.0e-12 || fabs(sr - sm) <= 1.0e-12;
  if (degenerate) {
    reverse_rusanov(l, r, cl, cr, inv_gm1, w, dl, dr);
    return;
  }
  const double ps = 0.5 * (l.p + al * (sm - l.un) + r.p + ar * (sm - r.un));
  const bool left = sm >= 0.0;
  const State q = left ? l : r;
  const double s = left ? sl : sr, a = left ? al : ar;
  const double inv = 1.0 / (s - sm);
  const double k = 0.5 * (q.un * q.un + q.ut * q.ut);
  const double E = q.p * inv_gm1 + q.rho * k;
  const double rs = a * inv;
  const double es = ((s - q.un) * E - q.p * q.un + ps * sm) * inv;
  // F = f(q) + s (U* - U), U* = (rs, rs sm, rs ut, es)
  double d_rs = s * (w.rho + w.mn * sm + w.mt * q.ut);
  double d_es = s * w.E;
  double d_sm = w.mn * s * rs;
  double d_s = w.rho * (rs - q.rho) + w.mn * (rs * sm - q.rho * q.un) + w.mt * (rs - q.rho) * q.ut + w.E * (es - E);
  State d{0.0, 0.0, w.mt * s * rs, 0.0};
  // es = ((s - un) E - p un + ps sm) inv, rs = a inv, inv = 1 / (s - sm)
  const double dM = d_es * inv;
  const double d_sd = -(d_es * es + d_rs * rs) * inv;
  d_s += dM * E + d_sd;
  d_sm += dM * ps - d_sd;
  d.un -= dM * (E + q.p);
  d.p -= dM * q.un;
  const double d_ps = dM * sm;
  const double d_a = d_rs * inv;
  // f(q), - s U, and E's share in es
  reverse_flux(q, inv_gm1, w, Flux{-s * w.rho, -s * w.mn, -s * w.mt, -s * w.E + dM * (s - q.un)}, d);
  // ps and sm of both sides
  const double h = 0.5 * d_ps;
  d_sm += h * (al + ar);
  const double dN = d_sm * iden;
  const double d_den = -dN * sm;
  const double d_al = h * (sm - l.un) + dN * l.un + d_den + (left ? d_a : 0.0);
  const double d_ar = h * (sm - r.un) - dN * r.un - d_den + (left ? 0.0 : d_a);
  const double d_sl = d_al * l.rho + (left ? d_s : 0.0), d_sr = d_ar * r.rho + (left ? 0.0 : d_s);
  dl.p += h - dN;
  dr.p += h + dN;
  dl.un += dN * al - h * al - d_al * l.rho;
  dr.un -= dN * ar + h * ar + d_ar * r.rho;
  dl.rho += d_al * (sl - l.un);
  dr.rho += d_ar * (sr - r.un);
  if (left) {
    dl.rho += d.rho;
    dl.un += d.un;
    dl.ut += d.ut;
    dl.p += d.p;
  } else {
    dr.rho += d.rho;
    dr.un += d.un;
    dr.ut += d.ut;
    dr.p += d.p;
  }
  // wave speeds
  const double d_cl = (sl_right ? 0.0 : -d_sl) + (sr_right ? 0.0 : d_sr);
  const double d_cr = (sl_right ? -d_sl : 0.0) + (sr_right ? d_sr : 0.0);
  dl.un += (sl_right ? 0.0 : d_sl) + (sr_right ? 0.0 : d_sr);
  dr.un += (sl_right ? d_sl : 0.0) + (sr_right ? d_sr : 0.0);
  dl.rho += d_cl * cl.drho;
  dl.p += d_cl * cl.dp;
  dr.rho += d_cr * cr.drho;
  dr.p += d_cr * cr.dp;
}

// The transposed Jacobian of interface_flux (reconstruction_fluxes.hpp:373-388)
// applied to w: cotangents dl, dr of the face states l, r.
template <int RK>
__device__ __forceinline__ void reverse_face(State l, State r, double g, double inv_gm1, const Flux& w, State& dl,
                                             State& dr)
{
  dl = dr = State{0.0, 0.0, 0.0, 0.0};
  const Sound cl = sound(l.rho, l.p, g), cr = sound(r.rho, r.p, g);
  if (RK == ECG_RIEMANN_RUSANOV) {
    reverse_rusanov(l, r, cl, cr, inv_gm1, w, dl, dr);
    return;
  }
  if (RK != ECG_RIEMANN_LOWMACH_HLLC) {
    reverse_hllc(l, r, cl, cr, inv_gm1, w, dl, dr);
    return;
  }
  // low_mach_correct_velocity_states, reconstruction_fluxes.hpp:212-232
  const State l0 = l, r0 = r;
  const double spl = sqrt(l.un * l.un + l.ut * l.ut), spr = sqrt(r.un * r.un + r.ut * r.ut);
  const bool floor_l = cl.c < 1.0e-12, floor_r = cr.c < 1.0e-12;
  const double icl = 1.0 / (floor_l ? 1.0e-12 : cl.c), icr = 1.0 / (floor_r ? 1.0e-12 : cr.c);
  const double ml = spl * icl, mr = spr * icr;
  const bool right = ml < mr;
  double z = right ? mr : ml;
  const bool capped = 1.0 < z || z < 0.0;
  z = z < 0.0 ? 0.0 : (1.0 < z ? 1.0 : z);
  const double hz = 0.5 * z;
  const double an = 0.5 * (l.un + r.un), at = 0.5 * (l.ut + r.ut);
  const double jn = l.un - r.un, jt = l.ut - r.ut;
  l.un = an + hz * jn;
  r.un = an - hz * jn;
  l.ut = at + hz * jt;
  r.ut = at - hz * jt;
  reverse_hllc(l, r, cl, cr, inv_gm1, w, dl, dr);
  const double sn = dl.un + dr.un, st = dl.ut + dr.ut, dn = dl.un - dr.un, dt = dl.ut - dr.ut;
  dl.un = 0.5 * sn + hz * dn;
  dr.un = 0.5 * sn - hz * dn;
  dl.ut = 0.5 * st + hz * dt;
  dr.ut = 0.5 * st - hz * dt;
  if (capped) return;
  const double d_m = 0.5 * (jn * dn + jt * dt);
  if (right) {
    const double k = spr > 0.0 ? d_m * icr / spr : 0.0;
    dr.un += k * r0.un;
    dr.ut += k * r0.ut;
    if (!floor_r) {
      dr.rho -= d_m * mr * icr * cr.drho;
      dr.p -= d_m * mr * icr * cr.dp;
    }
  } else {
    const double k = spl > 0.0 ? d_m * icl / spl : 0.0;
    dl.un += k * l0.un;
    dl.ut += k * l0.ut;
    if (!floor_l) {
      dl.rho -= d_m * ml * icl * cl.drho;
      dl.p -= d_m * ml * icl * cl.dp;
    }
  }
}

}  // namespace ecg_adj
