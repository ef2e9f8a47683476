// aph_adjoint_math.cuh -- hand-written reverse-mode derivatives of the hydro step's
// pointwise pieces: ConsToPrim (ideal gas, floors inactive), PLM, donor cell, and the
// HLLE / HLLC fluxes with their wave-speed and contact branches.
//
// Each *_vjp routine recomputes its forward intermediates and propagates the adjoint of
// its outputs to its inputs (vector-Jacobian product).  The branches taken are the
// forward's branches: at a kink (limiter switch, wave-speed clamp, contact direction)
// the derivative of the active branch is used.  The fluxes are differentiated through the
// fast-mode forward formulas (constant adiabatic index of the pack, sound speed
// sqrt(C^2 gamma p / (p (1 + 1/gm1) + rho C^2))), the same quantity as the reference's
// c-limited sound speed.
#pragma once
#include "aph_math.cuh"

namespace aph {

// ---- ConsToPrim: W = (rho, m/rho, p = gm1 (E - |m|^2 / (2 rho))) -----------------------
// The Jacobian depends on rho and v only, so it is evaluated from the primitives w.
__device__ __forceinline__ void cons_to_prim_vjp(const double *w, const double *gw, double gm1,
                                                 double *gu) {
  const double di = rcp_x(w[IDN]);
  const double v1 = w[IV1], v2 = w[IV2], v3 = w[IV3];
  const double gp = gw[IPR];
  const double v2sum = v1 * v1 + v2 * v2 + v3 * v3;
  gu[IDN] = gw[IDN] - (gw[IV1] * v1 + gw[IV2] * v2 + gw[IV3] * v3) * di + gp * 0.5 * gm1 * v2sum;
  gu[IM1] = gw[IV1] * di - gp * gm1 * v1;
  gu[IM2] = gw[IV2] * di - gp * gm1 * v2;
  gu[IM3] = gw[IV3] * di - gp * gm1 * v3;
  gu[IEN] = gp * gm1;
}

// ---- PLM (plm_simple.hpp:15-32) ---------------------------------------------------------
// Forward with the reciprocal kept: dqm = dq2 r, r = 1/(dql + dqr) where the slopes agree in
// sign, r = 0 where the limiter returns 0.
__device__ __forceinline__ double plm_keep(double q_im1, double q_i, double q_ip1, double &ql,
                                           double &qr) {
  const double dql = q_i - q_im1, dqr = q_ip1 - q_i;
  const double dq2 = dql * dqr;
  double r = 0.0, dqm = 0.0;
  if (is_pos(dq2)) {
    r = rcp_x(dql + dqr);
    dqm = dq2 * r;
  }
  ql = q_i + dqm;
  qr = q_i - dqm;
  return r;
}

// gL is the adjoint of ql_{i+1}, gR of qr_i; r as plm_keep returned it.
__device__ __forceinline__ void plm_vjp(double q_im1, double q_i, double q_ip1, double r, double gL,
                                        double gR, double &g_im1, double &g_i, double &g_ip1) {
  g_i = gL + gR;
  g_im1 = 0.0;
  g_ip1 = 0.0;
  if (!is_zero(r)) {
    const double dql = q_i - q_im1, dqr = q_ip1 - q_i;
    const double gr2 = (gL - gR) * r * r;  // adjoint of dqm times 1/(dql + dqr)^2
    const double gdql = gr2 * dqr * dqr;   // d dqm / d dql = dqr^2 / s^2
    const double gdqr = gr2 * dql * dql;   // d dqm / d dqr = dql^2 / s^2
    g_i += gdql - gdqr;
    g_im1 = -gdql;
    g_ip1 = gdqr;
  }
}

// ---- PPM (ppm_simple.hpp:32-161, in the face/cell split of aph_math.cuh) --------------------
// The forward is piecewise linear in q except the extremum limiter's ratio rho = qe / d2qf,
// so the reverse records the branch each face and cell took and applies the transposed
// linear map of that branch (and the quotient rule for rho).
constexpr int PF_OPEN = 0, PF_AVG = 1, PF_D2M = 2, PF_D20 = 3, PF_QA = 4;

// ppm_face (fast arithmetic) returning the branch: OPEN (unlimited), or limited with
// qd = 0 (AVG), C2 d2(f-1) (D2M), C2 d2(f) (D20), or qa (QA).
// TAME: every window value tame, the scalings on the integer pipe (the same bits).
template <bool TAME>
__device__ __forceinline__ double ppm_face_code(double qm1, double q0, double ddm1, double dd0,
                                                double d2m1, double d20, int &code) {
  const double s = qm1 + q0;
  const double avg = TAME ? half_x(s) : 0.5 * s;
  double dph = fma(ddm1 - dd0, 1.0 / 6.0, avg);
  code = PF_OPEN;
  if (strictly_outside(dph, qm1, q0)) {  // the forward's test (ppm_face, fast mode)
    const double qa_3 = fma(-2.0, dph, s);
    const double qa = TAME ? mulk_x<3, 0>(qa_3) : 3.0 * qa_3;
    double qd = 0.0;
    code = PF_AVG;
    const bool sa = is_neg(qa);
    if (sa == is_neg(d2m1) && sa == is_neg(d20)) {
      const unsigned long long mb = mag(d2m1), mc = mag(d20);
      const bool pick_c = mc < mb;
      const double m = from_bits(pick_c ? mc : mb);
      const unsigned long long mm = mag(TAME ? mulk_x<5, -2>(m) : PPM_C2 * m), ma = mag(qa);
      if (ma < mm) {
        qd = qa;
        code = PF_QA;
      } else {
        qd = flip_if(from_bits(mm), sa);
        code = pick_c ? PF_D20 : PF_D2M;
      }
    }
    dph = fma(qd, -1.0 / 6.0, avg);
  }
  return dph;
}

// d dph / d (q[f-2], q[f-1], q[f], q[f+1]) of a face with the given branch (dd and d2 are
// linear; the QA branch gives back the unlimited value).
__device__ __forceinline__ void ppm_face_coef(int code, double c[4]) {
  constexpr double a = 1.0 / 12.0, b = PPM_C2 / 6.0;
  if (code == PF_AVG) {
    c[0] = 0.0; c[1] = 0.5; c[2] = 0.5; c[3] = 0.0;
  } else if (code == PF_D2M) {
    c[0] = -b; c[1] = 0.5 + 2.0 * b; c[2] = 0.5 - b; c[3] = 0.0;
  } else if (code == PF_D20) {
    c[0] = 0.0; c[1] = 0.5 - b; c[2] = 0.5 + 2.0 * b; c[3] = -b;
  } else {
    c[0] = -a; c[1] = 7.0 * a; c[2] = 7.0 * a; c[3] = -a;
  }
}

// ppm_cell (fast arithmetic) returning its branch: bit 0 extremum; extremum: bits 1-3 the
// source of qe (0 none, 1..3 C2 d2 of cell i-1, i, i+1, 4 d2qf), bit 4 the ratio applied;
// monotone: bit 1 qr steepened, bit 2 ql steepened.  rho: the ratio used.
template <bool TAME>
__device__ __forceinline__ void ppm_cell_code(double q_im2, double q_im1, double q_i, double q_ip1,
                                              double q_ip2, double d2m1, double d20, double d2p1,
                                              double dph_lo, double dph_hi, double &ql, double &qr,
                                              int &code, double &rho) {
  qr = dph_lo;
  ql = dph_hi;
  const double dqf_minus = q_i - qr;
  const double dqf_plus = ql - q_i;
  code = 0;
  rho = 0.0;
  if (TAME) {
    double f = 2.0, xm = dqf_plus, xp = dqf_minus;
    bool sub_m = mag(dqf_minus) >= twice_mag(dqf_plus), add_p = mag(dqf_plus) >= twice_mag(dqf_minus);
    code = (sub_m ? 2 : 0) | (add_p ? 4 : 0);
    if (!strictly_between(qr, q_i, ql) | !strictly_between(q_im1, q_i, q_ip1)) {
      const double d2qf = mulk_x<3, 1>(fma(-2.0, q_i, dph_lo + dph_hi));
      bool guard;
      int src;
      const double qe = extremum_qe(d2qf, d2m1, d20, d2p1, q_im2, q_im1, q_i, q_ip1, q_ip2, guard, src);
      IntOps o;
      const double q = o.div0(qe, o.den(d2qf));
      rho = f = guard ? q : 0.0;
      xm = dqf_minus;
      xp = dqf_plus;
      sub_m = add_p = le(f, 1.0 - 1.0e-12);
      code = 1 | (src << 1) | (sub_m ? 16 : 0);
    }
    const double rm = fma(-f, xm, q_i), lp = fma(f, xp, q_i);
    qr = sub_m ? rm : qr;
    ql = add_p ? lp : ql;
    return;
  }
  if (!strictly_between(qr, q_i, ql) || !strictly_between(q_im1, q_i, q_ip1)) {  // as ppm_cell
    code = 1;
    const double d2qf = 6.0 * (dph_lo + dph_hi - 2.0 * q_i);
    double qe = 0.0;
    int src = 0;
    const bool sd = is_neg(d2qf);
    if (sd == is_neg(d2m1) && sd == is_neg(d20) && sd == is_neg(d2p1)) {
      unsigned long long m = mag(d2m1);
      int k = 1;
      const unsigned long long m0 = mag(d20), m1 = mag(d2p1);
      if (m0 < m) { m = m0; k = 2; }
      if (m1 < m) { m = m1; k = 3; }
      const unsigned long long ms = mag(PPM_C2 * from_bits(m)), md = mag(d2qf);
      if (md < ms) {
        qe = d2qf;
        src = 4;
      } else {
        qe = flip_if(from_bits(ms), sd);
        src = k;
      }
    }
    unsigned long long mx = mag(q_im2);
    const unsigned long long a1 = mag(q_im1), a2 = mag(q_i), a3 = mag(q_ip1), a4 = mag(q_ip2);
    mx = a1 > mx ? a1 : mx;
    mx = a2 > mx ? a2 : mx;
    mx = a3 > mx ? a3 : mx;
    mx = a4 > mx ? a4 : mx;
    if (mag(d2qf) > mag(1.0e-12 * from_bits(mx))) rho = div_x(qe, d2qf);
    code |= src << 1;
    if (le(rho, 1.0 - 1.0e-12)) {
      qr = fma(-rho, dqf_minus, q_i);
      ql = fma(rho, dqf_plus, q_i);
      code |= 16;
    }
  } else {
    if (mag(dqf_minus) >= twice_mag(dqf_plus)) {
      qr = q_i - 2.0 * dqf_plus;
      code |= 2;
    }
    if (mag(dqf_plus) >= twice_mag(dqf_minus)) {
      ql = q_i + 2.0 * dqf_minus;
      code |= 4;
    }
  }
}

// Reverse of ppm_cell_code: gL, gR adjoints of ql_{i+1}, qr_i; out: gq (q_{i-2..i+2}) and the
// adjoints of the two face values.
__device__ __forceinline__ void ppm_cell_vjp(double q_i, double dph_lo, double dph_hi, int code,
                                             double rho, double gL, double gR, double gq[5],
                                             double &g_lo, double &g_hi) {
#pragma unroll
  for (int k = 0; k < 5; ++k) gq[k] = 0.0;
  g_lo = 0.0;
  g_hi = 0.0;
  if (code & 1) {
    if (code & 16) {  // ql = q_i + rho (dph_hi - q_i), qr = q_i - rho (q_i - dph_lo)
      gq[2] += (gL + gR) * (1.0 - rho);
      g_hi += gL * rho;
      g_lo += gR * rho;
      const int src = (code >> 1) & 7;
      if (!is_zero(rho) && src >= 1 && src <= 3) {  // rho = C2 d2(i + src - 2) / d2qf
        const double d2qf = 6.0 * (dph_lo + dph_hi - 2.0 * q_i);
        const double g_rho = gL * (dph_hi - q_i) - gR * (q_i - dph_lo);
        const double g_qe = div_x(g_rho, d2qf);
        const double g_d2qf = -g_qe * rho;
        g_lo += 6.0 * g_d2qf;
        g_hi += 6.0 * g_d2qf;
        gq[2] -= 12.0 * g_d2qf;
        // d2 of cell i + src - 2 is q[c-1] + q[c+1] - 2 q[c], c at gq index src
        const double gd = PPM_C2 * g_qe;
        if (src == 1) {
          gq[0] += gd; gq[2] += gd; gq[1] -= 2.0 * gd;
        } else if (src == 2) {
          gq[1] += gd; gq[3] += gd; gq[2] -= 2.0 * gd;
        } else {
          gq[2] += gd; gq[4] += gd; gq[3] -= 2.0 * gd;
        }
      }
    } else {
      g_hi += gL;
      g_lo += gR;
    }
  } else {
    if (code & 2) {  // qr = 3 q_i - 2 dph_hi
      gq[2] += 3.0 * gR;
      g_hi -= 2.0 * gR;
    } else {
      g_lo += gR;
    }
    if (code & 4) {  // ql = 3 q_i - 2 dph_lo
      gq[2] += 3.0 * gL;
      g_lo -= 2.0 * gL;
    } else {
      g_hi += gL;
    }
  }
}

// ---- Riemann fluxes ------------------------------------------------------------------------
// The adjoint passes are bound by the FP64 pipe, so the reverse forms neither the fluxes (their
// products with the adjoint are sums it needs anyway) nor a factor twice, and its plain products
// take the integer pipe (OPS = FaceOps); every fused one is named.  The PLM + HLLE pass held the
// FP64 pipe for 384 warp instructions per 32 zones, 78 % of its cycles, before (now 245 and 66 %); the
// forward and backward of a 512^2 rollout with it went from 7.94 to 7.18 ms.
struct SoundSpeed {
  double c, dc_dp, dc_drho;
};
// c = sqrt(N/D), N = C^2 gamma p, D = p (1 + 1/gm1) + rho C^2; ip = 1/p, and
// 1/D = c^2 / N = c^2 ip / (C^2 gamma), so no division beyond ip.
template <class OPS>
__device__ __forceinline__ SoundSpeed sound_speed_d(double rho, double p, double ip,
                                                    const GasConsts &gc, double ic2g, OPS &o) {
  const double N = o.mul(gc.c2g, p);
  const double D = fma(p, gc.one_igm1, o.mul(rho, C_LIGHT2));
  SoundSpeed s;
  s.c = o.mul(N, o.rsqrt(o.mul(N, D)));
  const double iD = o.mul(o.mul(s.c, s.c), o.mul(ip, ic2g));
  const double hc = o.half(s.c);
  s.dc_dp = o.mul(hc, fma(-gc.one_igm1, iD, ip));
  s.dc_drho = -o.mul(hc, o.mul(C_LIGHT2, iD));
  return s;
}

// Adjoint of one side's physical flux  F = (rho vx, rho u vx + p, rho v vx, rho z vx, e vx + p u)
// with vx = u - b, m = rho vx and e = p/gm1 + rho |v|^2 / 2, for the flux adjoint g: gw
// (rho, u, v, z, p) without the part through vx, the adjoint gvx of vx, and g . F.
template <class OPS>
__device__ __forceinline__ void side_flux_vjp(const double *w, double vx, double m, double igm1,
                                              const double *g, double *gw, double &gvx, double &gF,
                                              OPS &o) {
  const double rho = w[IDN], u = w[IV1], v = w[IV2], z = w[IV3], p = w[IPR];
  const double hk = o.half(square3(u, v, z, o));
  const double e = fma(p, igm1, o.mul(rho, hk));
  const double A = fma(g[3], z, fma(g[2], v, fma(g[1], u, g[0])));  // shared by d/drho and d/dvx
  const double P = fma(g[4], u, g[1]);
  const double ge = o.mul(g[4], vx);  // adjoint of e
  gvx = fma(g[4], e, o.mul(rho, A));
  gF = fma(gvx, vx, o.mul(p, P));
  gw[IDN] = fma(A, vx, o.mul(ge, hk));
  gw[IV1] = fma(g[4], p, o.mul(m, P));
  gw[IV2] = o.mul(m, fma(g[4], v, g[2]));
  gw[IV3] = o.mul(m, fma(g[4], z, g[3]));
  gw[IPR] = fma(ge, igm1, P);
}

// The part of both solvers through the mean pressure  pm = (pl + pr) / 2 + du rhoa ca / 2, with
// adjoint g and du = ul - ur: adds to gw* and returns half the adjoint of ca.
template <class OPS>
__device__ __forceinline__ double mean_pressure_vjp(double g, double du, double rhoa, double ca,
                                                    double *gwl, double *gwr, OPS &o) {
  const double h = o.half(g);
  const double hd = o.mul(h, du), hc = o.mul(h, ca);
  const double grho = o.half(o.mul(hd, ca));
  gwl[IPR] = add(gwl[IPR], h);
  gwr[IPR] = add(gwr[IPR], h);
  gwl[IV1] = fma(hc, rhoa, gwl[IV1]);
  gwr[IV1] = fma(-hc, rhoa, gwr[IV1]);
  gwl[IDN] = add(gwl[IDN], grho);
  gwr[IDN] = add(gwr[IDN], grho);
  return o.half(o.mul(hd, rhoa));
}

// ---- HLLE (hydro_hlle.hpp:28-133) ----------------------------------------------------------
// w*: (rho, v_n, v_t1, v_t2, p); gf: adjoint of the 5 flux components; gwl/gwr: output.
template <class OPS>
__device__ __forceinline__ void hlle_vjp(const double *wl, const double *wr, const GasConsts &gc,
                                         double ic2g, const double *gf, double *gwl, double *gwr, OPS &o) {
  const double ipl = o.rcp(wl[IPR]), ipr = o.rcp(wr[IPR]);
  const SoundSpeed sl = sound_speed_d(wl[IDN], wl[IPR], ipl, gc, ic2g, o);
  const SoundSpeed sr = sound_speed_d(wr[IDN], wr[IPR], ipr, gc, ic2g, o);
  const double cl = sl.c, cr = sr.c;
  const double rhoa = o.half(add(wl[IDN], wr[IDN]));
  const double ca = o.half(add(cl, cr));
  const double du = sub(wl[IV1], wr[IV1]);
  const double pmid = o.half(fma(o.mul(du, rhoa), ca, add(wl[IPR], wr[IPR])));
  const bool bl = gt(pmid, wl[IPR]), br = gt(pmid, wr[IPR]);
  const double k = gc.hlle_k;
  const double ql = bl ? fma(k, fma(pmid, ipl, -1.0), 1.0) : 1.0;
  const double qr = br ? fma(k, fma(pmid, ipr, -1.0), 1.0) : 1.0;
  const double al = fma(-cl, ql, wl[IV1]);
  const double ar = fma(cr, qr, wr[IV1]);
  const bool bpos = is_pos(ar), bneg = is_neg(al);
  const double bp = bpos ? ar : 0.0;
  const double bm = bneg ? al : 0.0;
  const double vxl = sub(wl[IV1], bm), vxr = sub(wr[IV1], bp);
  const bool has = bpos || bneg;
  const double ibpm = o.rcp(has ? sub(bp, bm) : 1.0);
  const double tmp = has ? o.mul(o.half(add(bp, bm)), ibpm) : 0.0;
  // reverse: flux = (1/2 + tmp) F_l + (1/2 - tmp) F_r
  const double wtl = add(0.5, tmp), wtr = sub(0.5, tmp);
  double gvxl, gvxr, gFl, gFr;
  side_flux_vjp(wl, vxl, o.mul(wl[IDN], vxl), gc.igm1, gf, gwl, gvxl, gFl, o);
  side_flux_vjp(wr, vxr, o.mul(wr[IDN], vxr), gc.igm1, gf, gwr, gvxr, gFr, o);
#pragma unroll
  for (int n = 0; n < 5; ++n) {
    gwl[n] = o.mul(gwl[n], wtl);
    gwr[n] = o.mul(gwr[n], wtr);
  }
  gvxl = o.mul(gvxl, wtl);
  gvxr = o.mul(gvxr, wtr);
  // d tmp / d bp = -bm / (bp - bm)^2, d tmp / d bm = bp / (bp - bm)^2; vx = u - b
  const double gi = has ? o.mul(o.mul(sub(gFl, gFr), ibpm), ibpm) : 0.0;
  const double gar = bpos ? fma(-gi, bm, -gvxr) : 0.0;
  const double gal = bneg ? fma(gi, bp, -gvxl) : 0.0;
  gwl[IV1] = add(gwl[IV1], add(gvxl, gal));
  gwr[IV1] = add(gwr[IV1], add(gvxr, gar));
  // al = ul - cl ql ; ar = ur + cr qr
  double gcl = -o.mul(gal, ql), gcr = o.mul(gar, qr);
  if (bl || br) {
    double gpmid = 0.0;
    if (bl) {
      const double t = o.mul(o.mul(-o.mul(gal, cl), k), ipl);
      gpmid = t;
      gwl[IPR] = fma(-t, o.mul(pmid, ipl), gwl[IPR]);
    }
    if (br) {
      const double t = o.mul(o.mul(o.mul(gar, cr), k), ipr);
      gpmid = add(gpmid, t);
      gwr[IPR] = fma(-t, o.mul(pmid, ipr), gwr[IPR]);
    }
    const double gca = mean_pressure_vjp(gpmid, du, rhoa, ca, gwl, gwr, o);
    gcl = add(gcl, gca);
    gcr = add(gcr, gca);
  }
  gwl[IPR] = fma(gcl, sl.dc_dp, gwl[IPR]);
  gwl[IDN] = fma(gcl, sl.dc_drho, gwl[IDN]);
  gwr[IPR] = fma(gcr, sr.dc_dp, gwr[IPR]);
  gwr[IDN] = fma(gcr, sr.dc_drho, gwr[IDN]);
}

// ---- HLLC (hydro_hllc.hpp:14-146) -----------------------------------------------------------
template <class OPS>
__device__ __forceinline__ void hllc_vjp(const double *wl, const double *wr, const GasConsts &gc,
                                         double ic2g, const double *gf, double *gwl, double *gwr, OPS &o) {
  const double rl = wl[IDN], ul = wl[IV1], pl = wl[IPR];
  const double rr = wr[IDN], ur = wr[IV1], pr = wr[IPR];
  const double ipl = o.rcp(pl), ipr = o.rcp(pr);
  const SoundSpeed sdl = sound_speed_d(rl, pl, ipl, gc, ic2g, o);
  const SoundSpeed sdr = sound_speed_d(rr, pr, ipr, gc, ic2g, o);
  const double cl = sdl.c, cr = sdr.c;
  const double rhoa = o.half(add(rl, rr));
  const double ca = o.half(add(cl, cr));
  const double du = sub(ul, ur);
  const double pstar = fma(0.5, add(pl, pr), o.mul(o.mul(o.half(du), rhoa), ca));
  const double k = gc.hllc_k;
  const bool bl = gt(pstar, pl), br = gt(pstar, pr);
  const double argl = bl ? fma(k, fma(pstar, ipl, -1.0), 1.0) : 1.0;
  const double argr = br ? fma(k, fma(pstar, ipr, -1.0), 1.0) : 1.0;
  const double iql = bl ? o.rsqrt(argl) : 1.0;  // q = arg / sqrt(arg), 1/q kept for the reverse
  const double iqr = br ? o.rsqrt(argr) : 1.0;
  const double ql = bl ? o.mul(argl, iql) : 1.0;
  const double qr = br ? o.mul(argr, iqr) : 1.0;
  const double sl = fma(-cl, ql, ul);
  const double sr = fma(cr, qr, ur);
  const bool bpos = is_pos(sr), bneg = is_neg(sl);
  const double vxl = sub(ul, sl), vxr = sub(ur, sr);
  const double ml = o.mul(rl, vxl), mr = -o.mul(rr, vxr);
  const double tl = fma(ml, ul, pl), tr = fma(-mr, ur, pr);
  const double imm = o.rcp(add(ml, mr));
  const double sstar = o.mul(sub(tl, tr), imm);
  const double cp0 = o.mul(fma(ml, tr, o.mul(mr, tl)), imm);
  const bool cpos = is_pos(cp0);
  const double cp = cpos ? cp0 : 0.0;
  // flx = c_s F_s(w_s) + (0, ustar cp, 0, 0, ustar cp sstar) with the upwind side s of the
  // contact (left with b = bm when sstar >= 0, else right with b = bp); the other side's
  // weight is exactly 0, so only side s is differentiated
  const bool sp = !is_neg(sstar);
  double ws[5], gws[5], gwx, gcs;
#pragma unroll
  for (int n = 0; n < 5; ++n) ws[n] = sp ? wl[n] : wr[n];
  const double b = sp ? (bneg ? sl : -TINY_NUMBER) : (bpos ? sr : TINY_NUMBER);
  const double wx = sub(ws[IV1], b);
  // c = sstar / (sstar - b), ustar = -b / (sstar - b)
  const double idn = o.rcp(sub(sstar, b));
  const double cs = o.mul(sstar, idn);
  const double ustar = -o.mul(b, idn);
  side_flux_vjp(ws, wx, o.mul(ws[IDN], wx), gc.igm1, gf, gws, gwx, gcs, o);
#pragma unroll
  for (int n = 0; n < 5; ++n) gws[n] = o.mul(gws[n], cs);
  gwx = o.mul(gwx, cs);
  const double Q = fma(gf[4], sstar, gf[1]);
  // d c / d sstar = -b idn^2, d c / d b = sstar idn^2; d ustar / d sstar = b idn^2,
  // d ustar / d b = -sstar idn^2
  const double x2 = o.mul(sub(o.mul(cp, Q), gcs), o.mul(idn, idn));
  const double gsstar = fma(x2, b, o.mul(o.mul(gf[4], ustar), cp));
  const double gb = fma(-x2, sstar, -gwx);
  gws[IV1] = add(gws[IV1], gwx);
  // cp = max(cp0, 0)
  const double gcp0 = cpos ? o.mul(ustar, Q) : 0.0;
  // sstar = (tl - tr) imm; cp0 = (ml tr + mr tl) imm; imm = 1/(ml + mr)
  const double e1 = o.mul(gsstar, imm), e2 = o.mul(gcp0, imm);
  const double gtl = fma(e2, mr, e1), gtr = fma(e2, ml, -e1);
  const double gsum = -fma(e1, sstar, o.mul(e2, cp0));
  // tl = pl + ml ul ; tr = pr - mr ur ; ml = rl vxl ; mr = -rr vxr
  const double gml = fma(gtl, ul, fma(e2, tr, gsum));
  const double gmr = fma(-gtr, ur, fma(e2, tl, gsum));
  const double gvxl = o.mul(gml, rl), gvxr = -o.mul(gmr, rr);
  // vx = u - s, the clamped s being bm or bp: the two ways from vx to u cancel
  const double gbl = sp && bneg ? gb : 0.0, gbr = !sp && bpos ? gb : 0.0;
  const double gsl = sub(gbl, gvxl), gsr = sub(gbr, gvxr);
  gwl[IDN] = fma(gml, vxl, sp ? gws[IDN] : 0.0);
  gwr[IDN] = fma(-gmr, vxr, sp ? 0.0 : gws[IDN]);
  gwl[IV1] = add(fma(gtl, ml, sp ? gws[IV1] : 0.0), gbl);
  gwr[IV1] = add(fma(-gtr, mr, sp ? 0.0 : gws[IV1]), gbr);
#pragma unroll
  for (int n = IV2; n <= IV3; ++n) {
    gwl[n] = sp ? gws[n] : 0.0;
    gwr[n] = sp ? 0.0 : gws[n];
  }
  gwl[IPR] = add(sp ? gws[IPR] : 0.0, gtl);
  gwr[IPR] = add(sp ? 0.0 : gws[IPR], gtr);
  // sl = ul - cl ql ; sr = ur + cr qr
  double gcl = -o.mul(gsl, ql), gcr = o.mul(gsr, qr);
  if (bl || br) {  // q = sqrt(1 + k (pstar/p - 1)) when pstar > p
    double gpstar = 0.0;
    if (bl) {
      const double t = o.mul(o.mul(o.half(o.mul(-o.mul(gsl, cl), iql)), k), ipl);
      gpstar = t;
      gwl[IPR] = fma(-t, o.mul(pstar, ipl), gwl[IPR]);
    }
    if (br) {
      const double t = o.mul(o.mul(o.half(o.mul(o.mul(gsr, cr), iqr)), k), ipr);
      gpstar = add(gpstar, t);
      gwr[IPR] = fma(-t, o.mul(pstar, ipr), gwr[IPR]);
    }
    const double gca = mean_pressure_vjp(gpstar, du, rhoa, ca, gwl, gwr, o);
    gcl = add(gcl, gca);
    gcr = add(gcr, gca);
  }
  gwl[IPR] = fma(gcl, sdl.dc_dp, gwl[IPR]);
  gwl[IDN] = fma(gcl, sdl.dc_drho, gwl[IDN]);
  gwr[IPR] = fma(gcr, sdr.dc_dp, gwr[IPR]);
  gwr[IDN] = fma(gcr, sdr.dc_drho, gwr[IDN]);
}

// A face whose states, adjoints or products leave the integer pipe's range: the same with the IEEE
// instructions (the same bits, out of line).  x: wl, wr, gf; on return gwl, gwr.
template <int RS>
__device__ __noinline__ void riemann_vjp_ieee(double *x, const GasConsts &gc, double ic2g) {
  IeeeOps o;
  double gwl[5], gwr[5];
  if (RS == RS_HLLE) hlle_vjp(x, x + 5, gc, ic2g, x + 10, gwl, gwr, o);
  else hllc_vjp(x, x + 5, gc, ic2g, x + 10, gwl, gwr, o);
  for (int n = 0; n < 5; ++n) x[n] = gwl[n], x[5 + n] = gwr[n];
}
}  // namespace aph
