// adjoint_richards.cuh — closed-form reverse of one accepted substep of the
// moisture-form Richards solve, shared by the recording and the hand-written step
// adjoints.  ws, bb, suc, ks: the hydraulic parameters watsat, bsw, sucsat, hksat of
// levels 1..nl (1-based arrays).
#pragma once
#include "clmgb_device.cuh"
#include "launch.h"

namespace clmgb {

// ---------------------------------------------------------------------------
// Closed-form reverse of one accepted substep of the moisture-form solve
// (soil_water_movement.jl:1274-1483).  The substep's values are recomputed from its
// starting water (the clamps and decisions with the production arithmetic), then its
// adjoint is formed section by section, last to first:
//   update    liq' = liq + dwat*1000 dz,  qc += qcT*dtsub/dtime
//   solve     A dwat = rmx (tridiagonal): lambda = A^-T dwat_bar by the same Thomas
//             sweep on the transposed bands (the tridiagonal_solve! rule,
//             enzyme_rules.jl:160-201), rmx_bar = lambda, band_bar = -lambda dwat^T
//   assembly  amx = dqidw0 dt_dz, bmx = -1 - (-dqidw1 + dqodw1) dt_dz,
//             cmx = -dqodw2 dt_dz, rmx = -fnet dt_dz
//   fluxes    qout, dqodw1, dqodw2 of each interface and the lower boundary
//   hydraulics  hk = imp ksat s1^(2b+3), dhkdw, smp = -sucsat s^-b, dsmpdw, with
//             the clamps of s and s1 passing the derivative only where the value
//             was not clamped (the branch Julia's max/min took).
// The stages are functions of a level or an interface, used by the reverse on one thread
// (mf_substep_reverse) and by the one with a thread per level (adjoint_richards_packed.cu),
// so that both give the same bits.  Their products and sums are fused, divisions and powers
// run on the integer pipes, and each is written for few FP64 instructions (each holds
// GB300's FP64 unit for 65 cycles): with q the adjoint of an interface's flux, those of the
// flux's derivatives in the water of the levels on its sides are q dwat_j and q dwat_{j+1},
// and the conductivity's adjoint times the saturation power serves ksat, the impedance and
// the exponent.  About 75 FP64 instructions a level and substep; 115 before.
// ---------------------------------------------------------------------------
// Adjoints accumulated over the substeps, per level: 1/watsat's and watsat's, bsw's in the
// matric potential, the conductivity exponent's (2 bsw + 3), sucsat's, and the conductivity's
// times the saturation power (times imp it is ksat's, times ksat the impedance's).
struct RichardsBar {
  double ws[MAXSOI + 1], b[MAXSOI + 1], e[MAXSOI + 1], suc[MAXSOI + 1], hp[MAXSOI + 1];
};

__device__ __forceinline__ double rv_fma(double a, double b, double c) { return fma(a, b, c); }

// saturation (:1283-1287); dzw = dz DENH2O
struct RvSat {
  double s0, s;
  bool lpass, spass;               // Julia's max/min took the unclamped value
};
__device__ __forceinline__ RvSat rv_saturation(double liq, double dzw, double ws) {
  RvSat r;
  r.s0 = jl_div(jl_div(jl_max(liq, 1.0e-6), dzw), ws);
  r.s = jl_max(0.01, jl_min(r.s0, 1.0));
  r.lpass = at_least(liq, 1.0e-6);
  r.spass = above(r.s0, 0.01) && !above(r.s0, 1.0);
  return r;
}

// the powers of the saturation and their logarithms (:1288-1308); s_n: the next level's
struct RvPow {
  double rs, rs1, ls, l1, P, Q;    // 1/s, 1/s1, log s, log s1, s1^e, s^-b
  bool s1pass;
};
__device__ __forceinline__ RvPow rv_powers(double s, double s_n, bool last, double e, double b) {
  RvPow p;
  const double s1r = last ? s : 0.5 * (s + s_n);
  const double s1 = jl_max(0.01, jl_min(s1r, 1.0));
  p.s1pass = above(s1r, 0.01) && !above(s1r, 1.0);
  p.rs = jl_div(1.0, s);
  p.rs1 = jl_div(1.0, s1);
  p.ls = ::cm_log(s);
  p.l1 = ::cm_log(s1);
  p.P = cm_pow(s1, e);
  p.Q = cm_pow(s, -b);
  return p;
}
struct RvHyd {
  double hk, dh, smp, dsds, dsw;   // conductivity, its derivative, potential, its derivatives in s and water
};
__device__ __forceinline__ RvHyd rv_hydraulics(const RvPow& p, double ik, double e, double b, double suc, double rws) {
  RvHyd h;
  h.hk = ik * p.P;
  h.dh = e * h.hk * p.rs1;
  h.smp = -suc * p.Q;
  h.dsds = -b * h.smp * p.rs;
  h.dsw = h.dsds * rws;
  return h;
}

// the flux of an interface and its derivatives in the water of its levels (:1310-1378)
struct RvFlux {
  double dk1, dk2, r, qo, d1, d2;  // r = qo / hk
};
__device__ __forceinline__ RvFlux rv_flux(const RvHyd& h, double smp_n, double dsw_n, double rden, double hrw,
                                          double hrwn) {
  RvFlux f;
  f.dk1 = h.dh * hrw;
  f.dk2 = h.dh * hrwn;
  f.r = rv_fma(-(smp_n - h.smp), rden, 1.0);
  const double hr = h.hk * rden;
  f.qo = h.hk * f.r;
  f.d1 = rv_fma(hr, h.dsw, f.dk1 * f.r);
  f.d2 = rv_fma(-hr, dsw_n, f.dk2 * f.r);
  return f;
}
// wt: the water-table boundary is active (rden its distance); flux: the flux boundary
__device__ __forceinline__ RvFlux rv_flux_bottom(const RvHyd& h, bool wt, bool flux, double rden, double rws) {
  RvFlux f = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  if (wt) {
    f.dk1 = h.dh * rws;
    f.r = rv_fma(h.smp, rden, 1.0);
    f.qo = h.hk * f.r;
    f.d1 = rv_fma(h.hk * rden, h.dsw, f.dk1 * f.r);
  } else if (flux) {
    f.qo = h.hk;
    f.d1 = h.dh * rws;
  }
  return f;
}

// the level's row of the band and the right-hand sides of A dwat = x and A^T lambda = g
// (:1380-1412); i0, i1: the derivatives of the inflow, lam: the adjoint of the level's water
struct RvRow {
  double a, b, c, x, g;
};
__device__ __forceinline__ RvRow rv_row(double qin, double i0, double i1, const RvFlux& f, double root, double dt,
                                        double lam, double dzmm, bool last, double cq, bool flux, bool zero,
                                        const RvHyd& h) {
  RvRow w;
  w.a = i0 * dt;
  w.b = rv_fma(i1 - f.d1, dt, -1.0);
  w.c = last ? 0.0 : -f.d2 * dt;
  w.x = -(qin - f.qo - root) * dt;
  w.g = lam * dzmm;
  if (last) {
    if (flux) w.g += cq * h.dh;
    else if (!zero) w.g += cq * f.d1;
  }
  return w;
}
// one level of the elimination of A (tr: of A^T): x and the modified super-diagonal g
__device__ __forceinline__ void rv_eliminate(bool tr, bool first, double sub, double diag, double sup, double rhs,
                                             double& x, double& g) {
  double den = rv_fma(-sub, g, diag);
  if (!tr && abs_lt(den, 1.0e-30)) den = copysign(1.0e-30, first || den == 0.0 ? 1.0 : den);
  const double rd = div_chain(1.0, den);
  x = rv_fma(-sub, x, rhs) * rd;
  g = sup * rd;
}

// an interface in reverse: the adjoints of its upper level's hydraulics, and those of the
// next level's smp, dsmpdw and, through 1/watsat, watsat
struct RvItf {
  double hkb, smpb, dswb, dhb, wk;
  double n_smpb, n_dswb, n_wk;
};
__device__ __forceinline__ RvItf rv_interface(double q, const RvHyd& h, double dsw_n, const RvFlux& f, double rden,
                                              double hrw, double hrwn, double dw, double dwn) {
  RvItf t;
  const double qr = q * rden, qh = qr * h.hk, qk = q * f.r;
  t.hkb = q * rv_fma(rv_fma(dw, h.dsw, -(dwn * dsw_n)), rden, f.r);
  t.n_smpb = -qr * rv_fma(dwn, f.dk2, rv_fma(dw, f.dk1, h.hk));
  t.smpb = -t.n_smpb;
  t.dswb = qh * dw;
  t.n_dswb = -(qh * dwn);
  const double k1 = qk * dw, k2 = qk * dwn;
  t.dhb = rv_fma(k1, hrw, k2 * hrwn);
  t.wk = k1 * f.dk1;
  t.n_wk = k2 * f.dk2;
  return t;
}
__device__ __forceinline__ RvItf rv_interface_bottom(double q, double cq, const RvHyd& h, const RvFlux& f, bool wt,
                                                     bool flux, bool zero, double rden, double rws, double dw) {
  RvItf t = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  if (flux) {
    const double k1 = q * dw;
    t.hkb = q + cq;
    t.dhb = rv_fma(k1, rws, cq * dw);
    t.wk = k1 * f.d1;
  } else if (!zero && wt) {
    q += cq;
    const double qr = q * rden, k1 = q * f.r * dw;
    t.hkb = q * rv_fma(dw * h.dsw, rden, f.r);
    t.smpb = qr * rv_fma(dw, f.dk1, h.hk);
    t.dswb = qr * h.hk * dw;
    t.dhb = k1 * rws;
    t.wk = k1 * f.dk1;
  }
  return t;
}

// the level's accumulated adjoints (RichardsBar's members)
struct RvAcc {
  double ws, b, e, suc, hp;
};
// the hydraulics of a level in reverse: the adjoints sb of its saturation, wsb of watsat; s1b
// is half of s1's, which the next level's saturation receives too (all of it at the lowest)
__device__ __forceinline__ void rv_hydraulics_reverse(RvItf t, const RvHyd& h, const RvPow& p, bool last, double e,
                                                      double b, double rws, RvAcc& r, double& sb, double& wsb,
                                                      double& s1b) {
  const double dsb = t.dswb * rws, q1 = dsb * p.rs;
  wsb = -rv_fma(t.wk, rws, dsb * h.dsw);
  r.b = rv_fma(-q1, h.smp, r.b);
  const double smpb = rv_fma(-b, q1, t.smpb);
  r.suc = rv_fma(-smpb, p.Q, r.suc);
  const double m1 = smpb * h.smp;
  sb = -rv_fma(q1, h.dsds, m1 * (b * p.rs));
  r.b = rv_fma(-m1, p.ls, r.b);
  const double dd = t.dhb * p.rs1;
  const double hkb = rv_fma(dd, e, t.hkb);
  r.hp = rv_fma(hkb, p.P, r.hp);
  const double m2 = hkb * h.hk;
  r.e = rv_fma(dd, h.hk, rv_fma(m2, p.l1, r.e));
  s1b = rv_fma(-dd, h.dh, m2 * (e * p.rs1));
  if (!p.s1pass) s1b = 0.0;
  if (!last) s1b *= 0.5;
  sb += s1b;
}
__device__ __forceinline__ void rv_water_reverse(const RvSat& s, double sb, double wsb, double rws, double rdzw,
                                                 double& lam, RvAcc& r) {
  if (s.spass) {
    const double vb = sb * rws;
    wsb = rv_fma(-vb, s.s0, wsb);
    if (s.lpass) lam = rv_fma(vb, rdzw, lam);
  }
  r.ws += wsb;
}

// The ice impedance 10^(-e_ice icefrac) and set_soil_water_fractions! of a level in reverse:
// ib, half_above: the impedance exponent's adjoint of the level, and half that of the level
// above.  Returns the adjoint of the level's ice; adds watsat's to wsb.
__device__ __forceinline__ double rv_impedance_bar(double e_ice, double hp, double ks, double imp) {
  return -e_ice * (hp * ks * imp * 2.30258509299404568402);
}
__device__ __forceinline__ double rv_fractions_reverse(double ib, double half_above, bool last, double ws, double ice,
                                                       double exi, double dz, double& wsb) {
  const double icb = (last ? ib : 0.5 * ib) + half_above;
  if (icb == 0.0) return 0.0;
  const double dz_ice = (dz + jl_div(exi, DENICE)) * DENICE;
  const double vol_ice = jl_min(ws, jl_div(ice + exi, dz_ice));
  const double v = jl_div(vol_ice, ws);
  if (dbits(jl_min(1.0, v)) == dbits(1.0)) return 0.0;
  const double vb = jl_div(icb, ws);
  wsb -= vb * v;
  if (dbits(vol_ice) != dbits(ws)) return jl_div(vb, dz_ice);
  wsb += vb;
  return 0.0;
}

// One substep on one thread.  The forward values are kept as level arrays (the saturation
// powers and logs, the reciprocals, the band and the two sweeps); the hydraulic properties
// and fluxes are formed again from them where the reverse needs them.  The reverse is one
// downward sweep with the adjoints of the levels still open (at most three) in registers: at
// level j, interface j's adjoints, then level j+1's hydraulics, then level j+2's water.
static __device__ __noinline__ void mf_substep_reverse(const Dims& D, const clmgb_soilwater_fields& f,
                                                const clmgb_swm_config& cfg, double dtime, int64_t c, int nl,
                                                const double* dzv, const double* imp, const double* ws,
                                                const double* bb, const double* suc, const double* ks,
                                                double dtsub, const double* liq, double* lamL, double lamQ,
                                                RichardsBar& R) {
  const int64_t ld = D.ldc;
  const int joff = D.nlevsno;
  const bool flux = cfg.lower_boundary_condition == CLMGB_BC_FLUX;
  const bool zero = cfg.lower_boundary_condition == CLMGB_BC_ZERO_FLUX;
  const bool wt = cfg.lower_boundary_condition == CLMGB_BC_WATERTABLE && nl <= watertable_level(D, f, c);
  RvSat sat[MAXSOI + 2];
  RvPow pw[MAXSOI + 2];
  double rws[MAXSOI + 2], rden[MAXSOI + 2], dt[MAXSOI + 2], xf[MAXSOI + 2], xt[MAXSOI + 2], gf[MAXSOI + 2],
      gt[MAXSOI + 2], A[MAXSOI + 3], B[MAXSOI + 2], C[MAXSOI + 2];
  for (int j = 1; j <= nl; j++) {
    sat[j] = rv_saturation(liq[j], dzv[j] * DENH2O, ws[j]);
    rws[j] = jl_div(1.0, ws[j]);
  }
  for (int j = 1; j <= nl; j++) {
    pw[j] = rv_powers(sat[j].s, j < nl ? sat[j + 1].s : 0.0, j == nl, 2.0 * bb[j] + 3.0, bb[j]);
    rden[j] = 0.0;
    if (j < nl) rden[j] = jl_div(1.0, M_TO_MM * (LVc(f.z, c, joff + j + 1, ld) - LVc(f.z, c, joff + j, ld)));
    else if (wt) rden[j] = jl_div(1.0, M_TO_MM * (f.zwt[c] - LVc(f.z, c, joff + j, ld)));
  }
  auto hyd = [&](int j) { return rv_hydraulics(pw[j], imp[j] * ks[j], 2.0 * bb[j] + 3.0, bb[j], suc[j], rws[j]); };
  auto flx = [&](int j, const RvHyd& h, const RvHyd& n) {
    return j < nl ? rv_flux(h, n.smp, n.dsw, rden[j], 0.5 * rws[j], 0.5 * rws[j + 1])
                  : rv_flux_bottom(h, wt, flux, rden[j], rws[j]);
  };
  const double cq = lamQ * jl_div(dtsub, dtime);
  RvHyd h = hyd(1), n = h;
  RvFlux above_f = {0.0, 0.0, 0.0, f.qflx_infl[c], 0.0, 0.0};
  for (int j = 1; j <= nl; j++) {
    if (j < nl) n = hyd(j + 1);
    const RvFlux fl = flx(j, h, n);
    const double dzmm = M_TO_MM * dzv[j];
    dt[j] = jl_div(dtsub, dzmm);
    const RvRow w = rv_row(above_f.qo, above_f.d1, above_f.d2, fl, LVc(f.qflx_rootsoi, c, j, ld), dt[j], lamL[j], dzmm,
                           j == nl, cq, flux, zero, h);
    A[j] = w.a;
    B[j] = w.b;
    C[j] = w.c;
    xf[j] = w.x;
    xt[j] = w.g;
    above_f = fl;
    h = n;
  }
  double x = 0.0, g = 0.0, y = 0.0, k = 0.0;
  for (int j = 1; j <= nl; j++) {
    rv_eliminate(false, j == 1, j > 1 ? A[j] : 0.0, B[j], j < nl ? C[j] : 0.0, xf[j], x, g);
    rv_eliminate(true, j == 1, j > 1 ? C[j - 1] : 0.0, B[j], j < nl ? A[j + 1] : 0.0, xt[j], y, k);
    xf[j] = x;
    gf[j] = g;
    xt[j] = y;
    gt[j] = k;
  }
  for (int j = nl - 1; j >= 1; j--) {
    xf[j] = x = rv_fma(-gf[j], x, xf[j]);
    xt[j] = y = rv_fma(-gt[j], y, xt[j]);
  }
  RvItf open = {};                        // level j+1's interface adjoints, open until interface j's
  RvHyd hn = {};
  double sb_open = 0.0, wsb_open = 0.0;   // level j+2's saturation adjoints
  for (int j = nl; j >= -1; j--) {
    RvItf t = {};
    RvHyd hj = {};
    if (j >= 1) {
      hj = hyd(j);
      const RvFlux fl = flx(j, hj, hn);
      double q = xt[j] * dt[j];
      if (j < nl) {
        q = rv_fma(-xt[j + 1], dt[j + 1], q);
        t = rv_interface(q, hj, hn.dsw, fl, rden[j], 0.5 * rws[j], 0.5 * rws[j + 1], xf[j], xf[j + 1]);
        open.smpb += t.n_smpb;
        open.dswb += t.n_dswb;
        open.wk += t.n_wk;
      } else {
        t = rv_interface_bottom(q, cq, hj, fl, wt, flux, zero, rden[j], rws[j], xf[j]);
      }
    }
    double sb = 0.0, wsb = 0.0, s1b = 0.0;
    const int m = j + 1, w = j + 2;
    if (m >= 1 && m <= nl) {
      RvAcc r = {R.ws[m], R.b[m], R.e[m], R.suc[m], R.hp[m]};
      rv_hydraulics_reverse(open, hn, pw[m], m == nl, 2.0 * bb[m] + 3.0, bb[m], rws[m], r, sb, wsb, s1b);
      R.b[m] = r.b;
      R.e[m] = r.e;
      R.suc[m] = r.suc;
      R.hp[m] = r.hp;
    }
    if (w >= 1 && w <= nl) {
      RvAcc r = {R.ws[w], 0.0, 0.0, 0.0, 0.0};
      if (w > 1) sb_open += s1b;
      rv_water_reverse(sat[w], sb_open, wsb_open, rws[w], jl_div(1.0, dzv[w] * DENH2O), lamL[w], r);
      R.ws[w] = r.ws;
    }
    sb_open = sb;
    wsb_open = wsb;
    open = t;
    hn = hj;
  }
}

// Whether k_richards_reverse (adjoint_richards_packed.cu) reverses the solve of column c:
// the log holds both the solve and soil_temperature!'s outputs, which it starts from.
__device__ __forceinline__ bool richards_reversed_here(const Dims& D, const clmgb_soiltemp_fields& ft,
                                                       const clmgb_soilwater_fields& fw, const SubstepLogView& lg,
                                                       int64_t c) {
  if (!lg.rec || !lg.st || !fw.mask_hydrology[c]) return false;
  const int64_t snl = ft.col_snl[c], nl = fw.col_nbedrock[c];
  const int32_t n = lg.count[c];
  return snl <= 0 && snl >= -D.nlevsno && nl >= 1 && nl <= D.nlevsoi && n >= 0 && n <= lg.cap;
}

}  // namespace clmgb
