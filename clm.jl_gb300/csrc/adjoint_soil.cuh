// adjoint_soil.cuh — soil_temperature! in reverse: functions of a level or a row, used by
// the reverse on one thread (soil_temperature_reverse) and by the one with a thread per level
// (adjoint_soil_packed.cu), so that both give the same bits.  Divisions and powers run on the
// integer pipes.
#pragma once
#include "adjoint_richards.cuh"
#include "clmgb_device.cuh"

namespace clmgb {

// The factorisation of the column's band system: lu/x/piv point at the thread's own
// storage (soil_temperature! run here) or at the column's soil_temperature! record.
struct CfBand {
  int n;
  const double* lu;
  const double* x;
  const uint8_t* piv;
  double lu_s[MAXROWS * 7];
  double x_s[MAXROWS];
  uint8_t piv_s[MAXROWS];
};

__device__ __forceinline__ bool same_bits(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b);
}

// ---------------------------------------------------------------------------
// Phase change of one level (snow or soil), reversed.  T0: the temperature the
// band solve left, wice0/wliq0: ice and liquid water before the phase change,
// fct: the level's fact.  In: the adjoints of the level's temperature, liquid
// water and ice after the phase change.  Out (accumulated): the adjoints of T0,
// wice0, wliq0, fct, dhsdT and the level's watsat, bsw, sucsat (supercooled water).
// Columns with excess ice or snow without layers are flagged by the caller; their
// branches are not taken here.
// ---------------------------------------------------------------------------
struct PcLevelIn {
  int j, jtop;
  double T0, wice0, wliq0, fct, dhsdT, fse, fh, dtime;
  bool sc_type;
  double ws, bs, suc, dz;
};

static __device__ __noinline__ void phase_change_level_reverse(const PcLevelIn& in, double Tpc_b, double liqpc_b,
                                                        double icepc_b, double& T0_b, double& ice0_b,
                                                        double& liq0_b, double& fct_b, double& dhsdT_b,
                                                        double& ws_b, double& bs_b, double& suc_b) {
  const int j = in.j, jtop = in.jtop;
  const double T0 = in.T0, wice0 = in.wice0, wliq0 = in.wliq0, fct = in.fct, dhsdT = in.dhsdT;
  const double fse = in.fse, fh = in.fh, dtime = in.dtime;
  const double wmass0 = wice0 + wliq0 + 0.0;
  // ---- the melt / freeze decision (:1990-2040) ----
  int im = 0;
  double tinc = 0.0;
  bool sc_on = false;
  double sc = 0.0, P = 0.0, r = 0.0, e = 0.0, q = 0.0, g = 0.0;
  if (j <= 0) {
    if (pos(wice0) && above(T0, TFRZ)) {
      im = 1;
      tinc = TFRZ - T0;
    } else if (pos(wliq0) && below(T0, TFRZ)) {
      im = 2;
      tinc = TFRZ - T0;
    }
  } else {
    double T = T0;
    if (pos(wice0) && above(T0, TFRZ)) {
      im = 1;
      tinc = TFRZ - T0;
      T = TFRZ;
    }
    if (in.sc_type && below(T, TFRZ)) {
      sc_on = true;
      q = jl_div(HFUS * (TFRZ - T), GRAV * T);
      g = GRAV * T;
      const double smp = q * 1000.0;
      r = jl_div(smp, in.suc);
      e = jl_div(-1.0, in.bs);
      P = cm_pow(r, e);
      sc = in.ws * P;
      sc *= in.dz * 1000.0;
    }
    if (below(T, TFRZ) && wliq0 > sc) {
      im = 2;
      tinc = TFRZ - T;
    }
  }
  if (im == 0) {
    T0_b += Tpc_b;
    liq0_b += liqpc_b;
    ice0_b += icepc_b;
    return;
  }
  // ---- hm (:2060-2085) ----
  double hm;
  if (j == jtop) {
    if (j > 0) hm = dhsdT * tinc - jl_div(tinc, fct);
    else hm = fse * (dhsdT * tinc - jl_div(tinc, fct));
    if (j == 1 && !zero_bits(fh)) hm -= fh * dhsdT * tinc;
  } else if (j == 1) {
    hm = (1.0 - fse - fh) * dhsdT * tinc - jl_div(tinc, fct);
  } else {
    if (j < 1) hm = jl_div(-fse * tinc, fct);
    else hm = jl_div(-tinc, fct);
  }
  if ((im == 1 && negv(hm)) || (im == 2 && pos(hm))) im = 0;
  if (im == 0 || !(pos(hm) || negv(hm))) {
    // the temperature was set to freezing (a constant); the water is unchanged
    liq0_b += liqpc_b;
    ice0_b += icepc_b;
    return;
  }
  // ---- new ice and liquid water (:2090-2140) ----
  const double xm = jl_div(hm * dtime, HFUS);
  double ice = wice0, heatr = 0.0;
  int kind = 0;   // 0 ice unchanged, 1 wice0 - xm, 2 constant, 3 wmass0, 4 wmass0 - sc
  if (pos(xm)) {
    const double v = wice0 - xm;
    ice = jl_max(0.0, v);
    kind = same_bits(ice, 0.0) ? 2 : 1;
    heatr = hm - jl_div(HFUS * (wice0 - ice), dtime);
  } else if (negv(xm)) {
    if (j <= 0) {
      const double a = wmass0, b = wice0 - xm;
      ice = jl_min(a, b);
      kind = same_bits(ice, a) ? 3 : 1;
    } else {
      if (wmass0 - 0.0 < sc) {
        ice = 0.0;
        kind = 2;
      } else {
        const double a = wmass0 - 0.0 - sc, b = wice0 - xm;
        ice = jl_min(a, b);
        kind = same_bits(ice, a) ? 4 : 1;
      }
    }
    heatr = hm - jl_div(HFUS * (wice0 - ice), dtime);
  }
  const double liqv = wmass0 - ice - 0.0;
  const double liq = jl_max(0.0, liqv);
  const bool liq_pass = !same_bits(liq, 0.0);
  // ---- reverse (derivative coefficients with reciprocals) ----
  double heatr_b = 0.0, hm_b = 0.0, xm_b = 0.0, ice_b = icepc_b, wmass0_b = 0.0, wice0_b = 0.0, sc_b = 0.0;
  double tinc_b = 0.0;
  const double rf = jl_div(1.0, fct);
  if ((pos(heatr) || negv(heatr)) && !(j <= 0 && pos(liq * ice))) {
    // temperature correction (:2145-2165); the level starts from freezing
    if (j == 1) {
      const double k = (j == jtop) ? (1.0 - fh) : (1.0 - fse - fh);
      const double rden = jl_div(1.0, 1.0 - k * fct * dhsdT);
      const double incr = fct * heatr * rden;
      const double N_b = Tpc_b * rden, den_b = -Tpc_b * incr * rden;
      fct_b += N_b * heatr - den_b * k * dhsdT;
      heatr_b += N_b * fct;
      dhsdT_b += -den_b * k * fct;
    } else if (j == jtop) {      // top snow layer
      if (pos(fse)) {
        const double rfse = jl_div(1.0, fse);
        const double rden = jl_div(1.0, 1.0 - fct * dhsdT);
        const double incr = fct * rfse * heatr * rden;
        const double N_b = Tpc_b * rden, den_b = -Tpc_b * incr * rden;
        fct_b += N_b * heatr * rfse - den_b * dhsdT;
        heatr_b += N_b * fct * rfse;
        dhsdT_b += -den_b * fct;
      }
    } else if (j > 0) {
      fct_b += Tpc_b * heatr;
      heatr_b += Tpc_b * fct;
    } else if (pos(fse)) {
      const double rfse = jl_div(1.0, fse);
      fct_b += Tpc_b * heatr * rfse;
      heatr_b += Tpc_b * fct * rfse;
    }
  }
  if (liq_pass) {
    wmass0_b += liqpc_b;
    ice_b -= liqpc_b;
  }
  if (!zero_bits(xm)) {
    hm_b += heatr_b;
    const double d_b = -heatr_b * HFUS * jl_div(1.0, dtime);
    wice0_b += d_b;
    ice_b -= d_b;
  }
  switch (kind) {
    case 0: wice0_b += ice_b; break;
    case 1: wice0_b += ice_b; xm_b -= ice_b; break;
    case 3: wmass0_b += ice_b; break;
    case 4: wmass0_b += ice_b; sc_b -= ice_b; break;
    default: break;
  }
  hm_b += xm_b * dtime * (1.0 / HFUS);
  // hm
  if (j == jtop) {
    const double hb = (j > 0) ? hm_b : hm_b * fse;
    dhsdT_b += hb * tinc;
    tinc_b += hb * dhsdT - hb * rf;
    fct_b += hb * tinc * rf * rf;
    if (j == 1 && !zero_bits(fh)) {
      dhsdT_b -= hm_b * fh * tinc;
      tinc_b -= hm_b * fh * dhsdT;
    }
  } else if (j == 1) {
    const double k = 1.0 - fse - fh;
    dhsdT_b += hm_b * k * tinc;
    tinc_b += hm_b * k * dhsdT - hm_b * rf;
    fct_b += hm_b * tinc * rf * rf;
  } else {
    const double a = (j < 1) ? fse : 1.0;     // hm = -a tinc / fct
    tinc_b -= hm_b * a * rf;
    fct_b += hm_b * a * tinc * rf * rf;
  }
  T0_b -= tinc_b;
  // supercooled water sc = watsat (smp/sucsat)^(-1/bsw) dz 1000, smp = HFUS (TFRZ-T)/(GRAV T) 1000
  if (sc_on && !zero_bits(sc_b)) {
    const double sc0_b = sc_b * (in.dz * 1000.0);
    ws_b += sc0_b * P;
    const double P_b = sc0_b * in.ws;
    const double rr = jl_div(1.0, r), rsuc = jl_div(1.0, in.suc), rg = jl_div(1.0, g);
    const double r_b = !zero_bits(r) ? P_b * e * P * rr : 0.0;
    const double e_b = pos(r) ? P_b * P * cm_log(r) : 0.0;
    bs_b += e_b * (-e) * jl_div(1.0, in.bs);
    const double smp_b = r_b * rsuc;
    suc_b += r_b * (-r) * rsuc;
    const double q_b = smp_b * 1000.0;
    const double a_b = q_b * rg;
    const double g_b = -q_b * q * rg;
    T0_b += -a_b * HFUS + g_b * GRAV;
  }
  ice0_b += wice0_b + wmass0_b;
  liq0_b += wmass0_b;
}

// ---------------------------------------------------------------------------
// The column's scalars: decisions, and the ground heat flux sums with their derivative
// weights (:1200-1263).
// ---------------------------------------------------------------------------
struct StCol {
  int64_t snl, lit, nbedrock;
  int jtop, jjtop, snow_method;
  bool is_special, sc_type;
  double fse, fh, eg, dtime, tg0, th0;
  double dhsdT, hs_soil, hs_h2osfc, hs_top, w_set, wb_set, w_act, wb_act;
  double dtc, rdh;                  // surface water: dtime over its heat capacity, 1 / its distance to level 1
};
__device__ __forceinline__ void st_column(StCol& C, const Dims& D, const clmgb_soiltemp_fields& f, int64_t c,
                                          double dtime, int snow_method, double tg0, double th0) {
  C.snl = f.col_snl[c];
  C.jtop = (int)C.snl + 1;
  C.jjtop = C.jtop + D.nlevsno;
  C.lit = f.lun_itype[f.col_landunit[c] - 1];
  C.is_special = (C.lit == ISTWET || C.lit == ISTICE);
  C.sc_type = (C.lit == ISTSOIL || C.lit == ISTCROP || f.col_itype[c] == ICOL_ROAD_PERV);
  C.nbedrock = f.col_nbedrock[c];
  C.fse = f.frac_sno_eff[c];
  C.fh = f.frac_h2osfc[c];
  C.eg = f.emg[c];
  C.dtime = dtime;
  C.snow_method = snow_method;
  C.tg0 = tg0;
  C.th0 = th0;
}
// t_top, t_1: the step's temperatures of the top level and of soil level 1
__device__ __forceinline__ void st_sums(StCol& C, const Dims& D, const clmgb_soiltemp_fields& f, int64_t c, double forc,
                                     double t_top, double t_1) {
  const int64_t ldp = D.ldp;
  const double htvp = f.htvp[c];
  C.dhsdT = C.hs_soil = C.hs_h2osfc = C.hs_top = C.w_set = C.wb_set = C.w_act = C.wb_act = 0.0;
  const double dlwrad_emit = 4.0 * C.eg * SB * (C.tg0 * C.tg0 * C.tg0);
  const double lwe_snow = C.eg * SB * jl_pow4(t_top);
  const double lwe_soil = C.eg * SB * jl_pow4(t_1);
  const double lwe_h2osfc = C.eg * SB * jl_pow4(C.th0);
  for (int64_t p1 = f.col_patchi[c]; p1 <= f.col_patchf[c]; p1++) {
    const int64_t p = p1 - 1;
    if (f.patch_column[p] != c + 1 + D.c0) continue;
    double dh_p = 0.0, hsoil_p = 0.0, hh_p = 0.0;
    const bool act = f.mask_nolakep[p] != 0;
    const double cb = (1.0 - (double)f.frac_veg_nosno[p]) * C.eg;
    const double base = f.dlrad[p] + cb * forc;
    const double wt = f.patch_wtcol[p];
    if (act && !f.lun_urbpoi[f.patch_landunit[p] - 1]) {
      const double dg = -f.cgrnd[p] - dlwrad_emit;
      const double gsoil = f.sabg_soil[p] + base - lwe_soil - (f.eflx_sh_soil[p] + f.qflx_ev_soil[p] * htvp);
      const double gh2o = f.sabg_soil[p] + base - lwe_h2osfc - (f.eflx_sh_h2osfc[p] + f.qflx_ev_h2osfc[p] * htvp);
      if (!zero_bits(wt)) {
        dh_p = dg * wt;
        hsoil_p = gsoil * wt;
        hh_p = gh2o * wt;
        C.w_set += wt;
        C.wb_set += wt * cb;
      }
    }
    C.dhsdT += dh_p;
    C.hs_soil += hsoil_p;
    C.hs_h2osfc += hh_p;
    if (act) {
      const double sab = LVc(f.sabg_lyr, p, C.jjtop, ldp);
      const double gsnow = sab + base - lwe_snow - (f.eflx_sh_snow[p] + f.qflx_ev_snow[p] * htvp);
      C.hs_top += gsnow * wt;
      C.w_act += wt;
      C.wb_act += wt * cb;
    }
  }
  double ch, dz_h2osfc;
  if (above(f.h2osfc[c], THIN_SFCLAYER) && above(C.fh, THIN_SFCLAYER)) {
    ch = jl_max(THIN_SFCLAYER, jl_div(CPLIQ * f.h2osfc[c], C.fh));
    dz_h2osfc = jl_max(THIN_SFCLAYER, jl_div(1.0e-3 * f.h2osfc[c], C.fh));
  } else {
    ch = THIN_SFCLAYER;
    dz_h2osfc = THIN_SFCLAYER;
  }
  C.dtc = jl_div(C.dtime, ch);
  C.rdh = jl_div(1.0, 0.5 * dz_h2osfc + LVc(f.z, c, 1 + D.nlevsno, D.ldc));
}
// absorbed radiation of a level above soil level 2 (:1180-1198)
__device__ __forceinline__ double st_sabg(const Dims& D, const clmgb_soiltemp_fields& f, int64_t c, int jj) {
  double s = 0.0;
  for (int64_t p1 = f.col_patchi[c]; p1 <= f.col_patchf[c]; p1++) {
    const int64_t p = p1 - 1;
    if (f.patch_column[p] != c + 1 + D.c0 || !f.mask_nolakep[p]) continue;
    s += LVc(f.sabg_lyr, p, jj, D.ldp) * f.patch_wtcol[p];
  }
  return s;
}

// ---- layer conductivity and its partials in liquid water, ice and watsat (:647-776) ----
struct StLayer {
  double v, dl, di, dw;
};
__device__ __forceinline__ StLayer st_layer(const StCol& C, const Dims& D, const clmgb_soiltemp_fields& f,
                                         const clmgb_soilwater_fields& fw, int64_t c, int jj, double tin, double liq,
                                         double ice) {
  const int64_t ld = D.ldc;
  const int j = jj - D.nlevsno;
  constexpr double LN_TKWAT = -0.56211891815354124, LN_TKICE = 0.82855181756614826;   // of 0.57 and 2.29
  StLayer r = {0.0, 0.0, 0.0, 0.0};
  if (j >= 1) {
    if (C.is_special) {
      if (C.lit == ISTICE || j <= D.nlevsoi) r.v = below(tin, TFRZ) ? TKICE : TKWAT;
      else r.v = THK_BEDROCK;
      return r;
    }
    if (j > C.nbedrock) {
      r.v = THK_BEDROCK;
      return r;
    }
    const double exi = LV(f.excess_ice, c, j, ld);
    const double dzv = LVc(f.dz, c, jj, ld);
    const double ws = LVc(fw.watsat, c, j, ld);
    const double m = dzv * ws;
    const double satw0 = jl_div(jl_div(liq, DENH2O) + jl_div(ice, DENICE) + jl_div(exi, DENICE), m);
    const double satw = jl_min(1.0, satw0);
    const bool spass = !same_bits(satw, 1.0);
    const double tkdry = LVc(f.tkdry, c, j, ld);
    if (!above(satw, 1.0e-7)) {
      r.v = tkdry;
      return r;
    }
    double dke, ddke;
    if (at_least(tin, TFRZ)) {
      const double L = cm_log10(satw) + 1.0;
      dke = jl_max(0.0, L);
      ddke = same_bits(dke, 0.0) ? 0.0 : 0.43429448190325182765 * jl_div(1.0, satw);
    } else {
      dke = satw;
      ddke = 1.0;
    }
    // TKWAT^a TKICE^b as one exponential
    const double rm = jl_div(1.0, m), rdz = jl_div(1.0, dzv);
    const double a1 = liq * (1.0 / DENH2O) * rdz;
    const double fl_denom = rv_fma((ice + exi) * (1.0 / DENICE), rdz, a1);
    const double rfd = jl_div(1.0, fl_denom);
    const double fl = a1 * rfd;
    const double tkmg = LVc(f.tkmg, c, j, ld);
    const double mix = rv_fma(fl, LN_TKWAT - LN_TKICE, LN_TKICE);
    const double dksat = tkmg * cm_exp(ws * mix);
    r.v = rv_fma(dke, dksat - tkdry, tkdry);
    const double dk = dke * dksat, q = rfd * rdz, kfl = dk * (ws * (LN_TKWAT - LN_TKICE)) * q;
    const double cdke = spass ? (dksat - tkdry) * ddke * rm : 0.0;
    r.dl = rv_fma(kfl, (1.0 - fl) * (1.0 / DENH2O), cdke * (1.0 / DENH2O));
    r.di = rv_fma(kfl, -fl * (1.0 / DENICE), cdke * (1.0 / DENICE));
    r.dw = rv_fma(dk, mix, spass ? -cdke * (satw0 * dzv) : -0.0);      // satw0 may be infinite where it is clamped
    return r;
  }
  const double denom = jl_max(C.fse, 1.0e-6) * jl_max(LVc(f.dz, c, jj, ld), 1.0e-6);
  const double bwv = jl_div(ice + liq, denom);
  double dbw;
  if (C.snow_method == CLMGB_SNOW_JORDAN1991) {
    r.v = TKAIR + (7.75e-5 * bwv + 1.105e-6 * (bwv * bwv)) * (TKICE - TKAIR);
    dbw = (7.75e-5 + 1.105e-6 * (bwv + bwv)) * (TKICE - TKAIR);
  } else if (bwv <= 156.0) {
    r.v = 0.023 + 0.234 * jl_div(bwv, 1000.0);
    dbw = 0.234 / 1000.0;
  } else {
    const double k = jl_div(bwv, 1000.0);
    r.v = 0.138 - 1.01 * k + 3.233 * (k * k);
    dbw = jl_div(-1.01 + 3.233 * (2.0 * k), 1000.0);
  }
  r.dl = jl_div(dbw, denom);
  r.di = r.dl;
  return r;
}
// tk_h2osfc from the soil-1 layer conductivity
__device__ __forceinline__ void st_tkh(const Dims& D, const clmgb_soiltemp_fields& f, int64_t c, double tk1,
                                       double& tkh, double& dtkh) {
  const double zh2osfc = 1.0e-3 * (0.5 * f.h2osfc[c]);
  const double z1 = LVc(f.z, c, 1 + D.nlevsno, D.ldc);
  const double den = TKWAT * z1 + tk1 * zh2osfc;
  if (pos(den)) {
    tkh = jl_div(TKWAT * tk1 * (z1 + zh2osfc), den);
    dtkh = jl_div(TKWAT * (z1 + zh2osfc) - tkh * zh2osfc, den);
  } else {
    tkh = tk1;
    dtkh = 1.0;
  }
}
// the conductivity of the interface below a level, its partials in the two layers, the
// distance and the flux through it (:599-629, :1271-1319)
struct StItf {
  double tk, da, db, rdz, fn;
};
__device__ __forceinline__ StItf st_interface(const Dims& D, const clmgb_soiltemp_fields& f, int64_t c, int jj,
                                              double thk, double thk_n, double tin, double tin_n) {
  const int64_t ld = D.ldc;
  StItf r = {0.0, 0.0, 0.0, 0.0, 0.0};
  if (jj - D.nlevsno > D.nlevgrnd - 1) {
    r.fn = f.eflx_bot[c];
    return r;
  }
  const double zj = LVc(f.z, c, jj, ld), zj1 = LVc(f.z, c, jj + 1, ld), zij1 = LVc(f.zi, c, jj + 1, ld);
  const double A = zj1 - zj, Bz = zj1 - zij1, Cz = zij1 - zj;
  const double rden = jl_div(1.0, thk * Bz + thk_n * Cz);
  r.tk = thk * thk_n * A * rden;
  r.da = (thk_n * A - r.tk * Bz) * rden;
  r.db = (thk * A - r.tk * Cz) * rden;
  r.rdz = jl_div(1.0, A);
  r.fn = r.tk * (tin_n - tin) * r.rdz;
  return r;
}
// the partials of fact = dtime / cv in liquid water, ice and watsat (:599-942)
struct StCap {
  double l, i, w;
};
__device__ __forceinline__ StCap st_capacity(const StCol& C, const Dims& D, const clmgb_soiltemp_fields& f,
                                             const clmgb_soilwater_fields& fw, int64_t c, int jj, double liq,
                                             double ice, double fact) {
  const int64_t ld = D.ldc;
  const int j = jj - D.nlevsno;
  const double dzv = LVc(f.dz, c, jj, ld);
  double cv, dl = 0.0, di = 0.0, dw = 0.0;
  if (j >= 1) {
    cv = ice * CPICE + liq * CPLIQ;
    dl = CPLIQ;
    di = CPICE;
    if (!C.is_special) {
      const double ws = LVc(fw.watsat, c, j, ld), csol = LVc(f.csol, c, j, ld);
      cv = csol * (1.0 - ws) * dzv + cv + LV(f.excess_ice, c, j, ld) * CPICE;
      dw = -csol * dzv;
    }
    if (j > C.nbedrock) {
      cv = CSOL_BEDROCK * dzv;
      dl = di = dw = 0.0;
    }
    if (j == 1 && pos(f.h2osno_no_layers[c])) cv += CPICE * f.h2osno_no_layers[c];
  } else if (pos(C.fse)) {
    const double v = jl_div(CPLIQ * liq + CPICE * ice, C.fse);
    cv = jl_max(THIN_SFCLAYER, v);
    if (!same_bits(cv, THIN_SFCLAYER)) {
      dl = jl_div(CPLIQ, C.fse);
      di = jl_div(CPICE, C.fse);
    }
  } else {
    cv = THIN_SFCLAYER;
  }
  const double dfdcv = jl_div(-fact, cv);
  return StCap{dfdcv * dl, dfdcv * di, dfdcv * dw};
}

// ---- t_grnd in reverse: what it adds to the adjoint of a level's temperature, and of t_h2osfc ----
__device__ __forceinline__ double st_tgrnd_level(const StCol& C, int j, double tgb) {
  if (C.snl < 0) {
    double b = 0.0;
    if (j == C.jtop) b += C.fse * tgb;
    if (j == 1) b += (!zero_bits(C.fh) ? (1.0 - C.fse - C.fh) : (1.0 - C.fse)) * tgb;
    return b;
  }
  return j == 1 ? (!zero_bits(C.fh) ? (1.0 - C.fh) : 1.0) * tgb : 0.0;
}
__device__ __forceinline__ double st_tgrnd_h2osfc(const StCol& C, double tgb) { return !zero_bits(C.fh) ? C.fh * tgb : 0.0; }

// ---- phase change of a level in reverse ----
struct StPc {
  double t, ice, liq, f, dh, ws, bs, suc;
};
__device__ __forceinline__ StPc st_phase_change(const StCol& C, const Dims& D, const clmgb_soiltemp_fields& f,
                                                const clmgb_soilwater_fields& fw, int64_t c, int jj, double T0,
                                                double liq0, double ice0, double fact, double Tb, double liqb,
                                                double iceb) {
  const int64_t ld = D.ldc;
  const int j = jj - D.nlevsno;
  PcLevelIn in;
  in.j = j;
  in.jtop = C.jtop;
  in.T0 = T0;
  in.wice0 = ice0;
  in.wliq0 = liq0;
  in.fct = fact;
  in.dhsdT = C.dhsdT;
  in.fse = C.fse;
  in.fh = C.fh;
  in.dtime = C.dtime;
  in.sc_type = C.sc_type;
  in.ws = j >= 1 ? LVc(fw.watsat, c, j, ld) : 0.0;
  in.bs = j >= 1 ? LVc(fw.bsw, c, j, ld) : 0.0;
  in.suc = j >= 1 ? LVc(fw.sucsat, c, j, ld) : 0.0;
  in.dz = LVc(f.dz, c, jj, ld);
  StPc r = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  phase_change_level_reverse(in, Tb, liqb, iceb, r.t, r.ice, r.liq, r.f, r.dh, r.ws, r.bs, r.suc);
  return r;
}

// ---- a level's row of the band system in reverse (:1365-1748): the adjoints of its fact, of
// the conductivity of and the flux through its interface and the one above (kp, np), of its
// temperature, and of hs_top, hs_soil and dhsdT.  g[d] = -lambda x of the row's entry d. ----
struct StRow {
  double f, k, kp, n, np, t, hst, hss, dh;
};
struct StRowIn {
  int j;
  double lam, g0, g1, g2, g3, g4, fc, t, fn, fnp, tk, tkp, rp, rmn, sabg;
};
__device__ __forceinline__ StRow st_row(const StCol& C, int nlevgrnd, const StRowIn& a) {
  const double omc = 1.0 - CNFAC;
  StRow r = {0.0, 0.0, 0.0, 0.0, 0.0, a.lam, 0.0, 0.0, 0.0};
  const double of = omc * a.fc, ip = of * a.rp, im = of * a.rmn;      // d entry / d conductivity
  const double sp = omc * a.tk * a.rp, sm = omc * a.tkp * a.rmn;      // d entry / d fact
  const double ib = a.lam * a.fc, cb = ib * CNFAC;
  if (a.j == C.jtop) {
    r.f = rv_fma(a.lam, rv_fma(-C.dhsdT, a.t, C.hs_top) + CNFAC * a.fn, a.g2 * (sp - C.dhsdT));
    r.hst = ib;
    r.dh = -ib * a.t - a.g2 * a.fc;
    r.t -= ib * C.dhsdT;
    r.n = cb;
    r.k = a.g2 * ip;
    const double g = a.j == 0 ? a.g4 : a.g3;
    r.f -= g * sp;
    r.k -= g * ip;
  } else if (a.j <= 0) {
    const double g = a.j == 0 ? a.g4 : a.g3;
    r.f = a.lam * (CNFAC * (a.fn - a.fnp) + a.sabg) - a.g1 * sm + a.g2 * (sp + sm) - g * sp;
    r.n = cb;
    r.np = -cb;
    r.kp = (a.g2 - a.g1) * im;
    r.k = (a.g2 - g) * ip;
  } else if (a.j == 1) {
    const double s = 1.0 - C.fse, u = ib * s;
    r.f = a.lam * (s * (C.hs_soil - C.dhsdT * a.t) + CNFAC * (a.fn - C.fse * a.fnp) + C.fse * a.sabg) - a.g3 * sp +
          a.g2 * (sp + C.fse * sm - s * C.dhsdT) - a.g0 * C.fse * sm;
    r.hss = u;
    r.dh = -u * a.t - a.g2 * s * a.fc;
    r.t -= u * C.dhsdT;
    r.n = cb;
    r.np = -cb * C.fse;
    r.k = (a.g2 - a.g3) * ip;
    r.kp = (a.g2 - a.g0) * C.fse * im;
  } else if (a.j <= nlevgrnd - 1) {
    r.f = rv_fma(a.lam * CNFAC, a.fn - a.fnp, rv_fma(a.g2 - a.g3, sp, (a.g2 - a.g1) * sm));
    r.n = cb;
    r.np = -cb;
    r.k = (a.g2 - a.g3) * ip;
    r.kp = (a.g2 - a.g1) * im;
  } else {
    r.f = a.lam * (a.fn - CNFAC * a.fnp) + (a.g2 - a.g1) * sm;
    r.np = -cb;
    r.kp = (a.g2 - a.g1) * im;
  }
  return r;
}
// The surface-water row, and its corrections to soil level 1 (row lam1, entries g1, g2 of that
// row), in reverse.  t1, fact: soil level 1's.
struct StSurf {
  double f1, t1, th, hss, hsh, dh, tkh;
};
__device__ __forceinline__ StSurf st_surface(const StCol& C, double tkh, double t1, double fact, double lam,
                                             double s2, double s3, double lam1, double g1, double g2) {
  const double omc = 1.0 - CNFAC;
  StSurf r = {0.0, 0.0, lam, 0.0, 0.0, 0.0, 0.0};
  const double ib = lam * C.dtc, dT = t1 - C.th0;
  r.hsh = ib;
  r.dh = -ib * C.th0 - s2 * C.dtc;
  r.th -= ib * C.dhsdT;
  const double fnh_b = ib * CNFAC;
  r.tkh = (s2 - s3) * omc * C.dtc * C.rdh + fnh_b * dT * C.rdh;
  const double d_b = fnh_b * tkh * C.rdh;
  r.t1 = d_b;
  r.th -= d_b;
  if (!zero_bits(C.fh)) {
    const double fnh = tkh * dT * C.rdh, jb = -lam1 * C.fh, jf = jb * fact;
    r.f1 = jb * ((C.hs_soil - C.dhsdT * t1) + CNFAC * fnh) + g2 * C.fh * (omc * tkh * C.rdh + C.dhsdT) -
           g1 * C.fh * omc * tkh * C.rdh;
    r.hss = jf;
    r.dh += g2 * C.fh * fact - jf * t1;
    r.t1 -= jf * C.dhsdT;
    const double b = jf * CNFAC;
    r.tkh += b * dT * C.rdh + (g2 - g1) * C.fh * omc * fact * C.rdh;
    r.t1 += b * tkh * C.rdh;
    r.th -= b * tkh * C.rdh;
  }
  return r;
}
// the sums' adjoints: dhsdT's (phase change and rows of the top level and of soil level 1, the
// surface water) and the adjoints of t_grnd, t_h2osfc and the forcing that follow
__device__ __forceinline__ double st_dhsdT_bar(double pc_top, double pc_1, double row_top, double row_1, double surf) {
  return pc_top + pc_1 + row_top + row_1 + surf;
}
__device__ __forceinline__ double st_t4_bar(const StCol& C, double hs_b, double w, double t) {
  return hs_b * (-w) * (C.eg * SB * 4.0) * (t * t * t);
}

// ---------------------------------------------------------------------------
// soil_temperature! reversed for column c on one thread.  tin, liq0, ice0, tg0, th0 are the
// step's inputs, B the band factors.  Tb, liqb, iceb, tgb, thb hold on entry the adjoints of
// the quantities after the call and on return those of its inputs; forcb is the forcing's,
// and wsb/bsb/sucb are the parameters'.
// ---------------------------------------------------------------------------
static __device__ __noinline__ void soil_temperature_reverse(const Dims& D, const clmgb_soiltemp_fields& f,
                                                      const clmgb_soilwater_fields& fw, int64_t c, double dtime,
                                                      int snow_method, const double* fact, const double* tin,
                                                      const double* liq0, const double* ice0, double tg0, double th0,
                                                      double forc, const CfBand& B, double* Tb, double* liqb,
                                                      double* iceb, double& tgb, double& thb, double& forcb,
                                                      double* wsb, double* bsb, double* sucb) {
  const int nlevsno = D.nlevsno, nlevgrnd = D.nlevgrnd, nw = nlevsno + nlevgrnd;
  StCol C;
  st_column(C, D, f, c, dtime, snow_method, tg0, th0);
  const int jjtop = C.jjtop, jj1 = 1 + nlevsno, n = B.n, rsw = -(int)C.snl;
  st_sums(C, D, f, c, forc, tin[jjtop], tin[jj1]);
  StLayer ly[MAXL + 2];
  StItf it[MAXL + 2];
  StPc pc[MAXL + 2];
  StRow row[MAXL + 2];
  double w[MAXROWS];
  for (int jj = jjtop; jj <= nw; jj++) ly[jj] = st_layer(C, D, f, fw, c, jj, tin[jj], liq0[jj], ice0[jj]);
  double tkh, dtkh;
  st_tkh(D, f, c, ly[jj1].v, tkh, dtkh);
  auto row_of = [&](int jj) { return jj < jj1 ? jj - jjtop : rsw + jj - nlevsno; };
  for (int jj = jjtop; jj <= nw; jj++) {
    const int j = jj - nlevsno;
    it[jj] = st_interface(D, f, c, jj, ly[jj].v, jj < nw ? ly[jj + 1].v : 0.0, tin[jj], jj < nw ? tin[jj + 1] : 0.0);
    pc[jj] = st_phase_change(C, D, f, fw, c, jj, B.x[row_of(jj)], liq0[jj], ice0[jj], fact[jj],
                             Tb[jj] + st_tgrnd_level(C, j, tgb), liqb[jj], iceb[jj]);
    w[row_of(jj)] = pc[jj].t;
  }
  const double thpc = thb + st_tgrnd_h2osfc(C, tgb);
  if (zero_bits(C.fh)) {                    // t_h2osfc took the soil-1 temperature
    w[rsw + 1] += thpc;
    w[rsw] = 0.0;
  } else {
    w[rsw] = thpc;
  }
  band_lu_transpose_solve<2, 2>(B.lu, B.piv, w, n);    // w = lambda
  // -lambda x of row r's entry d
  auto entry = [&](int r, int d) { return r - 2 + d >= 0 && r - 2 + d < n ? -w[r] * B.x[r - 2 + d] : 0.0; };
  for (int jj = jjtop; jj <= nw; jj++) {
    const int j = jj - nlevsno, r = row_of(jj);
    const StItf p = jj > jjtop ? it[jj - 1] : StItf{0.0, 0.0, 0.0, 0.0, 0.0};
    const StRowIn a = {j,         w[r],      entry(r, 0), entry(r, 1), entry(r, 2), entry(r, 3), entry(r, 4), fact[jj],
                       tin[jj],   it[jj].fn, p.fn,        it[jj].tk,   p.tk,        it[jj].rdz,  p.rdz,
                       j <= 1 ? st_sabg(D, f, c, jj) : 0.0};
    row[jj] = st_row(C, nlevgrnd, a);
  }
  const StSurf sf = st_surface(C, tkh, tin[jj1], fact[jj1], w[rsw], entry(rsw, 2), entry(rsw, 3), w[rsw + 1],
                               entry(rsw + 1, 1), entry(rsw + 1, 2));
  const bool snow = C.snl < 0;
  const double dh = st_dhsdT_bar(pc[jjtop].dh, snow ? pc[jj1].dh : 0.0, row[jjtop].dh, snow ? row[jj1].dh : 0.0, sf.dh);
  const double hst = row[jjtop].hst, hss = row[jj1].hss + sf.hss;
  tgb = dh * (-C.w_set) * (4.0 * C.eg * SB) * (3.0 * (tg0 * tg0));
  forcb += (hss + sf.hsh) * C.wb_set + hst * C.wb_act;
  thb = sf.th + st_t4_bar(C, sf.hsh, C.w_set, th0);
  double d_p = 0.0, kb_p = 0.0;
  for (int jj = jjtop; jj <= nw; jj++) {
    const int j = jj - nlevsno;
    const StRow nx = jj < nw ? row[jj + 1] : StRow{0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    const double fnb = row[jj].n + nx.np;
    const double dT = jj < nw ? tin[jj + 1] - tin[jj] : 0.0;
    const double kb = row[jj].k + nx.kp + fnb * dT * it[jj].rdz;
    const double d = fnb * it[jj].tk * it[jj].rdz;
    double t = row[jj].t + d_p - d, fb = pc[jj].f + row[jj].f, hb = kb_p + kb * it[jj].da;
    if (j == 1) {
      t += sf.t1 + st_t4_bar(C, hss, C.w_set, tin[jj]);
      fb += sf.f1;
      hb += sf.tkh * dtkh;
    }
    if (jj == jjtop) t += st_t4_bar(C, hst, C.w_act, tin[jj]);
    const StCap q = st_capacity(C, D, f, fw, c, jj, liq0[jj], ice0[jj], fact[jj]);
    Tb[jj] = t;
    liqb[jj] = pc[jj].liq + fb * q.l + hb * ly[jj].dl;
    iceb[jj] = pc[jj].ice + fb * q.i + hb * ly[jj].di;
    if (j >= 1) {
      wsb[j] = pc[jj].ws + fb * q.w + hb * ly[jj].dw;
      bsb[j] = pc[jj].bs;
      sucb[j] = pc[jj].suc;
    }
    d_p = d;
    kb_p = kb * it[jj].db;
  }
}

// Whether k_soil_reverse (adjoint_soil_packed.cu) takes column c whole: its log holds
// soil_temperature!, and the solve of a hydrology column.
__device__ __forceinline__ bool step_reversed_here(const Dims& D, const clmgb_soiltemp_fields& ft,
                                                   const clmgb_soilwater_fields& fw, const SubstepLogView& lg,
                                                   int64_t c) {
  if (!lg.rec || !lg.st) return false;
  if (fw.mask_hydrology[c]) return richards_reversed_here(D, ft, fw, lg, c);
  const int64_t snl = ft.col_snl[c];
  return ft.mask_nolakec[c] && snl <= 0 && snl >= -D.nlevsno;
}

}  // namespace clmgb
