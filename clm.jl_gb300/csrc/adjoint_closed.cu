// adjoint_closed.cu — reverse of one column step written out by hand (no tape).
//
// The recording kernel (adjoint_step.cu) differentiates soil_temperature! by
// replaying it through a recording scalar and sweeping the tape.  This kernel runs
// the production arithmetic on plain values (soil_temperature_col with a per-thread
// state accessor, so the forward is the production step bit for bit) and then
// applies the transpose of every stage's derivative, last stage first:
//
//   t_grnd        tg = fse ts + (1-fse-fh) t1 + fh th, or (1-fh) t1 + fh th
//                 (_tgrnd_kernel!, soil_temperature.jl:224-247)
//   phase change  per level: the melt/freeze decision, hm, xm, the new ice and
//                 liquid water and the temperature correction
//                 (_phase_change_beta_kernel!, :1929-2230)
//   band solve    lambda = A^-T xbar from the factors the forward kept,
//                 rbar = lambda, Abar = -lambda x^T (band_solve! rule,
//                 enzyme_rules.jl:80-107)
//   assembly      the rows of set_rhs_vec! / set_matrix! (:1365-1748)
//   heat flux     fn, the ground heat flux sums dhsdT, hs_soil, hs_h2osfc,
//                 hs_top_snow (:1200-1263, :1271-1319)
//   capacity      fact = dtime/cv (top layer with the CAPR factor), cv (:599-942)
//   conductivity  interface tk, tk_h2osfc, layer thk (Johansen for soil, Jordan or
//                 Sturm for snow) (:647-776)
//
// The Richards substeps are reversed by mf_substep_reverse (adjoint_richards.cuh,
// shared with the recording kernel); set_soil_water_fractions! and the ice
// impedance are reversed here in closed form.  Every decision (branch, clamp,
// pivot) is the forward's; the derivative of a Julia max/min passes to the
// argument it returned (the constant when a tie returned it), as in the recording
// kernel, so both kernels differentiate the same piecewise function.
//
// Elementwise stages keep their local partial derivatives from the forward sweep
// (thk and fact with respect to liquid water, ice and watsat; the interface
// conductivity with respect to its two layers), so the reverse is a few
// multiply-adds per level.
//
// With a substep log (clmgb_substep_log, written by clmgb_column_step_logged) the
// Richards forward is not run again: its accepted substeps' starting water comes
// from the log, and so do the solve's outputs; with the soil_temperature! records
// too, the solve is reversed beforehand by a kernel with a thread per level
// (k_richards_reverse, adjoint_richards_packed.cu).  Without a log (or for a column
// the log could not hold) the substep loop runs on values here, keeping the same
// checkpoints in the reserved per-slot storage, and is reversed here.
#include "adjoint_richards.cuh"
#include "adjoint_soil.cuh"
#include "clmgb_device.cuh"
#include "launch.h"
#include "work_order.cuh"

namespace clmgb {

constexpr int CF_BLOCK = 64;

// The column's active state in per-thread storage, values only.
struct CfState {
  typedef double S;
  double t[MAXL + 2], liq[MAXL + 2], ice[MAXL + 2], fact[MAXL + 2];
  double icefrac[MAXSOI + 2];
  double tg, th, qc, forc;
  const double *ws, *bs, *suc, *ks;
  int64_t c, ld;
  CfBand* band;
  __device__ __forceinline__ double& T(int jj) { return t[jj]; }
  __device__ __forceinline__ double& Liq(int jj) { return liq[jj]; }
  __device__ __forceinline__ double& Ice(int jj) { return ice[jj]; }
  __device__ __forceinline__ double& Fact(int jj) { return fact[jj]; }
  __device__ __forceinline__ double& Icefrac(int j) { return icefrac[j]; }
  __device__ __forceinline__ double& Tgrnd() { return tg; }
  __device__ __forceinline__ double& Th2osfc() { return th; }
  __device__ __forceinline__ double& Qcharge() { return qc; }
  __device__ __forceinline__ double ForcLwrad() const { return forc; }
  __device__ __forceinline__ double Watsat(int j) const { return LVc(ws, c, j, ld); }
  __device__ __forceinline__ double Bsw(int j) const { return LVc(bs, c, j, ld); }
  __device__ __forceinline__ double Sucsat(int j) const { return LVc(suc, c, j, ld); }
  __device__ __forceinline__ double Hksat(int j) const { return LVc(ks, c, j, ld); }
  // the production factorisation, keeping the factors, pivots and solution
  __device__ __forceinline__ void band_solve(double* ab, double* x, int n) {
    band_lu_factor_solve<2, 2>(ab, x, band->piv_s, n);
    band->n = n;
    for (int k = 0; k < n * 7; k++) band->lu_s[k] = ab[k];
    for (int r = 0; r < n; r++) band->x_s[r] = x[r];
    band->lu = band->lu_s;
    band->x = band->x_s;
    band->piv = band->piv_s;
  }
};

// ---------------------------------------------------------------------------
// The kernel: one thread per column, columns handed out by a work counter.
// ---------------------------------------------------------------------------
struct CfSub {
  double* sub;
  int maxsub;
  int64_t slots;
};

__device__ __forceinline__ double& cf_sub(const CfSub& S, int64_t slot, int sidx, int j) {
  return S.sub[((slot >> 5) * ((int64_t)S.maxsub * SUB_REC) + (int64_t)sidx * SUB_REC + j) * 32 + (slot & 31)];
}

// 8 blocks of 64 per SM (128 registers): 1,216 resident blocks, so each thread of a
// 65,536-column launch takes one column and no second round of columns trails the
// first (6 blocks at the 168 registers the compiler chose otherwise)
__global__ void __launch_bounds__(CF_BLOCK, 8)
k_column_step_vjp_cf(Dims D, int64_t nc, clmgb_soiltemp_fields ft, clmgb_soilwater_fields fw, clmgb_swm_config cfg,
                     double dtime, int snow_method, double* t_ssbef, double* t_h2osfc_bef, clmgb_step_adjoint adj,
                     CfSub S, SubstepLogView lg, unsigned long long* queue, const uint32_t* order,
                     uint32_t* col_status, uint32_t* dev_status) {
  const int64_t ld = D.ldc;
  const int nlevsno = D.nlevsno, nlevgrnd = D.nlevgrnd, nlevsoi = D.nlevsoi;
  const int nlev = nlevsno + D.nlevmax;
  const int nw = nlevsno + nlevgrnd;
  const int joff = nlevsno;
  const int64_t slot = (int64_t)blockIdx.x * CF_BLOCK + threadIdx.x;
  CfBand band;
  for (;;) {
    const int64_t k = (int64_t)atomicAdd(queue, 1ULL);
    if (k >= nc) break;
    const int64_t c = order ? (int64_t)order[k] : k;
    const bool do_t = ft.mask_nolakec[c] != 0, do_w = fw.mask_hydrology[c] != 0;
    if (step_reversed_here(D, ft, fw, lg, c)) continue;     // k_richards_reverse and k_soil_reverse have
    if (!do_t && !do_w) {     // the step leaves the column alone: identity
      if (col_status) col_status[c] = 0;
      continue;
    }
    uint32_t st = 0;
    const int64_t snl = ft.col_snl[c];
    if (snl > 0 || snl < -nlevsno) {
      st = CLMGB_COL_LEVEL_RANGE;
      if (col_status) col_status[c] = st;
      if (dev_status) atomicOr(dev_status, st);
      continue;
    }
    const int jjtop = (int)snl + 1 + nlevsno;
    if (ft.frac_h2osfc[c] > 0.0 || ft.h2osno_no_layers[c] > 0.0) st |= CLMGB_COL_ADJ_UNSUPPORTED;
    for (int j = 1; j <= nlevgrnd; j++)
      if (LV(ft.excess_ice, c, j, ld) != 0.0) st |= CLMGB_COL_ADJ_UNSUPPORTED;
    // ---- load the state, keep the inputs ----
    CfState V;
    V.c = c;
    V.ld = ld;
    V.ws = fw.watsat;
    V.bs = fw.bsw;
    V.suc = fw.sucsat;
    V.ks = fw.hksat;
    V.band = &band;
    band.n = 0;
    double tin[MAXL + 2], liq0[MAXL + 2], ice0[MAXL + 2];
    for (int jj = 1; jj <= nlev; jj++) {
      V.t[jj] = LV(ft.t_soisno, c, jj, ld);
      V.liq[jj] = LV(ft.h2osoi_liq, c, jj, ld);
      V.ice[jj] = LV(ft.h2osoi_ice, c, jj, ld);
      tin[jj] = V.t[jj];
      liq0[jj] = V.liq[jj];
      ice0[jj] = V.ice[jj];
    }
    for (int jj = 1; jj <= nw; jj++) V.fact[jj] = LV(ft.fact, c, jj, ld);
    for (int j = 1; j <= nlevsoi; j++) V.icefrac[j] = LV(fw.icefrac, c, j, ld);
    V.tg = ft.t_grnd[c];
    V.th = ft.t_h2osfc[c];
    V.forc = ft.forc_lwrad[c];
    V.qc = fw.qcharge[c];
    const double tg0 = V.tg, th0 = V.th;
    // ---- soil_temperature!: run here, or its record read from the log ----
    bool st_full = false;
    if (do_t) {
      if (t_ssbef)
        for (int jj = 1; jj <= nlev; jj++) LV(t_ssbef, c, jj, ld) = V.t[jj];
      if (t_h2osfc_bef) t_h2osfc_bef[c] = V.th;
      uint32_t s1;
      if (lg.st) {
        const double* rec = lg.st + c * (int64_t)CLMGB_LOG_ST_STRIDE;
        s1 = (uint32_t)rec[ST_STATUS];
        band.n = (int)rec[ST_N];
        band.lu = rec + ST_LU;
        band.x = rec + ST_X;
        band.piv = reinterpret_cast<const uint8_t*>(rec + ST_PIV);
        for (int jj = jjtop; jj <= nlev; jj++) V.t[jj] = rec[ST_T + jj - 1];
        for (int jj = jjtop; jj <= nw; jj++) {
          V.liq[jj] = rec[ST_LIQ + jj - 1];
          V.ice[jj] = rec[ST_ICE + jj - 1];
          V.fact[jj] = rec[ST_FACT + jj - 1];
        }
        V.tg = rec[ST_TG];
        V.th = rec[ST_TH];
      } else {
        s1 = soil_temperature_col(D, ft, c, dtime, snow_method, V);
      }
      st |= s1;
      st_full = !(s1 & (CLMGB_COL_URBAN | CLMGB_COL_PATCH_RANGE | CLMGB_COL_LEVEL_RANGE)) && band.n > 0;
    }
    // ---- set_soil_water_fractions! and soil_water! ----
    MfLane L;
    bool rich = false;
    int nacc = 0;
    const double* logc = nullptr;     // this column's log region, when it holds the solve
    if (do_w) {
      water_fractions_col(D, fw, c, V);
      rich = mf_begin(L, D, fw, cfg, dtime, c, V);
      if (!rich) {
        st |= L.status;
      } else {
        const int32_t cnt = lg.rec ? lg.count[c] : -1;
        if (cnt >= 0 && cnt <= lg.cap) {
          logc = lg.rec + c * lg.stride;
          nacc = cnt;
          const double* fin = logc + (int64_t)lg.cap * SUB_REC;
          uint32_t rs = (uint32_t)fin[3 * MAXSOI + 2];
          for (int j = 1; j <= L.nlayers; j++) {
            V.liq[joff + j] = fin[j - 1];
            LV(fw.smp_l, c, j, ld) = fin[MAXSOI + j - 1];
            LV(fw.hk_l, c, j, ld) = fin[2 * MAXSOI + j - 1];
          }
          V.qc = fin[3 * MAXSOI];
          fw.num_substeps[c] = fin[3 * MAXSOI + 1];
          st |= rs;
        } else {
          bool done = false;
          while (!done) {
            if (L.fresh && nacc < S.maxsub)
              for (int j = 1; j <= L.nlayers; j++) cf_sub(S, slot, nacc, j - 1) = L.liq[j];
            const double dts = L.dtsub, dtd = L.dtdone;
            done = mf_attempt(L, D, fw, cfg, dtime, V);
            if (L.dtdone != dtd) {
              if (nacc < S.maxsub) {
                cf_sub(S, slot, nacc, MAXSOI) = dts;
                cf_sub(S, slot, nacc, MAXSOI + 1) = dtd;
              }
              nacc++;
            }
          }
          st |= mf_end(L, D, fw, V);
          if (nacc > S.maxsub) st |= CLMGB_COL_TAPE_FULL;
        }
      }
    }
    // ---- the final forward state ----
    for (int jj = jjtop; jj <= nlev; jj++) LV(ft.t_soisno, c, jj, ld) = V.t[jj];
    for (int jj = jjtop; jj <= nw; jj++) {
      LV(ft.h2osoi_liq, c, jj, ld) = V.liq[jj];
      LV(ft.h2osoi_ice, c, jj, ld) = V.ice[jj];
      if (do_t) LV(ft.fact, c, jj, ld) = V.fact[jj];
    }
    if (do_w)
      for (int j = 1; j <= nlevsoi; j++) LV(fw.icefrac, c, j, ld) = V.icefrac[j];
    ft.t_grnd[c] = V.tg;
    ft.t_h2osfc[c] = V.th;
    if (do_w) fw.qcharge[c] = V.qc;

    if (!(st & CLMGB_COL_TAPE_FULL)) {
      // ---- seeds: the adjoints of the step's outputs ----
      double Tb[MAXL + 2], liqb[MAXL + 2], iceb[MAXL + 2];
      for (int jj = jjtop; jj <= nw; jj++) {
        Tb[jj] = LV(adj.lam_t_soisno, c, jj, ld);
        liqb[jj] = LV(adj.lam_h2osoi_liq, c, jj, ld);
        iceb[jj] = LV(adj.lam_h2osoi_ice, c, jj, ld);
      }
      double tgb = adj.lam_t_grnd[c], thb = adj.lam_t_h2osfc[c], forcb = 0.0;
      double wsb[MAXGRND + 2], bsb[MAXGRND + 2], sucb[MAXGRND + 2];
      for (int j = 1; j <= nlevgrnd; j++) {
        wsb[j] = 0.0;
        bsb[j] = 0.0;
        sucb[j] = 0.0;
      }
      // ---- the substeps in reverse ----
      if (rich) {
        const int nl = L.nlayers;
        const double lamQ = adj.lam_qcharge && !qcharge_replaced(D, fw, cfg, c) ? adj.lam_qcharge[c] : 0.0;
        double lamL[MAXSOI + 1], liqs[MAXSOI + 1];
        double wsv[MAXSOI + 2], bbv[MAXSOI + 2], sucv[MAXSOI + 2], ksv[MAXSOI + 2];
        RichardsBar RB;
        for (int j = 1; j <= nl; j++) {
          lamL[j] = liqb[joff + j];
          RB.ws[j] = 0.0; RB.b[j] = 0.0; RB.e[j] = 0.0; RB.suc[j] = 0.0; RB.hp[j] = 0.0;
          wsv[j] = LV(fw.watsat, c, j, ld);
          bbv[j] = LV(fw.bsw, c, j, ld);
          sucv[j] = LV(fw.sucsat, c, j, ld);
          ksv[j] = LV(fw.hksat, c, j, ld);
        }
        for (int sidx = nacc - 1; sidx >= 0; sidx--) {
          double dts;
          if (logc) {
            const double* rec = logc + (int64_t)sidx * SUB_REC;
            for (int j = 1; j <= nl; j++) liqs[j] = rec[j - 1];
            dts = rec[MAXSOI];
          } else {
            for (int j = 1; j <= nl; j++) liqs[j] = cf_sub(S, slot, sidx, j - 1);
            dts = cf_sub(S, slot, sidx, MAXSOI);
          }
          mf_substep_reverse(D, fw, cfg, dtime, c, nl, L.dzv, L.imp, wsv, bbv, sucv, ksv, dts, liqs, lamL, lamQ, RB);
        }
        // the ice impedance 10^(-e_ice icefrac) and set_soil_water_fractions!
        double half_above = 0.0;
        for (int j = 1; j <= nl; j++) {
          const double ib = rv_impedance_bar(cfg.e_ice, RB.hp[j], ksv[j], L.imp[j]);
          iceb[j + joff] += rv_fractions_reverse(ib, half_above, j == nl, wsv[j], V.ice[j + joff],
                                                 LV(ft.excess_ice, c, j, ld), LVc(fw.dz, c, j + joff, ld), RB.ws[j]);
          half_above = 0.5 * ib;
          liqb[joff + j] = lamL[j];
          if (adj.grad_watsat) LV(adj.grad_watsat, c, j, ld) += RB.ws[j];
          if (adj.grad_bsw) LV(adj.grad_bsw, c, j, ld) += rv_fma(2.0, RB.e[j], RB.b[j]);
          if (adj.grad_sucsat) LV(adj.grad_sucsat, c, j, ld) += RB.suc[j];
          if (adj.grad_hksat) LV(adj.grad_hksat, c, j, ld) += RB.hp[j] * L.imp[j];
        }
      }
      // ---- soil_temperature! in reverse ----
      if (st_full)
        soil_temperature_reverse(D, ft, fw, c, dtime, snow_method, V.fact, tin, liq0, ice0, tg0, th0, V.forc, band,
                                 Tb, liqb, iceb, tgb, thb, forcb, wsb, bsb, sucb);
      // ---- adjoints of the step's inputs ----
      for (int jj = jjtop; jj <= nw; jj++) {
        LV(adj.lam_t_soisno, c, jj, ld) = Tb[jj];
        LV(adj.lam_h2osoi_liq, c, jj, ld) = liqb[jj];
        LV(adj.lam_h2osoi_ice, c, jj, ld) = iceb[jj];
      }
      adj.lam_t_grnd[c] = tgb;
      adj.lam_t_h2osfc[c] = thb;
      if (adj.lam_forc_lwrad) adj.lam_forc_lwrad[c] = forcb;
      for (int j = 1; j <= nlevsoi; j++) {
        if (adj.grad_watsat) LV(adj.grad_watsat, c, j, ld) += wsb[j];
        if (adj.grad_bsw) LV(adj.grad_bsw, c, j, ld) += bsb[j];
        if (adj.grad_sucsat) LV(adj.grad_sucsat, c, j, ld) += sucb[j];
      }
    }
    if (col_status) col_status[c] = st;
    if (st && dev_status) atomicOr(dev_status, st);
  }
}

// Work order of the adjoint: the 32 columns a warp runs side by side should take
// the same paths, so the key is the Richards work (accepted substeps from the log, else
// the previous call's attempt count) and the number of snow layers.  Columns the step
// leaves alone come last.
struct VjpKey {
  clmgb_soiltemp_fields ft;
  clmgb_soilwater_fields fw;
  SubstepLogView lg;
  __device__ int operator()(int64_t c) const {
    if (!ft.mask_nolakec[c] && !fw.mask_hydrology[c]) return 0;
    int a;
    if (lg.rec) {
      const int32_t n = lg.count[c];
      a = n < 0 ? 0 : (n > lg.cap ? 15 : n);
    } else {
      const double ns = fw.num_substeps[c];
      a = ns > 0.0 ? (ns >= 15.0 ? 15 : (int)ns) : 0;
    }
    if (a > 15) a = 15;
    const int64_t snl = ft.col_snl[c];
    int sb = (int)((-snl + 3) / 4);
    sb = sb < 0 ? 0 : (sb > 3 ? 3 : sb);
    return a * 4 + sb;
  }
  __device__ void unlisted(int64_t) const {}
};

int vjp_cf_blocks_per_sm() {
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_column_step_vjp_cf, CF_BLOCK, 0) != cudaSuccess) nb = 1;
  return nb > 0 ? nb : 1;
}

cudaError_t launch_column_step_vjp_cf(const Dims& D, int64_t nc, const clmgb_soiltemp_fields& ft,
                                      const clmgb_soilwater_fields& fw, const clmgb_swm_config& cfg, double dtime,
                                      int snow_method, double* t_ssbef, double* t_h2osfc_bef,
                                      const clmgb_step_adjoint& adj, const AdjTape& tp, const SubstepLogView& lg,
                                      const QueueScratch& qs, unsigned long long* queue, int grid_blocks,
                                      uint32_t* col_status, uint32_t* dev_status, cudaStream_t s) {
  int64_t blocks = grid_blocks;
  const int64_t max_blocks = tp.slots / CF_BLOCK;
  if (blocks > max_blocks) blocks = max_blocks;
  const int64_t need = (nc + CF_BLOCK - 1) / CF_BLOCK;
  if (blocks > need) blocks = need;
  if (blocks < 1) return cudaErrorInvalidValue;
  cudaError_t e = cudaMemsetAsync(queue, 0, sizeof(unsigned long long), s);
  if (e != cudaSuccess) return e;
  const uint32_t* order = nullptr;
  if (qs.capacity >= nc && qs.order && qs.bins && nc < (int64_t)0xffffffffLL) {
    if ((e = launch_order(nc, VjpKey{ft, fw, lg}, qs.bins, qs.order, s)) != cudaSuccess) return e;
    order = qs.order;
  }
  // The logged columns.  A launch each before the others' kernel, which writes nothing that
  // they read (their columns are its `continue`).
  if (lg.rec && lg.st) {
    if ((e = launch_richards_reverse(D, nc, ft, fw, cfg, dtime, adj, lg, order, s)) != cudaSuccess) return e;
    if ((e = launch_soil_reverse(D, nc, ft, fw, dtime, snow_method, t_ssbef, t_h2osfc_bef, adj, lg, order, col_status,
                                 dev_status, s)) != cudaSuccess)
      return e;
  }
  CfSub S{tp.sub, (int)tp.maxsub, tp.slots};
  k_column_step_vjp_cf<<<(unsigned int)blocks, CF_BLOCK, 0, s>>>(D, nc, ft, fw, cfg, dtime, snow_method, t_ssbef,
                                                                 t_h2osfc_bef, adj, S, lg, queue, order,
                                                                 col_status, dev_status);
  return cudaGetLastError();
}

}  // namespace clmgb
