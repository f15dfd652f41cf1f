// adjoint_richards_packed.cu — the reverse of the moisture-form solve of logged columns, a
// thread per (level, column) item.
//
// mf_substep_reverse (adjoint_richards.cuh) reverses a substep on one thread per column:
// 16,384 columns are 512 warps, one per sub-partition, each a chain of some 2,000 dependent
// FP64 instructions a level through arrays in local memory (FP64 unit 30 % busy, half of the
// stalls on local memory).  Here a block takes RV_COLS columns of the work order, a half-warp
// per level, and a level's values stay in the registers of its thread across a substep:
//
//   saturation | powers and hydraulics | interface flux | band row and right-hand sides |
//   the solve and the transposed solve | interface adjoints | hydraulic adjoints | water
//
// with neighbours' values through shared memory and a block barrier between the stages.  The
// two tridiagonal systems, A dwat = r and A^T lambda = g, run side by side on the half-warps
// of warp 0 as one recurrence (A^T's bands are A's, shifted), their divisions in line; a
// second block of the SM works meanwhile.
//
// Measured, 16,384 columns with one to some ten substeps: 3,120 us of the column kernel for
// the solve on a thread per column, 372 us here.  What bounds it: instructions of the powers
// and divisions and the two tridiagonal chains (20 levels of about 450 cycles) on one warp
// of a block.
#include "adjoint_richards.cuh"
#include "clmgb_device.cuh"
#include "launch.h"

namespace clmgb {

namespace {

constexpr int RV_COLS = 16;
// arrays of (levels + 2) rows of RV_COLS in shared memory; those of one line share storage
enum RvArray {
  RV_S = 0, RV_HALF = 0,          // saturation; half a level's s1 adjoint, for the next level
  RV_SMP, RV_DSW,                 // matric potential and its derivative in water
  RV_QO, RV_NUM = RV_QO,          // interface flux; its adjoint in the next level's smp
  RV_D1, RV_DSB = RV_D1,          // the flux's derivatives; the adjoint in the next level's dsmpdw
  RV_D2, RV_WSB = RV_D2,          // ... and in 1/watsat
  RV_A, RV_B, RV_C,               // the band
  RV_XF, RV_XT, RV_GF, RV_GT,     // solutions and modified super-diagonals: A, A^T
  RV_DT,                          // dtsub / dz
  RV_ARRAYS
};

// T: threads of a block (a half-warp per level), two blocks to an SM
template <int T>
__global__ void __launch_bounds__(T, 2)
k_richards_reverse(Dims D, int64_t nc, clmgb_soiltemp_fields ft, clmgb_soilwater_fields fw, clmgb_swm_config cfg,
                   double dtime, clmgb_step_adjoint adj, SubstepLogView lg, const uint32_t* __restrict__ order) {
  extern __shared__ double rv_smem[];
  const int64_t ld = D.ldc;
  const int nlevsoi = D.nlevsoi, joff = D.nlevsno, rows = nlevsoi + 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k = lane & (RV_COLS - 1), j = 2 * warp + (lane >> 4) + 1;
  double* const sm = rv_smem + k;
  auto at = [&](int a, int jj) -> double& { return sm[(a * rows + jj) * RV_COLS]; };
  const int64_t i = (int64_t)blockIdx.x * RV_COLS + k;
  // ---- the column, the same for its threads ----
  int64_t c = 0;
  int nl = 0, nacc = 0;
  if (i < nc) {
    c = order ? (int64_t)order[i] : i;
    if (richards_reversed_here(D, ft, fw, lg, c)) {
      nl = (int)fw.col_nbedrock[c];
      nacc = lg.count[c];
    }
  }
  if (!__syncthreads_or(nl)) return;
  const bool on = j <= nl;
  const bool flux = cfg.lower_boundary_condition == CLMGB_BC_FLUX;
  const bool zero = cfg.lower_boundary_condition == CLMGB_BC_ZERO_FLUX;
  const double* const rec = lg.rec + c * lg.stride;
  // ---- the level's constants ----
  double ws = 1.0, bb = 1.0, suc = 1.0, ks = 0.0, imp = 0.0, dz = 1.0, root = 0.0, rden = 0.0;
  double ice = 0.0, exi = 0.0, icef = 0.0;
  if (nl && j <= nlevsoi) {
    // set_soil_water_fractions! of the level
    exi = LV(fw.excess_ice, c, j, ld);
    dz = LVc(fw.dz, c, j + joff, ld);
    ws = LV(fw.watsat, c, j, ld);
    ice = ft.mask_nolakec[c] ? lg.st[c * (int64_t)CLMGB_LOG_ST_STRIDE + ST_ICE + j + joff - 1]
                             : LV(ft.h2osoi_ice, c, j + joff, ld);
    const double vol_ice = jl_min(ws, jl_div(ice + exi, (dz + jl_div(exi, DENICE)) * DENICE));
    icef = jl_min(1.0, jl_div(vol_ice, ws));
    LV(fw.eff_porosity, c, j, ld) = jl_max(0.01, ws - vol_ice);
    LV(fw.icefrac, c, j, ld) = icef;
    at(RV_S, j) = icef;
  }
  __syncthreads();
  double lamQ = 0.0, lamL = 0.0;
  bool wt = false;
  if (on) {
    const double f = (j == nl) ? icef : 0.5 * (icef + at(RV_S, j + 1));
    imp = cm_pow(10.0, -cfg.e_ice * f);
    bb = LV(fw.bsw, c, j, ld);
    suc = LV(fw.sucsat, c, j, ld);
    ks = LV(fw.hksat, c, j, ld);
    root = LVc(fw.qflx_rootsoi, c, j, ld);
    lamL = LV(adj.lam_h2osoi_liq, c, joff + j, ld);
    if (adj.lam_qcharge && !qcharge_replaced(D, fw, cfg, c)) lamQ = adj.lam_qcharge[c];
    const double z = LVc(fw.z, c, joff + j, ld);
    wt = cfg.lower_boundary_condition == CLMGB_BC_WATERTABLE && nl <= watertable_level(D, fw, c);
    if (j < nl) rden = jl_div(1.0, M_TO_MM * (LVc(fw.z, c, joff + j + 1, ld) - z));
    else if (wt) rden = jl_div(1.0, M_TO_MM * (fw.zwt[c] - z));
  }
  const bool last = j == nl;
  const double rws = jl_div(1.0, ws), dzw = dz * DENH2O, rdzw = jl_div(1.0, dzw), dzmm = M_TO_MM * dz;
  const double e = 2.0 * bb + 3.0, ik = imp * ks, infl = on ? fw.qflx_infl[c] : 0.0;
  __syncthreads();
  at(RV_S, j) = rws;                                 // (rows beyond the levels exist: j <= nlevsoi + 1)
  __syncthreads();
  const double hrw = 0.5 * rws, hrwn = on && !last ? 0.5 * at(RV_S, j + 1) : 0.0;
  RvAcc acc = {0.0, 0.0, 0.0, 0.0, 0.0};
  const int steps = __reduce_max_sync(0xffffffffu, nacc);   // of the block: every warp has all its columns
  double liq_n = on && steps && nacc == steps ? rec[(int64_t)(steps - 1) * SUB_REC + j - 1] : 0.0;
  for (int s = steps - 1; s >= 0; s--) {
    const bool act = on && s < nacc;
    double dts = 0.0;
    RvSat sat = {};
    __syncthreads();
    if (act) {
      dts = rec[(int64_t)s * SUB_REC + MAXSOI];
      sat = rv_saturation(liq_n, dzw, ws);
      at(RV_S, j) = sat.s;
    }
    if (on && s > 0 && s - 1 < nacc) liq_n = rec[(int64_t)(s - 1) * SUB_REC + j - 1];
    __syncthreads();
    RvPow p = {};
    RvHyd h = {};
    if (act) {
      p = rv_powers(sat.s, last ? 0.0 : at(RV_S, j + 1), last, e, bb);
      h = rv_hydraulics(p, ik, e, bb, suc, rws);
      at(RV_SMP, j) = h.smp;
      at(RV_DSW, j) = h.dsw;
    }
    __syncthreads();
    RvFlux fl = {};
    double dsw_n = 0.0;
    if (act) {
      if (!last) {
        dsw_n = at(RV_DSW, j + 1);
        fl = rv_flux(h, at(RV_SMP, j + 1), dsw_n, rden, hrw, hrwn);
      } else {
        fl = rv_flux_bottom(h, wt, flux, rden, rws);
      }
      at(RV_QO, j) = fl.qo;
      at(RV_D1, j) = fl.d1;
      at(RV_D2, j) = fl.d2;
    }
    __syncthreads();
    const double cq = last ? lamQ * jl_div(dts, dtime) : 0.0;
    double dt = 0.0;
    if (act) {
      dt = jl_div(dts, dzmm);
      const RvRow w = rv_row(j == 1 ? infl : at(RV_QO, j - 1), j == 1 ? 0.0 : at(RV_D1, j - 1),
                             j == 1 ? 0.0 : at(RV_D2, j - 1), fl, root, dt, lamL, dzmm, last, cq, flux, zero, h);
      at(RV_A, j) = w.a;
      at(RV_B, j) = w.b;
      at(RV_C, j) = w.c;
      at(RV_XF, j) = w.x;
      at(RV_XT, j) = w.g;
      at(RV_DT, j) = dt;
    }
    __syncthreads();
    // A dwat = x on the lower half-warp, A^T lambda = g on the upper one
    if (warp == 0 && nl && s < nacc) {
      const bool tr = lane >= RV_COLS;
      const int ax = tr ? RV_XT : RV_XF, ag = tr ? RV_GT : RV_GF;
      double x = 0.0, g = 0.0;
      for (int jj = 1; jj <= nl; jj++) {
        const double sub = jj == 1 ? 0.0 : (tr ? at(RV_C, jj - 1) : at(RV_A, jj));
        const double sup = jj == nl ? 0.0 : (tr ? at(RV_A, jj + 1) : at(RV_C, jj));
        rv_eliminate(tr, jj == 1, sub, at(RV_B, jj), sup, at(ax, jj), x, g);
        at(ax, jj) = x;
        at(ag, jj) = g;
      }
      for (int jj = nl - 1; jj >= 1; jj--) {
        x = rv_fma(-at(ag, jj), x, at(ax, jj));
        at(ax, jj) = x;
      }
    }
    __syncthreads();
    RvItf t = {};
    if (act) {
      const double dw = at(RV_XF, j);
      double q = at(RV_XT, j) * dt;
      if (!last) {
        q = rv_fma(-at(RV_XT, j + 1), at(RV_DT, j + 1), q);
        t = rv_interface(q, h, dsw_n, fl, rden, hrw, hrwn, dw, at(RV_XF, j + 1));
        at(RV_NUM, j + 1) = t.n_smpb;
        at(RV_DSB, j + 1) = t.n_dswb;
        at(RV_WSB, j + 1) = t.n_wk;
      } else {
        t = rv_interface_bottom(q, cq, h, fl, wt, flux, zero, rden, rws, dw);
      }
    }
    __syncthreads();
    double sb = 0.0, wsb = 0.0;
    if (act) {
      if (j > 1) {
        t.smpb += at(RV_NUM, j);
        t.dswb += at(RV_DSB, j);
        t.wk += at(RV_WSB, j);
      }
      double s1b;
      rv_hydraulics_reverse(t, h, p, last, e, bb, rws, acc, sb, wsb, s1b);
      if (!last) at(RV_HALF, j + 1) = s1b;
    }
    __syncthreads();
    if (act) {
      if (j > 1) sb += at(RV_HALF, j);
      rv_water_reverse(sat, sb, wsb, rws, rdzw, lamL, acc);
    }
  }
  // the ice impedance 10^(-e_ice icefrac) and set_soil_water_fractions!
  const double ib = on ? rv_impedance_bar(cfg.e_ice, acc.hp, ks, imp) : 0.0;
  __syncthreads();
  at(RV_S, j) = 0.5 * ib;
  __syncthreads();
  if (!on) return;
  LV(adj.lam_h2osoi_ice, c, j + joff, ld) +=
      rv_fractions_reverse(ib, j > 1 ? at(RV_S, j - 1) : 0.0, last, ws, ice, exi, dz, acc.ws);
  LV(adj.lam_h2osoi_liq, c, j + joff, ld) = lamL;
  if (adj.grad_watsat) LV(adj.grad_watsat, c, j, ld) += acc.ws;
  if (adj.grad_bsw) LV(adj.grad_bsw, c, j, ld) += rv_fma(2.0, acc.e, acc.b);
  if (adj.grad_sucsat) LV(adj.grad_sucsat, c, j, ld) += acc.suc;
  if (adj.grad_hksat) LV(adj.grad_hksat, c, j, ld) += acc.hp * imp;
}

}  // namespace

cudaError_t launch_richards_reverse(const Dims& D, int64_t nc, const clmgb_soiltemp_fields& ft,
                                    const clmgb_soilwater_fields& fw, const clmgb_swm_config& cfg, double dtime,
                                    const clmgb_step_adjoint& adj, const SubstepLogView& lg, const uint32_t* order,
                                    cudaStream_t s) {
  const size_t smem = sizeof(double) * (size_t)RV_ARRAYS * (D.nlevsoi + 2) * RV_COLS;
  const unsigned grid = (unsigned)((nc + RV_COLS - 1) / RV_COLS);
  const int threads = 32 * ((D.nlevsoi + 1) / 2);
  auto kern = threads <= 320 ? k_richards_reverse<320> : k_richards_reverse<32 * ((MAXSOI + 1) / 2)>;
  const cudaError_t e = allow_dynamic_smem(kern, sizeof(double) * (size_t)RV_ARRAYS * (MAXSOI + 2) * RV_COLS);
  if (e != cudaSuccess) return e;
  kern<<<grid, threads, smem, s>>>(D, nc, ft, fw, cfg, dtime, adj, lg, order);
  return cudaGetLastError();
}

}  // namespace clmgb
