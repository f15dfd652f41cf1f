// adjoint_soil_packed.cu — the rest of the reverse of logged columns, a thread per (level,
// column) item: the step's final state from the log, and soil_temperature! in reverse.
//
// On a thread per column (k_column_step_vjp_cf) it is a chain through some 40 arrays of
// levels in local memory, 20 KB a thread; here a block takes SV_COLS columns of the work
// order, 8 lanes per level, and a level's values stay in registers:
//
//   sums, layer conductivity | interface, phase change | transposed band solve | rows | sums
//   of the rows' parts
//
// with neighbours' values through shared memory and a block barrier between the stages (the
// functions and their order are soil_temperature_reverse's, adjoint_soil.cuh: the same bits).
// The band solve runs a column per lane, its right-hand side, factors and pivots staged in
// shared memory by all threads.
//
// Measured, 16,384 columns: 1,100 us on a thread per column, 470 us here.  What bounds it: the
// stages in turn, the band solve's chain and the barriers (26 of 45 stall cycles an issue,
// FP64 unit 35 % busy with two blocks to an SM).  Hence four blocks of 8 columns to an SM at
// 48 registers, spills included (two at 96: 570 us, three 503; 16 columns a block 604, 4
// columns 522).
#include "adjoint_soil.cuh"
#include "clmgb_device.cuh"
#include "launch.h"

namespace clmgb {

namespace {

constexpr int SV_COLS = 8, SV_PER = 32 / SV_COLS;           // columns of a block, levels of a warp
constexpr int SV_THREADS = 32 * ((MAXL + SV_PER - 1) / SV_PER);
// arrays of rows of SV_COLS: levels 0..nw + 1, or rows of the band system
enum SvArray {
  SV_T = 0,                        // temperature at the step's start
  SV_THK, SV_KB = SV_THK,          // layer conductivity; an interface's adjoint to the layer below
  SV_TK, SV_RDZ, SV_FN,            // interface: conductivity, 1 / distance, flux
  SV_KP, SV_NP, SV_D,              // the row's adjoints of the interface above; the flux's
  SV_X, SV_W,                      // band system: solution; right-hand side, then lambda
  SV_ARRAYS
};
// the column's scalars
enum SvScalar {
  SS_DHSDT = 0, SS_SOIL, SS_H2OSFC, SS_TOP, SS_WSET, SS_WBSET, SS_WACT, SS_WBACT, SS_DTC, SS_RDH,
  SS_PC_TOP, SS_PC_1, SS_ROW_TOP, SS_ROW_1, SS_HST, SS_HSS, SS_TKH, SS_DTKH, SS_STATUS, SS_COUNT
};
constexpr int SV_ROWS = SV_THREADS / SV_COLS + 2;
constexpr size_t SV_SMEM = sizeof(double) * SV_COLS * ((size_t)SV_ARRAYS * SV_ROWS + SS_COUNT + 7 * MAXROWS) +
                           (size_t)SV_COLS * MAXROWS;

__global__ void __launch_bounds__(SV_THREADS, 4)
k_soil_reverse(Dims D, int64_t nc, clmgb_soiltemp_fields ft, clmgb_soilwater_fields fw, double dtime,
               int snow_method, double* t_ssbef, double* t_h2osfc_bef, clmgb_step_adjoint adj,
               SubstepLogView lg, const uint32_t* __restrict__ order, uint32_t* col_status, uint32_t* dev_status) {
  extern __shared__ double sv_smem[];
  const int64_t ld = D.ldc;
  const int nlevsno = D.nlevsno, nlevgrnd = D.nlevgrnd, nw = nlevsno + nlevgrnd, nlev = nlevsno + D.nlevmax;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k = lane & (SV_COLS - 1), jj = SV_PER * warp + lane / SV_COLS + 1, j = jj - nlevsno, jj1 = nlevsno + 1;
  double* const sm = sv_smem + k;
  double* const scal = sm + SV_ARRAYS * SV_ROWS * SV_COLS;
  double* const lu = scal + SS_COUNT * SV_COLS;                       // [n rows of 7][SV_COLS]
  uint8_t* const piv = reinterpret_cast<uint8_t*>(sv_smem + SV_COLS * (SV_ARRAYS * SV_ROWS + SS_COUNT + 7 * MAXROWS)) + k;
  auto at = [&](int a, int r) -> double& { return sm[(a * SV_ROWS + r) * SV_COLS]; };
  auto sc = [&](int a) -> double& { return scal[a * SV_COLS]; };
  const int64_t i = (int64_t)blockIdx.x * SV_COLS + k;
  int64_t c = 0;
  bool in = false;
  if (i < nc) {
    c = order ? (int64_t)order[i] : i;
    in = step_reversed_here(D, ft, fw, lg, c);
  }
  if (!__syncthreads_or(in)) return;
  const bool do_t = in && ft.mask_nolakec[c], do_w = in && fw.mask_hydrology[c];
  const double* const rec = lg.st + c * (int64_t)CLMGB_LOG_ST_STRIDE;
  const uint32_t s1 = do_t ? (uint32_t)rec[ST_STATUS] : 0u;
  const int n = do_t ? (int)rec[ST_N] : 0;
  const bool full = do_t && !(s1 & (CLMGB_COL_URBAN | CLMGB_COL_PATCH_RANGE | CLMGB_COL_LEVEL_RANGE)) && n > 0;
  StCol C;
  double forc = 0.0;
  if (in) {
    st_column(C, D, ft, c, dtime, snow_method, ft.t_grnd[c], ft.t_h2osfc[c]);
    forc = ft.forc_lwrad[c];
  }
  const bool on = in && jj >= C.jjtop && jj <= nw;
  // ---- the level's inputs, then the step's outputs from the log to the state ----
  double tin = 0.0, liq0 = 0.0, ice0 = 0.0, fact = 0.0;
  uint32_t st = 0;
  if (in && jj <= nw && j >= 1 && LV(ft.excess_ice, c, j, ld) != 0.0) st = CLMGB_COL_ADJ_UNSUPPORTED;
  if (on) {
    tin = LV(ft.t_soisno, c, jj, ld);
    liq0 = LV(ft.h2osoi_liq, c, jj, ld);
    ice0 = LV(ft.h2osoi_ice, c, jj, ld);
    fact = do_t ? rec[ST_FACT + jj - 1] : LV(ft.fact, c, jj, ld);
  }
  at(SV_T, jj) = tin;
  if (in && do_t && t_ssbef)
    if (jj <= nlev) LV(t_ssbef, c, jj, ld) = LV(ft.t_soisno, c, jj, ld);
  for (int r = jj - 1; full && r < n; r += SV_THREADS / SV_COLS) {
    for (int d = 0; d < 7; d++) lu[(r * 7 + d) * SV_COLS] = rec[ST_LU + r * 7 + d];
    piv[r * SV_COLS] = reinterpret_cast<const uint8_t*>(rec + ST_PIV)[r];
    at(SV_X, r) = rec[ST_X + r];
  }
  // (loads ahead of the barrier, stores behind it: the state's old values are read by then)
  double tout = 0.0, liq1 = liq0, ice1 = ice0, smp = 0.0, hk = 0.0;
  const bool solved = do_w && on && j >= 1 && j <= (int)C.nbedrock;
  if (do_t && jj >= C.jjtop && jj <= nlev) tout = rec[ST_T + jj - 1];
  if (on && do_t) {
    liq1 = rec[ST_LIQ + jj - 1];
    ice1 = rec[ST_ICE + jj - 1];
  }
  const double* const fin = lg.rec + c * lg.stride + (int64_t)lg.cap * SUB_REC;
  if (solved) {
    liq1 = fin[j - 1];
    smp = fin[MAXSOI + j - 1];
    hk = fin[2 * MAXSOI + j - 1];
  }
  __syncthreads();
  if (do_t && jj >= C.jjtop && jj <= nlev) LV(ft.t_soisno, c, jj, ld) = tout;
  if (on) {
    LV(ft.h2osoi_liq, c, jj, ld) = liq1;
    LV(ft.h2osoi_ice, c, jj, ld) = ice1;
    if (do_t) LV(ft.fact, c, jj, ld) = fact;
  }
  if (solved) {
    LV(fw.smp_l, c, j, ld) = smp;
    LV(fw.hk_l, c, j, ld) = hk;
  }
  if (do_w && j == 1) {
    fw.qcharge[c] = fin[3 * MAXSOI];
    fw.num_substeps[c] = fin[3 * MAXSOI + 1];
    st |= (uint32_t)fin[3 * MAXSOI + 2];
  }
  if (in && j == 1) {
    st |= s1;
    if (ft.frac_h2osfc[c] > 0.0 || ft.h2osno_no_layers[c] > 0.0) st |= CLMGB_COL_ADJ_UNSUPPORTED;
    if (do_t) {
      if (t_h2osfc_bef) t_h2osfc_bef[c] = C.th0;
      ft.t_grnd[c] = rec[ST_TG];
      ft.t_h2osfc[c] = rec[ST_TH];
    }
  }
  // ---- the column's status: its levels' together ----
  uint32_t* const bits = reinterpret_cast<uint32_t*>(&sc(SS_STATUS));
  if (j == 1) *bits = 0;
  __syncthreads();
  if (st) atomicOr(bits, st);
  __syncthreads();
  if (in && j == 1) {
    st = *bits;
    if (col_status) col_status[c] = st;
    if (st && dev_status) atomicOr(dev_status, st);
    if (!full && adj.lam_forc_lwrad) adj.lam_forc_lwrad[c] = 0.0;
  }
  if (!__syncthreads_or(full)) return;
  const bool act = on && full;
  const int rsw = full ? -(int)C.snl : 0;
  const int r = jj < jj1 ? jj - C.jjtop : rsw + j;
  // ---- the column's sums (on the thread of soil level 1), layer conductivity ----
  if (act && j == 1) {
    st_sums(C, D, ft, c, forc, at(SV_T, C.jjtop), tin);
    const double v[10] = {C.dhsdT, C.hs_soil, C.hs_h2osfc, C.hs_top, C.w_set, C.wb_set, C.w_act, C.wb_act, C.dtc, C.rdh};
#pragma unroll
    for (int q = 0; q < 10; q++) sc(q) = v[q];
  }
  StLayer ly = {0.0, 0.0, 0.0, 0.0};
  if (act) {
    ly = st_layer(C, D, ft, fw, c, jj, tin, liq0, ice0);
    at(SV_THK, jj) = ly.v;
  }
  __syncthreads();
  C.dhsdT = sc(SS_DHSDT);
  C.hs_soil = sc(SS_SOIL);
  C.hs_top = sc(SS_TOP);
  StItf it = {0.0, 0.0, 0.0, 0.0, 0.0};
  StPc pc = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  double tgb = 0.0, thb = 0.0, tn = 0.0;
  if (act) {
    tgb = adj.lam_t_grnd[c];
    thb = adj.lam_t_h2osfc[c];
    tn = jj < nw ? at(SV_T, jj + 1) : 0.0;
    it = st_interface(D, ft, c, jj, ly.v, jj < nw ? at(SV_THK, jj + 1) : 0.0, tin, tn);
    at(SV_TK, jj) = it.tk;
    at(SV_RDZ, jj) = it.rdz;
    at(SV_FN, jj) = it.fn;
    pc = st_phase_change(C, D, ft, fw, c, jj, at(SV_X, r), liq0, ice0, fact,
                         LV(adj.lam_t_soisno, c, jj, ld) + st_tgrnd_level(C, j, tgb), LV(adj.lam_h2osoi_liq, c, jj, ld),
                         LV(adj.lam_h2osoi_ice, c, jj, ld));
    double w = pc.t;
    const double thpc = thb + st_tgrnd_h2osfc(C, tgb);
    if (j == 1) {
      at(SV_W, rsw) = C.fh == 0.0 ? 0.0 : thpc;
      if (C.fh == 0.0) w += thpc;
      double tkh, dtkh;
      st_tkh(D, ft, c, ly.v, tkh, dtkh);
      sc(SS_TKH) = tkh;
      sc(SS_DTKH) = dtkh;
    }
    at(SV_W, r) = w;
    if (jj == C.jjtop) sc(SS_PC_TOP) = pc.dh;
    if (j == 1) sc(SS_PC_1) = C.snl < 0 ? pc.dh : 0.0;
  }
  __syncthreads();
  // ---- A^T lambda = w, band_lu_transpose_solve on a column per lane ----
  if (warp == 0 && lane < SV_COLS && full) {
    auto ab = [&](int row, int col) -> double { return lu[(row * 7 + col - row + 2) * SV_COLS]; };
    // U^T: a row's sum loses each product as soon as lambda is known, the next row's first
    double s0 = at(SV_W, 0), s1 = at(SV_W, 1), s2 = at(SV_W, 2), s3 = at(SV_W, 3);
    for (int p = 0; p < n; p++) {
      const double x = div_chain(s0, ab(p, p)), s4 = p + 4 < n ? at(SV_W, p + 4) : 0.0;
      at(SV_W, p) = x;
      s0 = p + 1 < n ? less_product(s1, ab(p, p + 1), x) : 0.0;
      s1 = p + 2 < n ? less_product(s2, ab(p, p + 2), x) : 0.0;
      s2 = p + 3 < n ? less_product(s3, ab(p, p + 3), x) : 0.0;
      s3 = p + 4 < n ? less_product(s4, ab(p, p + 4), x) : 0.0;
    }
    for (int p = n - 2; p >= 0; p--) {
      double s = at(SV_W, p);
      const int last = min(n - 1, p + 2);
      for (int q = p + 1; q <= last; q++) s = less_product(s, ab(q, p), at(SV_W, q));
      const int x = p + (int)piv[p * SV_COLS];
      at(SV_W, p) = s;
      if (x != p) {
        at(SV_W, p) = at(SV_W, x);
        at(SV_W, x) = s;
      }
    }
  }
  __syncthreads();
  // ---- the level's row ----
  auto entry = [&](int q, int d) -> double {
    return q - 2 + d >= 0 && q - 2 + d < n ? -at(SV_W, q) * at(SV_X, q - 2 + d) : 0.0;
  };
  StRow row = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  if (act) {
    const bool up = jj > C.jjtop;
    const StRowIn a = {j,   at(SV_W, r), entry(r, 0), entry(r, 1), entry(r, 2), entry(r, 3), entry(r, 4), fact,
                       tin, it.fn,       up ? at(SV_FN, jj - 1) : 0.0, it.tk, up ? at(SV_TK, jj - 1) : 0.0, it.rdz,
                       up ? at(SV_RDZ, jj - 1) : 0.0, j <= 1 ? st_sabg(D, ft, c, jj) : 0.0};
    row = st_row(C, nlevgrnd, a);
    at(SV_KP, jj) = row.kp;
    at(SV_NP, jj) = row.np;
    if (jj == C.jjtop) {
      sc(SS_ROW_TOP) = row.dh;
      sc(SS_HST) = row.hst;
    }
    if (j == 1) {
      sc(SS_ROW_1) = C.snl < 0 ? row.dh : 0.0;
      sc(SS_HSS) = row.hss;
    }
  }
  __syncthreads();
  // ---- the interfaces' adjoints ----
  double kb = 0.0, d = 0.0;
  if (act) {
    const double fnb = row.n + (jj < nw ? at(SV_NP, jj + 1) : 0.0);
    const double dT = jj < nw ? tn - tin : 0.0;
    kb = row.k + (jj < nw ? at(SV_KP, jj + 1) : 0.0) + fnb * dT * it.rdz;
    d = fnb * it.tk * it.rdz;
    at(SV_D, jj) = d;
    at(SV_KB, jj) = kb * it.db;
  }
  __syncthreads();
  // ---- the adjoints of the step's inputs ----
  if (!act) return;
  const bool up = jj > C.jjtop;
  double t = row.t + (up ? at(SV_D, jj - 1) : 0.0) - d, fb = pc.f + row.f;
  double hb = (up ? at(SV_KB, jj - 1) : 0.0) + kb * it.da;
  if (j == 1) {
    C.hs_h2osfc = sc(SS_H2OSFC);
    C.w_set = sc(SS_WSET);
    C.dtc = sc(SS_DTC);
    C.rdh = sc(SS_RDH);
    const StSurf sf = st_surface(C, sc(SS_TKH), tin, fact, at(SV_W, rsw), entry(rsw, 2), entry(rsw, 3),
                                 at(SV_W, rsw + 1), entry(rsw + 1, 1), entry(rsw + 1, 2));
    const double dh = st_dhsdT_bar(sc(SS_PC_TOP), sc(SS_PC_1), sc(SS_ROW_TOP), sc(SS_ROW_1), sf.dh);
    const double hst = sc(SS_HST), hss = sc(SS_HSS) + sf.hss;
    adj.lam_t_grnd[c] = dh * (-C.w_set) * (4.0 * C.eg * SB) * (3.0 * (C.tg0 * C.tg0));
    adj.lam_t_h2osfc[c] = sf.th + st_t4_bar(C, sf.hsh, C.w_set, C.th0);
    if (adj.lam_forc_lwrad) adj.lam_forc_lwrad[c] = 0.0 + ((hss + sf.hsh) * sc(SS_WBSET) + hst * sc(SS_WBACT));
    t += sf.t1 + st_t4_bar(C, hss, C.w_set, tin);
    fb += sf.f1;
    hb += sf.tkh * sc(SS_DTKH);
  }
  if (jj == C.jjtop) t += st_t4_bar(C, sc(SS_HST), sc(SS_WACT), tin);
  const StCap q = st_capacity(C, D, ft, fw, c, jj, liq0, ice0, fact);
  LV(adj.lam_t_soisno, c, jj, ld) = t;
  LV(adj.lam_h2osoi_liq, c, jj, ld) = pc.liq + fb * q.l + hb * ly.dl;
  LV(adj.lam_h2osoi_ice, c, jj, ld) = pc.ice + fb * q.i + hb * ly.di;
  if (j >= 1 && j <= D.nlevsoi) {
    if (adj.grad_watsat) LV(adj.grad_watsat, c, j, ld) += pc.ws + fb * q.w + hb * ly.dw;
    if (adj.grad_bsw) LV(adj.grad_bsw, c, j, ld) += pc.bs;
    if (adj.grad_sucsat) LV(adj.grad_sucsat, c, j, ld) += pc.suc;
  }
}

}  // namespace

cudaError_t launch_soil_reverse(const Dims& D, int64_t nc, const clmgb_soiltemp_fields& ft,
                                const clmgb_soilwater_fields& fw, double dtime, int snow_method, double* t_ssbef,
                                double* t_h2osfc_bef, const clmgb_step_adjoint& adj, const SubstepLogView& lg,
                                const uint32_t* order, uint32_t* col_status, uint32_t* dev_status, cudaStream_t s) {
  const cudaError_t e = allow_dynamic_smem(k_soil_reverse, SV_SMEM);
  if (e != cudaSuccess) return e;
  const unsigned grid = (unsigned)((nc + SV_COLS - 1) / SV_COLS);
  k_soil_reverse<<<grid, SV_THREADS, SV_SMEM, s>>>(D, nc, ft, fw, dtime, snow_method, t_ssbef, t_h2osfc_bef, adj,
                                                   lg, order, col_status, dev_status);
  return cudaGetLastError();
}

}  // namespace clmgb
