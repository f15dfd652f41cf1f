// soil_temperature_packed.cu — soil_temperature! (soil_temperature.jl:358-593), and for
// the column step set_soil_water_fractions! behind it, with a column's levels spread over
// threads.
//
// Every stage whose levels do not depend on one another (conductivities, heat capacities,
// fluxes, the band rows, phase change, the fractions) runs over (level, column) items; the
// ground heat flux, the banded solve and the column's sums run a thread per column.  Two
// forms:
//   * few columns: a warp owns ks = 1, 2 or 4 neighbouring columns and its lanes their
//     levels, column fastest, so that a column's chain is as short as its banded solve;
//   * many columns: a block owns 32 columns, a lane each in all its four warps, which
//     share the levels; one warp (another one in neighbouring blocks) runs the banded
//     solve for all 32.  The blocks of SORTED neighbouring columns share them by
//     snow-layer count, so that a warp's lanes have levels of about the same number.
// The 38-row system and what the stages hand on stay in shared memory, [array][row][slot].
//
// The banded elimination keeps its window of three rows in registers.  The systems are
// tridiagonal but for the couplings around the surface-water row, so most of the
// reference's operations subtract a zero: a step (or a row of the back substitution)
// whose zeros are zeros in all the warp's lanes leaves them out, 4 and 2 FP64
// instructions in place of 20 and 8.  The arithmetic is otherwise soil_temperature_col's
// and phase_change_beta_col's (clmgb_device.cuh), expression by expression; quotients that
// two levels share are formed once, products with 1/2 through the exponent, comparisons on
// the bits: the same values.
//
// On GB300 an FP64 instruction holds its sub-partition's FP64 unit for about 65 cycles
// whatever the lanes.  The kernel this one replaced ran a column per thread, 4,200 FP64
// instructions and some 200 divisions one after another over a 4 KB stack: 562 us for
// 61 columns and 700 for 1,000.  Measured per call (snow and frozen-soil columns, us),
// that kernel and this: 61 columns 562 -> 66, 1,000 708 -> 78, 4,000 710 -> 112, 16,000 750
// -> 187, 65,536 1,165 -> 640; 262,144 3,130 -> 2,690.  What bounds it: at few columns
// the chain of the banded solve (about 45 % of the time) and of the divisions; at many
// (ncu, 262,144 columns) latency at 16 warps per SM, the FP64 unit 46 % busy, a third of
// the warps' time at the block's barriers, most of it beside the banded solve, and a sixth
// waiting for instructions.  The loops over patches and over single values of a level are not
// unrolled for that reason (2.69 -> 2.62 ms).
#include "clmgb_device.cuh"
#include "launch.h"

namespace clmgb {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int TWARPS = 4, TBLOCK = 32 * TWARPS;
constexpr int WARP_FORM = 40;
constexpr int TROWS = MAXROWS;                 // snow levels, the surface-water row, ground levels

// -0, or a number so small that its upper word is -0's
__device__ __forceinline__ bool minus_zero(double x) { return (uint32_t)((unsigned long long)dbits(x) >> 32) == 0x80000000u; }

// a column's rows in shared memory, [array][row][slot]: row jj-1 of snow level jj, row
// nlevsno of the surface water, row jj of soil level jj.  RS, RD, RP hold A[r, r-1 .. r+1],
// RX the right-hand side; the two entries further out, row 1 of the soil to the lowest snow
// row and back, are the slot area's.  After the elimination RD, RP, RS hold U[r, r .. r+2]
// (U[r, r+3 .. r+4], which only a row exchange fills, go to the lane's own store).  Before
// the rows are assembled RX holds the temperatures and RS the layer conductivities; after
// the solve RS, RD, RP hold the levels' contributions to the column's phase-change sums.
// RK keeps the interface conductivities.
enum RowArray { RS = 0, RD, RP, RX, RK, R_ARRAYS };
template <int N>
struct SlotArea {
  // the column's scalars its other lanes read
  double dhsdT[N], hs_soil[N], hs_top[N], tk_h2osfc[N], fn_h2osfc[N], dz_h2osfc[N];
  double to_snow[N], to_soil[N];  // A[soil row 1, lowest snow row], A[lowest snow row, soil row 1]
  double fn1[N];                  // fn of soil level 1
  int bad_patches[N];
  unsigned long long melt[N];     // levels with a phase change
  int bad[N];                     // a temperature is not finite
  int reset[N];                   // unresolved snow melted on level 1: qsm starts the sums again
  double qsm[N];
};
// bytes of ks columns, the slot area of at most N columns behind their rows
template <int N>
__host__ __device__ constexpr int64_t group_bytes(int ks) {
  return (int64_t)R_ARRAYS * TROWS * ks * 8 + (int64_t)((sizeof(SlotArea<N>) + 15) / 16 * 16);
}

// The columns of a block in the BLOCK form: SORTED neighbouring columns are ordered by
// snow-layer count, so that the 32 lanes of a warp have levels of about the same number,
// and the SORTED / 32 blocks that share them take 32 each.  Every block forms the same
// order (by count, then by column).  All threads call it; -1 past the last column.
constexpr int SORTED = 256;
__device__ __forceinline__ int64_t sorted_column(int64_t nc, const int64_t* col_snl, int nlevsno) {
  __shared__ uint32_t key4[SORTED / 4];
  __shared__ uint8_t mine[32];
  uint8_t* key = reinterpret_cast<uint8_t*>(key4);
  const int64_t base = (int64_t)(blockIdx.x / (SORTED / 32)) * SORTED;
  const int first = (int)(blockIdx.x % (SORTED / 32)) * 32;
  for (int i = threadIdx.x; i < SORTED; i += TBLOCK) {
    int k = 255;
    if (base + i < nc) {
      const int64_t n = -col_snl[base + i];
      k = n < 0 || n > nlevsno ? 254 : (int)n;
    }
    key[i] = (uint8_t)k;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < SORTED; i += TBLOCK) {
    const uint32_t k4 = 0x01010101u * key[i];
    int rank = 0;
    for (int q = 0; q < SORTED / 4; q++) {
      const uint32_t v = key4[q];
      const uint32_t le = q < i / 4 ? __vcmpleu4(v, k4) : __vcmpltu4(v, k4);
      rank += __popc(le & 0x01010101u);
    }
    for (int q = i & ~3; q < i; q++) rank += key[q] == key[i];
    if (rank >= first && rank < first + 32) mine[rank - first] = (uint8_t)i;
  }
  __syncthreads();
  const int64_t c = base + mine[threadIdx.x & 31];
  return c < nc ? c : -1;
}

// FRAC: the first half of a column step (masks, t_ssbef, fractions); LOG: with the
// soil_temperature! record (StLog) of every column soil_temperature! runs on.
// BLOCK: a block owns 32 columns, a lane each, and its warps share the levels; else a warp
// owns ks = 1 << sh neighbouring columns and its lanes share their levels.
template <bool FRAC, bool LOG, bool BLOCK>
__global__ void __launch_bounds__(TBLOCK)
k_soil_temperature_packed(Dims D, int64_t nc, clmgb_soiltemp_fields f, clmgb_soilwater_fields fw, double dtime,
                          int snow_method, double* t_ssbef, double* t_h2osfc_bef, uint32_t* col_status,
                          uint32_t* dev_status, double* st_log, int sh) {
  extern __shared__ __align__(16) unsigned char smem_st[];
  constexpr int NS = BLOCK ? 32 : 4;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  // this thread's column slot and its place among the levels: levels lo, lo + nper, ...
  const int ks = BLOCK ? 32 : 1 << sh, s = lane & (ks - 1), lo = BLOCK ? wib : lane >> sh;
  const int nper = BLOCK ? TWARPS : 32 >> sh;
  auto sync = [&]() {
    if (BLOCK) __syncthreads();
    else __syncwarp();
  };
  double* const rows = reinterpret_cast<double*>(smem_st + (BLOCK ? 0 : wib * group_bytes<NS>(ks)));
  SlotArea<NS>& SA = *reinterpret_cast<SlotArea<NS>*>(rows + (int64_t)R_ARRAYS * TROWS * ks);
  const int64_t ld = D.ldc, ldp = D.ldp;
  int64_t c;
  if (BLOCK) {
    c = sorted_column(nc, f.col_snl, D.nlevsno);
  } else {
    const int64_t w = (int64_t)blockIdx.x * TWARPS + wib;
    if (w * ks >= nc) return;                             // the whole warp leaves together
    c = w * ks + s;
    if (c >= nc) c = -1;
  }
  const bool in = c >= 0;
  const int nlevsno = D.nlevsno, joff = nlevsno, nlevgrnd = D.nlevgrnd, nlev = nlevsno + D.nlevmax;
  const int nlevsoi = D.nlevsoi;
  auto R = [&](int a, int row) -> double& { return rows[(a * TROWS + row) * ks + s]; };
  auto row_of = [&](int jj) -> int { return jj <= nlevsno ? jj - 1 : jj; };
  const bool masked = in && f.mask_nolakec[c];
  uint32_t st = 0;
  double* const rec = LOG ? st_log + c * (int64_t)CLMGB_LOG_ST_STRIDE : nullptr;
  if (masked) {
    if (FRAC && t_ssbef)
#pragma unroll 1
      for (int jj = 1 + lo; jj <= nlev; jj += nper) LV(t_ssbef, c, jj, ld) = LV(f.t_soisno, c, jj, ld);
    if (FRAC && t_h2osfc_bef && lo == 0) t_h2osfc_bef[c] = f.t_h2osfc[c];
    if (LOG && lo == 0) rec[ST_N] = 0.0;
  }
  // ---- the column's scalars, the same in all its lanes ----
  bool on = masked;
  int64_t snl64 = 0, it = 0, lit = 0, nbedrock = 0;
  if (on) {
    snl64 = f.col_snl[c];
    if (snl64 > 0 || snl64 < -nlevsno) {
      st = CLMGB_COL_LEVEL_RANGE;
      on = false;
    }
  }
  const bool snl_ok = on;
  if (on) {
    const int64_t l = f.col_landunit[c] - 1;
    it = f.col_itype[c];
    lit = f.lun_itype[l];
    if (f.lun_urbpoi[l] || is_wallroof(it) || it == ICOL_ROAD_IMPERV || it == ICOL_ROAD_PERV) {
      st = CLMGB_COL_URBAN;
      on = false;
    }
  }
  const int snl = (int)snl64;
  const int jtop = snl + 1, jjtop = on ? jtop + joff : nlev + 1;
  // the first level of the warp's columns (the same columns in all warps of a block)
  const int jj0 = (int)__reduce_min_sync(FULL, (unsigned)jjtop);
  if (jj0 <= nlev) {
    const bool is_special = lit == ISTWET || lit == ISTICE, issoilcrop = lit == ISTSOIL || lit == ISTCROP;
    double fse = 0.0, fh = 0.0, no_layers = 0.0, h2osfc = 0.0, th = 0.0, ebot = 0.0;
    if (on) {
      nbedrock = f.col_nbedrock[c];
      fse = f.frac_sno_eff[c];
      fh = f.frac_h2osfc[c];
      no_layers = f.h2osno_no_layers[c];
      h2osfc = f.h2osfc[c];
      th = f.t_h2osfc[c];
      ebot = f.eflx_bot[c];
    }
    // ---- layer conductivity thk (_soil_snow_tk_kernel! :647-716) ----
    for (int base = jj0; base <= nlev; base += nper) {
      const int jj = base + lo, j = jj - nlevsno;
      if (!(on && jj >= jjtop && jj <= nlev)) continue;
      const double t0 = LV(f.t_soisno, c, jj, ld);
      R(RX, row_of(jj)) = t0;
      double thkv = 0.0;
      if (j >= 1) {
        if (!is_special) {
          if (j > nbedrock) {
            thkv = THK_BEDROCK;             // bedrock overrides the soil value (:684-686)
          } else {
            const double liq = LV(f.h2osoi_liq, c, jj, ld), ice = LV(f.h2osoi_ice, c, jj, ld);
            const double exi = LV(f.excess_ice, c, j, ld);
            const double dzv = LVc(f.dz, c, jj, ld), ws = LVc(f.watsat, c, j, ld);
            const double tkdry = LVc(f.tkdry, c, j, ld);
            double satw = jl_div(jl_div(liq, DENH2O) + jl_div(ice, DENICE) + jl_div(exi, DENICE), dzv * ws);
            satw = jl_min(1.0, satw);
            if (above(satw, 1.0e-7)) {
              double dke;
              if (at_least(t0, TFRZ)) dke = jl_max(0.0, cm_log10(satw) + 1.0);
              else dke = satw;
              const double a1 = jl_div(liq, DENH2O * dzv);
              const double fl_denom = a1 + jl_div(ice, DENICE * dzv) + jl_div(exi, DENICE * dzv);
              const double fl = jl_div(a1, fl_denom);
              const double dksat =
                  LVc(f.tkmg, c, j, ld) * cm_pow(TKWAT, fl * ws) * cm_pow(TKICE, (1.0 - fl) * ws);
              thkv = dke * dksat + (1.0 - dke) * tkdry;
            } else {
              thkv = tkdry;
            }
          }
        } else if (lit == ISTICE) {
          thkv = below(t0, TFRZ) ? TKICE : TKWAT;
        } else {  // ISTWET
          if (j > nlevsoi) thkv = THK_BEDROCK;
          else thkv = below(t0, TFRZ) ? TKICE : TKWAT;
        }
      } else {
        // snow layer (snl+1 <= j <= 0) — Jordan1991 or Sturm1997
        const double denom = jl_max(fse, 1.0e-6) * jl_max(LVc(f.dz, c, jj, ld), 1.0e-6);
        const double bwv = jl_div(LV(f.h2osoi_ice, c, jj, ld) + LV(f.h2osoi_liq, c, jj, ld), denom);
        LV(f.bw, c, jj, ld) = bwv;
        if (snow_method == CLMGB_SNOW_JORDAN1991) {
          thkv = TKAIR + (7.75e-5 * bwv + 1.105e-6 * (bwv * bwv)) * (TKICE - TKAIR);
        } else {
          const double q = jl_div(bwv, 1000.0);
          if (bwv <= 156.0) thkv = 0.023 + 0.234 * q;
          else thkv = 0.138 - 1.01 * q + 3.233 * (q * q);
        }
      }
      LV(f.thk, c, jj, ld) = thkv;
      R(RS, row_of(jj)) = thkv;
    }
    sync();
    // ---- column scalars: surface-water conductivity (:762-776), ground heat flux and its
    // derivative (:1200-1263), surface-water heat capacity (:116-130) and row ----
    if (on && lo == 0) {
      double dhsdT = 0.0, hs_soil = 0.0, hs_top = 0.0, tk_h2osfc = 0.0, fn_h2osfc = 0.0, dz_h2osfc = 0.0;
      int bad_patches = 0;
      const int r1 = nlevsno + 1;
      const double t1 = R(RX, r1), tk1 = R(RS, r1), z1 = LVc(f.z, c, 1 + joff, ld);
      {
        const double zh2osfc = 1.0e-3 * (0.5 * h2osfc);
        const double denom = TKWAT * z1 + tk1 * zh2osfc;
        if (pos(denom)) tk_h2osfc = jl_div(TKWAT * tk1 * (z1 + zh2osfc), denom);
        else tk_h2osfc = tk1;
      }
      const double eg = f.emg[c], tg = f.t_grnd[c], htvp = f.htvp[c], forc = f.forc_lwrad[c];
      const double tt = R(RX, row_of(jjtop));
      const double lw_emit = eg * SB * jl_pow4(tg);
      const double dlw_emit = 4.0 * eg * SB * (tg * tg * tg);
      const double lw_snow = eg * SB * jl_pow4(tt);
      const double lw_soil = eg * SB * jl_pow4(t1);
      const double lw_h2osfc = eg * SB * jl_pow4(th);
      const int64_t pi = f.col_patchi[c], pf = f.col_patchf[c];
      double hs_h2osfc = 0.0;
      if (pi < 1 || pf > D.np || pf < pi - 1) {
        bad_patches = 1;
      } else {
#pragma unroll 1
        for (int64_t p1 = pi; p1 <= pf; p1++) {
          const int64_t p = p1 - 1;
          if (f.patch_column[p] != c + 1 + D.c0) continue;
          double dh_p = 0.0, hsoil_p = 0.0, hh_p = 0.0;
          const bool act = f.mask_nolakep[p] != 0;
          const double base = f.dlrad[p] + (1.0 - (double)f.frac_veg_nosno[p]) * eg * forc;
          if (act && !f.lun_urbpoi[f.patch_landunit[p] - 1]) {
            const double gnet = f.sabg[p] + base - lw_emit - (f.eflx_sh_grnd[p] + f.qflx_evap_soi[p] * htvp);
            f.eflx_gnet[p] = gnet;
            f.sabg_chk[p] = fse * f.sabg_snow[p] + (1.0 - fse) * f.sabg_soil[p];
            const double dg = -f.cgrnd[p] - dlw_emit;
            f.dgnetdT[p] = dg;
            const double wt = f.patch_wtcol[p];
            const double gsoil = f.sabg_soil[p] + base - lw_soil - (f.eflx_sh_soil[p] + f.qflx_ev_soil[p] * htvp);
            const double gh2o = f.sabg_soil[p] + base - lw_h2osfc - (f.eflx_sh_h2osfc[p] + f.qflx_ev_h2osfc[p] * htvp);
            if (wt != 0.0) {
              dh_p = dg * wt;
              hsoil_p = gsoil * wt;
              hh_p = gh2o * wt;
            }
          }
          dhsdT += dh_p;
          hs_soil += hsoil_p;
          hs_h2osfc += hh_p;
          if (act) {   // SNICAR top-layer flux (:1139-1167)
            const double sab = LVc(f.sabg_lyr, p, jjtop, ldp);
            const double gsnow = sab + base - lw_snow - (f.eflx_sh_snow[p] + f.qflx_ev_snow[p] * htvp);
            hs_top += gsnow * f.patch_wtcol[p];
          }
        }
        double ch;
        if (h2osfc > THIN_SFCLAYER && fh > THIN_SFCLAYER) {
          ch = jl_max(THIN_SFCLAYER, jl_div(CPLIQ * h2osfc, fh));
          dz_h2osfc = jl_max(THIN_SFCLAYER, jl_div(1.0e-3 * h2osfc, fh));
        } else {
          ch = THIN_SFCLAYER;
          dz_h2osfc = THIN_SFCLAYER;
        }
        f.c_h2osfc[c] = ch;
        // the surface-water row
        const double dzm = 0.5 * dz_h2osfc + z1;
        fn_h2osfc = jl_div(tk_h2osfc * (t1 - th), dzm);
        const double dc = jl_div(dtime, ch);
        const double g = jl_div(half_of(dc) * tk_h2osfc, dzm);
        R(RX, nlevsno) = th + dc * (hs_h2osfc - dhsdT * th + half_of(fn_h2osfc));
        R(RS, nlevsno) = 0.0;
        R(RD, nlevsno) = 1.0 + g - dc * dhsdT;
        R(RP, nlevsno) = -g;
      }
      SA.dhsdT[s] = dhsdT;
      SA.hs_soil[s] = hs_soil;
      SA.hs_top[s] = hs_top;
      SA.tk_h2osfc[s] = tk_h2osfc;
      SA.fn_h2osfc[s] = fn_h2osfc;
      SA.dz_h2osfc[s] = dz_h2osfc;
      SA.bad_patches[s] = bad_patches;
    }
    sync();
    const double dhsdT = on ? SA.dhsdT[s] : 0.0;
    const bool bad_patches = on && SA.bad_patches[s];
    // ---- interface conductivity (:599-629), heat capacity and fact, fn (:1271-1319), the
    // rows of set_rhs_vec! and set_matrix! (:1365-1748).  A row takes the conductivity, the
    // flux and their quotient of the level above: in the BLOCK form a thread runs down a
    // stretch of levels and keeps them (the first level's are formed twice), else they
    // come from that level's lane ----
    {
      double tk = 0.0, fn = 0.0, q1 = 0.0, t0 = 0.0, z0 = 0.0, dzp = 0.0, z1 = 0.0;
      // the conductivity, flux and quotient between level jj and the next, whose layer
      // conductivity and temperature are k1 and t1
      auto interface = [&](int jj, double k1, double t1) {
        const int j = jj - nlevsno, r = row_of(jj);
        t0 = R(RX, r);
        z0 = LVc(f.z, c, jj, ld);
        tk = q1 = dzp = 0.0;
        if (j <= nlevgrnd - 1) {
          const double k0 = R(RS, r);
          z1 = LVc(f.z, c, jj + 1, ld);
          const double zi1 = LVc(f.zi, c, jj + 1, ld);
          dzp = z1 - z0;
          tk = jl_div(k0 * k1 * dzp, k0 * (z1 - zi1) + k1 * (zi1 - z0));
          fn = jl_div(tk * (t1 - t0), dzp);
          q1 = jl_div(tk, dzp);
        } else {
          fn = ebot;
        }
      };
      const int stretch = BLOCK ? (nlev - jj0 + TWARPS) / TWARPS : 1;
      const int begin = BLOCK ? jj0 + wib * stretch : jj0;
      const int end = BLOCK ? min(begin + stretch - 1, nlev) : nlev;
      double tk_n = 0.0, fn_n = 0.0, q1_n = 0.0;               // BLOCK: of the level above the stretch
      if (BLOCK && on && begin <= end && begin > jjtop) {
        interface(begin - 1, R(RS, row_of(begin)), R(RX, row_of(begin)));
        tk_n = tk;
        fn_n = fn;
        q1_n = q1;
      }
      // the last level of a stretch reads the conductivity and the temperature below it,
      // where the next stretch's thread is about to leave its row
      double k_below = 0.0, t_below = 0.0;
      if (BLOCK && on && end < nlev && begin <= end) {
        k_below = R(RS, row_of(end + 1));
        t_below = R(RX, row_of(end + 1));
      }
      if (BLOCK) __syncthreads();
      for (int base = begin; base <= end; base += BLOCK ? 1 : nper) {
        const int jj = BLOCK ? base : base + lo, j = jj - nlevsno;
        const bool ok = on && jj >= jjtop && jj <= nlev;
        const double tk_o = tk, fn_o = fn, q1_o = q1;          // the iteration before
        double fc = 0.0;
        tk = fn = q1 = 0.0;
        if (ok) {
          const bool edge = BLOCK && jj == end;
          const int rn = jj < nlev ? row_of(jj + 1) : row_of(jj);
          interface(jj, edge ? k_below : R(RS, rn), edge ? t_below : R(RX, rn));
          const double dzv = LVc(f.dz, c, jj, ld);
          const double liq = LV(f.h2osoi_liq, c, jj, ld), ice = LV(f.h2osoi_ice, c, jj, ld);
          double cv;
          if (j >= 1) {
            if (!is_special) {
              cv = LVc(f.csol, c, j, ld) * (1.0 - LVc(f.watsat, c, j, ld)) * dzv + (ice * CPICE + liq * CPLIQ) +
                   LV(f.excess_ice, c, j, ld) * CPICE;
            } else {
              cv = ice * CPICE + liq * CPLIQ;
            }
            if (j > nbedrock) cv = CSOL_BEDROCK * dzv;
            if (j == 1 && pos(no_layers)) cv += CPICE * no_layers;
          } else {
            if (pos(fse)) cv = jl_max(THIN_SFCLAYER, jl_div(CPLIQ * liq + CPICE * ice, fse));
            else cv = THIN_SFCLAYER;
          }
          fc = jl_div(dtime, cv);
          if (j == jtop) {
            const double zi0 = LVc(f.zi, c, jj, ld);
            fc = jl_div(fc * dzv, 0.5 * (z0 - zi0 + CAPR * (z1 - zi0)));
          }
          LV(f.fact, c, jj, ld) = fc;
        }
        double tkm, fnm, q2;
        if (BLOCK) {
          tkm = base == begin ? tk_n : tk_o;
          fnm = base == begin ? fn_n : fn_o;
          q2 = base == begin ? q1_n : q1_o;
        } else {
          const int src = (lane - ks) & 31;                    // the lane of the level above
          const bool wrap = lane < ks;
          const double tk_s = __shfl_sync(FULL, tk, src), tk_w = __shfl_sync(FULL, tk_o, src);
          const double fn_s = __shfl_sync(FULL, fn, src), fn_w = __shfl_sync(FULL, fn_o, src);
          const double q1_s = __shfl_sync(FULL, q1, src), q1_w = __shfl_sync(FULL, q1_o, src);
          tkm = wrap ? tk_w : tk_s;
          fnm = wrap ? fn_w : fn_s;
          q2 = wrap ? q1_w : q1_s;
          __syncwarp();        // the rows these levels read are read
        }
        if (ok) {
          const double h = half_of(fc);
          double x, b0 = 0.0, b1 = 0.0, b2, b3 = 0.0, b4 = 0.0;
          const double g = j <= nlevgrnd - 1 ? jl_div(h * tk, dzp) : 0.0;
          double dzm = 0.0, sab = 0.0;
          if (j > jtop) {
            dzm = z0 - LVc(f.z, c, jj - 1, ld);
            if (j <= 1 && !bad_patches) {   // absorbed solar of the level (:1139-1167)
#pragma unroll 1
              for (int64_t p1 = f.col_patchi[c]; p1 <= f.col_patchf[c]; p1++) {
                const int64_t p = p1 - 1;
                if (f.patch_column[p] != c + 1 + D.c0) continue;
                if (f.mask_nolakep[p] != 0) sab += LVc(f.sabg_lyr, p, jj, ldp) * f.patch_wtcol[p];
              }
            }
          }
          if (j == jtop) {
            x = t0 + fc * (SA.hs_top[s] - dhsdT * t0 + half_of(fn));
            b2 = 1.0 + g - fc * dhsdT;
            b3 = -g;
          } else if (j == 1) {
            x = t0 + fc * ((1.0 - fse) * (SA.hs_soil[s] - dhsdT * t0) + half_of(fn - fse * fnm));
            x += fse * fc * sab;
            b3 = -g;
            b2 = 1.0 + h * (q1 + jl_div(fse * tkm, dzm)) - (1.0 - fse) * fc * dhsdT;
            b0 = -jl_div(half_of(fse) * fc * tkm, dzm);
          } else if (j <= nlevgrnd - 1) {
            x = t0 + h * (fn - fnm);
            if (j <= 0) x += fc * sab;
            b3 = -g;
            b2 = 1.0 + h * (q1 + q2);
            b1 = -jl_div(h * tkm, dzm);
          } else {
            x = t0 - h * fnm + fc * fn;
            const double gm = jl_div(h * tkm, dzm);
            b2 = 1.0 + gm;
            b1 = -gm;
          }
          if (j == 0) {       // the snow-soil coupling skips the surface-water row
            b4 = b3;
            b3 = 0.0;
          }
          if (j == 1 && !zero_bits(fh)) {   // surface-water corrections (:1480-1494, :1689-1707)
            x -= fh * fc * ((SA.hs_soil[s] - dhsdT * t0) + half_of(SA.fn_h2osfc[s]));
            const double dzs = 0.5 * SA.dz_h2osfc[s] + z0;
            b2 += fh * (jl_div(h * SA.tk_h2osfc[s], dzs) + fc * dhsdT);
            b1 = -jl_div(half_of(fh) * fc * SA.tk_h2osfc[s], dzs);
          }
          const int r = row_of(jj);     // this level's T and conductivity are read by no later level
          if (j == 0) SA.to_soil[s] = b4;
          if (j == 1) SA.to_snow[s] = b0;
          R(RS, r) = b1;
          R(RD, r) = b2;
          R(RP, r) = b3;
          R(RX, r) = x;
          R(RK, r) = tk;
          // fn waits for the new temperatures where eflx_fgr goes
          if (j == 1) SA.fn1[s] = fn;
          if (j >= 1 && issoilcrop && !bad_patches) LV(f.eflx_fgr, c, j, ld) = fn;
        }
      }
    }
    sync();
    if (bad_patches) {
      if (lo == 0) st = CLMGB_COL_PATCH_RANGE;
      on = false;
    }
    // ---- batched_band_solve! (band_diagonal.jl:87-170): pivoted elimination, a lane per
    // column (in the BLOCK form by one warp, another one in neighbouring blocks) ----
    const int last = nlevsno + nlevgrnd;                               // the systems' last row
    const int first = on ? nlevsno + snl : last + 1;                   // this column's first
    if (BLOCK ? wib == (int)(blockIdx.x & (TWARPS - 1)) : true) {
      const bool mine = on && (BLOCK || lo == 0);
      const int begin = (int)__reduce_min_sync(FULL, (unsigned)first);
      if (LOG && mine) {
        rec[ST_N] = (double)(last - first + 1);
        rec[ST_LU] = rec[ST_LU + 1] = rec[ST_LU + 7] = 0.0;
      }
      // the window: rows k, k+1, k+2 over columns k..k+4, and their right-hand sides
      double w0[5] = {0.0, 0.0, 0.0, 0.0, 0.0}, w1[5] = {0.0, 0.0, 0.0, 0.0, 0.0}, w2[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
      double x0 = 0.0, x1 = 0.0, x2 = 0.0;
      double far3[TROWS], far4[TROWS];                                 // U[r, r+3], U[r, r+4] of the rows in `wide`
      unsigned long long wide = 0ULL;
      auto outer_lo = [&](int r) -> double { return r == nlevsno + 1 ? SA.to_snow[s] : 0.0; };
      auto outer_hi = [&](int r) -> double { return r == nlevsno - 1 ? SA.to_soil[s] : 0.0; };
      for (int k = begin; k <= last; k++) {
        const bool act = mine && k >= first;
        const bool have1 = act && k + 1 <= last, have2 = act && k + 2 <= last;
        if (act && k == first) {                                       // at least three rows
          w0[0] = R(RD, k);
          w0[1] = R(RP, k);
          w0[2] = outer_hi(k);
          x0 = R(RX, k);
          w1[0] = R(RS, k + 1);
          w1[1] = R(RD, k + 1);
          w1[2] = R(RP, k + 1);
          w1[3] = outer_hi(k + 1);
          x1 = R(RX, k + 1);
          w2[0] = outer_lo(k + 2);
          w2[1] = R(RS, k + 2);
          w2[2] = R(RD, k + 2);
          w2[3] = R(RP, k + 2);
          w2[4] = outer_hi(k + 2);
          x2 = R(RX, k + 2);
        }
        // the row that enters below
        double n0 = 0.0, n1 = 0.0, n2 = 0.0, n3 = 0.0, n4 = 0.0, nx = 0.0;
        if (act && k + 3 <= last) {
          n0 = outer_lo(k + 3);
          n1 = R(RS, k + 3);
          n2 = R(RD, k + 3);
          n3 = R(RP, k + 3);
          n4 = outer_hi(k + 3);
          nx = R(RX, k + 3);
        }
        // The systems are tridiagonal but for the couplings around the surface-water row.
        // A step without a row exchange whose pivot row ends at column k+1 and whose
        // second row below has no entry in column k changes the row below alone, in the
        // diagonal and the right-hand side: every other entry has a zero subtracted.
        // (Entries of -0, whose sign that would change, and non-finite pivot rows take
        // the general step.)
        const bool plain =
            !act || (have2 && !abs_gt(w1[0], w0[0]) && finite_nonzero(w0[0]) && finite_bits(w0[1]) && finite_bits(x0) &&
                     (dbits(w0[2]) | dbits(w0[3]) | dbits(w0[4]) | dbits(w2[0])) == 0 && !minus_zero(w1[2]) &&
                     !minus_zero(w1[3]) && !minus_zero(w1[4]) && !minus_zero(w2[1]) && !minus_zero(w2[2]) &&
                     !minus_zero(w2[3]) && !minus_zero(w2[4]) && !minus_zero(x2));
        if (__all_sync(FULL, plain)) {
          if (act) {
            const double f1 = div_chain(w1[0], w0[0]);
            w1[1] = w1[1] - f1 * w0[1];
            x1 = x1 - f1 * x0;
            R(RD, k) = w0[0];
            R(RP, k) = w0[1];
            R(RS, k) = 0.0;
            R(RX, k) = x0;
            if (LOG) {
              double* u = rec + ST_LU + (k - first) * 7 + 2;
              u[0] = w0[0];
              u[1] = w0[1];
              u[2] = u[3] = u[4] = 0.0;
              reinterpret_cast<uint8_t*>(rec + ST_PIV)[k - first] = 0;
              rec[ST_LU + (k - first + 1) * 7 + 1] = f1;
              rec[ST_LU + (k - first + 2) * 7] = zero_quotient(w2[0], w0[0]);
            }
          }
        } else if (act) {
          int piv = 0;
          double m = w0[0];
          if (have1 && abs_gt(w1[0], m)) {
            m = w1[0];
            piv = 1;
          }
          if (have2 && abs_gt(w2[0], m)) piv = 2;
#pragma unroll
          for (int i = 0; i < 5; i++) {
            const double t = w0[i];
            w0[i] = piv == 1 ? w1[i] : piv == 2 ? w2[i] : t;
            w1[i] = piv == 1 ? t : w1[i];
            w2[i] = piv == 2 ? t : w2[i];
          }
          const double t = x0;
          x0 = piv == 1 ? x1 : piv == 2 ? x2 : t;
          x1 = piv == 1 ? t : x1;
          x2 = piv == 2 ? t : x2;
          double f1 = 0.0, f2 = 0.0;
          if (have1) {
            f1 = jl_div(w1[0], w0[0]);
#pragma unroll
            for (int i = 1; i < 5; i++) w1[i] = w1[i] - f1 * w0[i];
            x1 = x1 - f1 * x0;
          }
          if (have2) {
            f2 = jl_div(w2[0], w0[0]);
#pragma unroll
            for (int i = 1; i < 5; i++) w2[i] = w2[i] - f2 * w0[i];
            x2 = x2 - f2 * x0;
          }
          R(RD, k) = w0[0];
          R(RP, k) = w0[1];
          R(RS, k) = w0[2];
          R(RX, k) = x0;
          if ((dbits(w0[3]) | dbits(w0[4])) != 0) {
            far3[k] = w0[3];
            far4[k] = w0[4];
            wide |= 1ULL << k;
          }
          if (LOG) {
            double* u = rec + ST_LU + (k - first) * 7 + 2;
#pragma unroll
            for (int i = 0; i < 5; i++) u[i] = w0[i];
            reinterpret_cast<uint8_t*>(rec + ST_PIV)[k - first] = (uint8_t)piv;
            if (have1) rec[ST_LU + (k - first + 1) * 7 + 1] = f1;
            if (have2) rec[ST_LU + (k - first + 2) * 7] = f2;
          }
        }
        if (act) {
          // slide down a row and right a column
#pragma unroll
          for (int i = 0; i < 4; i++) {
            w0[i] = w1[i + 1];
            w1[i] = w2[i + 1];
          }
          w0[4] = w1[4] = 0.0;
          w2[0] = n0;
          w2[1] = n1;
          w2[2] = n2;
          w2[3] = n3;
          w2[4] = n4;
          x0 = x1;
          x1 = x2;
          x2 = nx;
        }
      }
      // ---- back substitution; a zero U[i, i+2] .. U[i, i+4] with finite x leaves the sum
      // as it is, unless that is -0 ----
      double y1 = 0.0, y2 = 0.0, y3 = 0.0, y4 = 0.0;                   // x of the rows below
      for (int i = last; i >= begin; i--) {
        const bool act = mine && i >= first;
        double sx = 0.0, u0 = 1.0, u1 = 0.0, u2 = 0.0;
        if (act) {
          sx = R(RX, i);
          u0 = R(RD, i);
          u1 = R(RP, i);
          u2 = R(RS, i);
          if (i + 1 <= last) sx = sx - u1 * y1;
        }
        const bool more = act && (!zero_bits(u2) || ((wide >> i) & 1ULL) || !finite_bits(y2) || !finite_bits(y3) ||
                                  !finite_bits(y4) || minus_zero(sx));
        if (more) {
          const bool w = (wide >> i) & 1ULL;
          if (i + 2 <= last) sx = sx - u2 * y2;
          if (i + 3 <= last) sx = sx - (w ? far3[i] : 0.0) * y3;
          if (i + 4 <= last) sx = sx - (w ? far4[i] : 0.0) * y4;
        }
        if (act) {
          const double x = div_chain(sx, u0);
          y4 = y3;
          y3 = y2;
          y2 = y1;
          y1 = x;
          R(RX, i) = x;
          if (LOG) rec[ST_X + i - first] = x;
        }
      }
    }
    sync();
    // ---- the new temperatures (:149-167), fn1 and eflx_fgr (:170-206, :250-269) ----
    for (int base = jj0; base <= nlev; base += nper) {
      const int jj = base + lo, j = jj - nlevsno;
      const bool ok = on && jj >= jjtop && jj <= nlev;
      double tn = 0.0;
      if (ok) {
        const int r = row_of(jj);
        tn = R(RX, r);
        if (j == 1 || (j > 1 && issoilcrop)) {
          double v = 0.0;
          if (j <= nlevgrnd - 1) {
            const double fn = j == 1 ? SA.fn1[s] : LV(f.eflx_fgr, c, j, ld);
            const double fn1 = jl_div(R(RK, r) * (R(RX, r + 1) - tn), LVc(f.z, c, jj + 1, ld) - LVc(f.z, c, jj, ld));
            v = -half_of(fn) - half_of(fn1);
            if (j == 1) f.eflx_fgr12[c] = v;
          }
          if (issoilcrop) LV(f.eflx_fgr, c, j, ld) = v;
        }
        LV(f.t_soisno, c, jj, ld) = tn;
      }
    }
    // the zeros phase_change_beta! starts the snow levels with, inactive ones included
    if (on)
#pragma unroll 1
      for (int jj = 1 + lo; jj <= nlevsno; jj += nper) {
        LV(f.qflx_snomelt_lyr, c, jj, ld) = 0.0;
        LV(f.qflx_snofrz_lyr, c, jj, ld) = 0.0;
      }
    if (lo == 0) {
      SA.melt[s] = 0ULL;
      SA.bad[s] = 0;
      SA.reset[s] = 0;
    }
    sync();
    if (on && lo == 0) {
      const double tnew = zero_bits(fh) ? R(RX, nlevsno + 1) : R(RX, nlevsno);
      f.t_h2osfc[c] = tnew;
      phase_change_h2osfc_col(D, f, c, dtime, dhsdT);
      if (snl < 0) R(RX, nlevsno - 1) = LV(f.t_soisno, c, joff, ld);   // it may have changed the lowest snow level
    }
    sync();
    // ---- phase_change_beta! (:1929-2230) ----
    if (on) no_layers = f.h2osno_no_layers[c];
    sync();
    const bool supercool_type = lit == ISTSOIL || lit == ISTCROP || it == ICOL_ROAD_PERV;
    for (int base = jj0; base <= nlev; base += nper) {
      const int jj = base + lo, j = jj - nlevsno;
      if (!(on && jj >= jjtop && jj <= nlev)) continue;
      const int r = row_of(jj);
      const double t_in = R(RX, r);
      const double wice0 = LV(f.h2osoi_ice, c, jj, ld), wliq0 = LV(f.h2osoi_liq, c, jj, ld);
      double exi = j >= 1 ? LV(f.excess_ice, c, j, ld) : 0.0;
      const double wexice0 = exi;
      double exsubs = 0.0, tt = t_in, tinc = 0.0, sc = 0.0;
      int im = 0;
      // melt / freeze decision
      auto take = [&](int kind) {
        im = kind;
        tinc = TFRZ - tt;
        tt = TFRZ;
      };
      if (pos(wice0) && above(tt, TFRZ)) take(1);
      if (j <= 0) {
        if (pos(wliq0) && below(tt, TFRZ)) take(2);
      } else {
        if (pos(exi) && above(tt, TFRZ)) take(1);
        if (supercool_type && below(tt, TFRZ)) {
          const double smp = jl_div(HFUS * (TFRZ - tt), GRAV * tt) * 1000.0;
          double scv = LVc(f.watsat, c, j, ld) * cm_pow(jl_div(smp, LVc(f.sucsat, c, j, ld)),
                                                        jl_div(-1.0, LVc(f.bsw, c, j, ld)));
          scv *= LVc(f.dz, c, jj, ld) * 1000.0;
          sc = scv;
        }
        if (wliq0 > sc && below(tt, TFRZ)) take(2);
        if (j == 1 && pos(no_layers) && above(tt, TFRZ)) take(1);
      }
      if (im > 0) {
        const double wmass0 = wice0 + wliq0 + wexice0;
        const double fct = LV(f.fact, c, jj, ld);
        double hm, xm;
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
        if (im == 1 && negv(hm)) { hm = 0.0; im = 0; }
        if (im == 2 && pos(hm)) { hm = 0.0; im = 0; }
        if (im > 0 && (pos(hm) || negv(hm))) {
          xm = jl_div(hm * dtime, HFUS);
          if (j == 1 && pos(no_layers) && pos(xm)) {
            const double temp1 = no_layers;
            const double h2n = jl_max(0.0, temp1 - xm);
            f.h2osno_no_layers[c] = h2n;
            const double propor = jl_div(h2n, temp1);
            f.snow_depth[c] = propor * f.snow_depth[c];
            const double heatr0 = hm - jl_div(HFUS * (temp1 - h2n), dtime);
            if (pos(heatr0)) {
              xm = jl_div(heatr0 * dtime, HFUS);
              hm = heatr0;
            } else {
              xm = 0.0;
              hm = 0.0;
            }
            SA.qsm[s] = jl_div(jl_max(0.0, temp1 - h2n), dtime);
            SA.reset[s] = 1;
          }
          double heatr = 0.0, ice = wice0;
          if (pos(xm)) {
            ice = jl_max(0.0, wice0 - xm);
            heatr = hm - jl_div(HFUS * (wice0 - ice), dtime);
            const double xm2 = xm - ice;
            if (zero_bits(ice) && wexice0 >= 0.0 && pos(xm2) && j >= 2) {
              exi = jl_max(0.0, wexice0 - xm2);
              LV(f.excess_ice, c, j, ld) = exi;
              heatr = hm - jl_div(HFUS * (wexice0 - exi + wice0 - ice), dtime);
            }
          } else if (negv(xm)) {
            if (j <= 0) {
              ice = jl_min(wmass0, wice0 - xm);
            } else {
              if (wmass0 - wexice0 < sc) ice = 0.0;
              else ice = jl_min(wmass0 - wexice0 - sc, wice0 - xm);
            }
            heatr = hm - jl_div(HFUS * (wice0 - ice), dtime);
          }
          LV(f.h2osoi_ice, c, jj, ld) = ice;
          const double liq = jl_max(0.0, wmass0 - ice - exi);
          LV(f.h2osoi_liq, c, jj, ld) = liq;
          if (pos(heatr) || negv(heatr)) {
            if (j == jtop) {
              if (j == 1) tt += jl_div(fct * heatr, 1.0 - (1.0 - fh) * fct * dhsdT);
              else if (pos(fse)) tt += jl_div(jl_div(fct, fse) * heatr, 1.0 - fct * dhsdT);
            } else if (j == 1) {
              tt += jl_div(fct * heatr, 1.0 - (1.0 - fse - fh) * fct * dhsdT);
            } else {
              if (j > 0) tt += fct * heatr;
              else if (pos(fse)) tt += jl_div(fct, fse) * heatr;
            }
            if (j <= 0 && liq * ice > 0.0) tt = TFRZ;
          }
          double xmf = jl_div(HFUS * (wice0 - ice), dtime);
          if (j >= 1) {
            xmf = xmf + jl_div(HFUS * (wexice0 - exi), dtime);
            exsubs = jl_max(0.0, jl_div(wexice0 - exi, DENICE));
          }
          double qm = 0.0, qf = 0.0;
          if (j < 1) {
            if (im == 1) {
              qm = jl_div(jl_max(0.0, wice0 - ice), dtime);
              LV(f.qflx_snomelt_lyr, c, jj, ld) = qm;
            } else {
              qf = jl_div(jl_max(0.0, ice - wice0), dtime);
              LV(f.qflx_snofrz_lyr, c, jj, ld) = qf;
            }
          }
          R(RS, r) = xmf;
          R(RD, r) = qm;
          R(RP, r) = qf;
          atomicOr(&SA.melt[s], 1ULL << r);
        }
        R(RX, r) = tt;
        LV(f.t_soisno, c, jj, ld) = tt;
      }
      LV(f.imelt, c, jj, ld) = im;
      if (j >= 1) LV(f.exice_subs, c, j, ld) = exsubs;
      if (!finite_bits(tt)) SA.bad[s] = 1;
    }
    sync();
    // ---- the column's sums in ascending level order, t_grnd (:224-247) ----
    if (on && lo == 0) {
      double xmf = 0.0, qm = 0.0, qf = 0.0, drain = 0.0, accum = f.snomelt_accum[c];
      unsigned long long m = SA.melt[s];
      while (m) {
        const int r = __ffsll((long long)m) - 1;
        m &= m - 1;
        if (r == nlevsno + 1 && SA.reset[s]) {
          qm = SA.qsm[s];
          xmf = HFUS * qm;
          drain = qm;
        }
        xmf += R(RS, r);
        if (r < nlevsno) {
          const double q = R(RD, r);
          if (LV(f.imelt, c, r + 1, ld) == 1) {
            qm += q;
            accum += q * dtime * 1.0e-3;
          } else {
            qf += R(RP, r);
          }
        }
      }
      f.snomelt_accum[c] = accum;
      f.xmf[c] = xmf;
      f.qflx_snomelt[c] = qm;
      f.qflx_snofrz[c] = qf;
      f.qflx_snow_drain[c] = drain;
      const double melt = qm * HFUS;
      f.eflx_snomelt[c] = melt;
      if (issoilcrop) f.eflx_snomelt_r[c] = melt;
      const double t1 = R(RX, nlevsno + 1), thn = f.t_h2osfc[c];
      double tgn;
      if (snl < 0) {
        const double ts = R(RX, row_of(jjtop));
        if (!zero_bits(fh)) tgn = fse * ts + (1.0 - fse - fh) * t1 + fh * thn;
        else tgn = fse * ts + (1.0 - fse) * t1;
      } else {
        if (!zero_bits(fh)) tgn = (1.0 - fh) * t1 + fh * thn;
        else tgn = t1;
      }
      f.t_grnd[c] = tgn;
      if (SA.bad[s]) st |= CLMGB_COL_NONFINITE;
    }
  }
  sync();
  if (LOG && masked) {
    if (lo == 0) {
      rec[ST_STATUS] = (double)st;
      rec[ST_TG] = f.t_grnd[c];
      rec[ST_TH] = f.t_h2osfc[c];
    }
    if (snl_ok) {                                  // the levels the call may have changed
#pragma unroll 1
      for (int jj = jtop + joff + lo; jj <= nlev; jj += nper) {
        rec[ST_T + jj - 1] = LV(f.t_soisno, c, jj, ld);
        rec[ST_LIQ + jj - 1] = LV(f.h2osoi_liq, c, jj, ld);
        rec[ST_ICE + jj - 1] = LV(f.h2osoi_ice, c, jj, ld);
        rec[ST_FACT + jj - 1] = LV(f.fact, c, jj, ld);
      }
    }
  }
  // ---- set_soil_water_fractions! (soil_hydrology.jl:110-130) ----
  if (FRAC && in && fw.mask_hydrology[c])
#pragma unroll 1
    for (int j = 1 + lo; j <= nlevsoi; j += nper) water_fractions_level(D, fw, c, j);
  if (in && lo == 0) {
    if (col_status) col_status[c] = st;
    if (st && dev_status) atomicOr(dev_status, st);
  }
}

// Columns per SM up to which the warp form runs: at 4,000 columns (26 per SM) it took 112
// us against 139 of the block form, at 8,000 (53) 159 against 150.  Within it, columns
// per warp: as few as 12 warps per SM allow (shared memory and registers hold 16 to 20).
int64_t warp_form_limit(int nsm) { return (int64_t)nsm * WARP_FORM; }

template <bool FRAC, bool LOG, bool BLOCK>
cudaError_t launch_form(const Dims& D, int64_t nc, const clmgb_soiltemp_fields& ft, const clmgb_soilwater_fields& fw,
                        double dtime, int snow_method, double* t_ssbef, double* t_h2osfc_bef, uint32_t* col_status,
                        uint32_t* dev_status, double* st_log, int sh, cudaStream_t s) {
  const size_t smem = BLOCK ? (size_t)group_bytes<32>(32) : (size_t)TWARPS * (size_t)group_bytes<4>(1 << sh);
  auto kern = k_soil_temperature_packed<FRAC, LOG, BLOCK>;
  const cudaError_t e =
      allow_dynamic_smem(kern, BLOCK ? (size_t)group_bytes<32>(32) : (size_t)TWARPS * (size_t)group_bytes<4>(4));
  if (e != cudaSuccess) return e;
  const int64_t cols = BLOCK ? 32 : (int64_t)TWARPS << sh;
  int64_t grid = (nc + cols - 1) / cols;
  if (BLOCK) grid = (nc + SORTED - 1) / SORTED * (SORTED / 32);
  kern<<<(unsigned)grid, TBLOCK, smem, s>>>(D, nc, ft, fw, dtime, snow_method, t_ssbef, t_h2osfc_bef, col_status,
                                           dev_status, st_log, sh);
  return cudaGetLastError();
}

template <bool FRAC, bool LOG>
cudaError_t launch(const Dims& D, int64_t nc, const clmgb_soiltemp_fields& ft, const clmgb_soilwater_fields& fw,
                   double dtime, int snow_method, double* t_ssbef, double* t_h2osfc_bef, uint32_t* col_status,
                   uint32_t* dev_status, double* st_log, cudaStream_t s) {
  int dev = 0, nsm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || (e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
    return e;
  if (nc > warp_form_limit(nsm))
    return launch_form<FRAC, LOG, true>(D, nc, ft, fw, dtime, snow_method, t_ssbef, t_h2osfc_bef, col_status,
                                        dev_status, st_log, 0, s);
  int sh = 0;
  while (sh < 2 && (nc >> sh) > (int64_t)nsm * 12) sh++;
  return launch_form<FRAC, LOG, false>(D, nc, ft, fw, dtime, snow_method, t_ssbef, t_h2osfc_bef, col_status,
                                       dev_status, st_log, sh, s);
}

}  // namespace

cudaError_t launch_soil_temperature(const Dims& D, int64_t nc, const clmgb_soiltemp_fields& f, double dtime,
                                    int snow_method, uint32_t* col_status, uint32_t* dev_status, cudaStream_t s) {
  return launch<false, false>(D, nc, f, clmgb_soilwater_fields{}, dtime, snow_method, nullptr, nullptr, col_status,
                              dev_status, nullptr, s);
}

cudaError_t launch_soiltemp_fractions(const Dims& D, int64_t nc, const clmgb_soiltemp_fields& ft,
                                      const clmgb_soilwater_fields& fw, double dtime, int snow_method,
                                      double* t_ssbef, double* t_h2osfc_bef, uint32_t* col_status,
                                      uint32_t* dev_status, cudaStream_t s, double* st_log) {
  if (st_log)
    return launch<true, true>(D, nc, ft, fw, dtime, snow_method, t_ssbef, t_h2osfc_bef, col_status, dev_status,
                              st_log, s);
  return launch<true, false>(D, nc, ft, fw, dtime, snow_method, t_ssbef, t_h2osfc_bef, col_status, dev_status,
                             nullptr, s);
}

}  // namespace clmgb
