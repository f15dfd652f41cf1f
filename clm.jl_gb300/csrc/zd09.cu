// zd09.cu — soilwater_zengdecker2009! (soil_water_movement.jl:1616-1764), the
// Zeng & Decker (2009) soil water method: equilibrium water content and matric
// potential from the water-table depth, one implicit tridiagonal solve over the
// soil layers plus an aquifer layer, aquifer recharge and the water deficit.
//
// The reference runs ten kernels over [nc, nlevsoi(+1)] scratch matrices with a
// synchronisation between each.  Here one kernel runs them in the reference's order with
// the scratch in shared memory ([array][level][column]) and the levels spread over
// threads: _soilwm_mm_icefrac_kernel! (:97-127), _soilwm_zwtmm_kernel! (:143-150),
// _soilwm_jwt_vwczwt_kernel! (:289-327), _soilwm_voleq_zq_kernel! (:171-205),
// _soilwm_voleq_zq_aqu_kernel! (:346-366), _soilwm_hk_smp_kernel! (:223-270),
// _soilwm_aqu_zmm_kernel! (:385-397), _soilwm_tridiag_assemble_kernel! (:430-539),
// _tridiag_multi_kernel! (tridiagonal.jl:86-127), _soilwm_renew_qcharge_kernel!
// (:561-605), _soilwm_deficit_kernel! (:621-635).  smooth_min/max/ifelse are exact for
// Float64 (smooth_ad.jl:91-149, 253-256); ^ is Julia's Float64 pow (cm_pow).
//
// Two forms, as in soil_temperature_packed.cu: a warp with ks = 1, 2 or 4 columns and
// its lanes their levels, or a block of 32 columns, a lane each, whose four warps share the
// levels.  The fluxes between two levels, which the reference forms as the outflow of the
// upper and the inflow of the lower one by the same expressions, are formed once.  Only the
// tridiagonal sweep and the column scalars run a thread per column.
//
// Measured per call (us), against one thread per column with hardware divisions (and the
// FP64 pow): 61 columns 451 -> 35, 1,000 485 -> 42, 8,000 495 -> 105, 16,000 502 -> 136,
// 40,009 1,231 -> 286.  What bounds it: the powers (five to seven a level) and divisions,
// by latency at 20 warps per SM.
#include "clmgb_device.cuh"
#include "launch.h"

namespace clmgb {

namespace {

constexpr int ZWARPS = 4, ZD_BLOCK = 32 * ZWARPS;
constexpr int ZD_WARP_FORM = 48;
// Level arrays, of nlevsoi + 1 rows (the aquifer level's behind the soil's).  VWC and ICE
// (liquid volume and ice fractions) give way to the outflow of each level and its first
// derivative, HK, DHK, DSM (conductivity, its derivative, that of the matric potential) to
// the matrix, whose upper diagonal the outflow's second derivative is; ZQ and SMP stay for
// the recharge.
enum ZArray { Z_VWC = 0, Z_ICE, Z_ZQ, Z_HK, Z_DHK, Z_SMP, Z_DSM, Z_D2, Z_ARRAYS,
              Z_QO = Z_VWC, Z_D1 = Z_ICE, Z_A = Z_HK, Z_B = Z_DHK, Z_R = Z_DSM, Z_C = Z_D2 };
template <int N>
struct ZArea {
  int jwt[N];                     // the level above the water table
  unsigned int negative[N];       // levels whose new water is not >= 0
};
template <int N>
__host__ __device__ constexpr int64_t zd_bytes(int ks, int rows) {
  return (int64_t)Z_ARRAYS * rows * ks * 8 + (int64_t)((sizeof(ZArea<N>) + 15) / 16 * 16);
}

template <bool BLOCK>
__global__ void __launch_bounds__(ZD_BLOCK)
k_zd09(Dims D, int64_t nc, clmgb_zd09_fields f, double e_ice, double dtime, int sh) {
  extern __shared__ __align__(16) unsigned char smem_zd[];
  constexpr int NS = BLOCK ? 32 : 4;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int ks = BLOCK ? 32 : 1 << sh, s = lane & (ks - 1), lo = BLOCK ? wib : lane >> sh;
  const int nper = BLOCK ? ZWARPS : 32 >> sh;
  auto sync = [&]() {
    if (BLOCK) __syncthreads();
    else __syncwarp();
  };
  double* const rows = reinterpret_cast<double*>(smem_zd + (BLOCK ? 0 : wib * zd_bytes<NS>(ks, D.nlevsoi + 1)));
  ZArea<NS>& SA = *reinterpret_cast<ZArea<NS>*>(rows + (int64_t)Z_ARRAYS * (D.nlevsoi + 1) * ks);
  const int64_t group = BLOCK ? blockIdx.x : (int64_t)blockIdx.x * ZWARPS + wib;
  if (group * ks >= nc) return;                           // the whole group leaves together
  const int64_t c = group * ks + s, ld = D.ldc;
  const bool on = c < nc && f.mask_hydrology[c];
  const int nls = D.nlevsoi, nlevgrnd = D.nlevgrnd, joff = D.nlevsno, joff_zi = D.nlevsno + 1;
  auto A = [&](int a, int j) -> double& { return rows[(a * (nls + 1) + (j - 1)) * ks + s]; };
  const double zwt_m = on ? f.zwt[c] : 0.0, smpmin = on ? f.smpmin[c] : 0.0;
  const double zwt = zwt_m * 1.0e3;                       // water table in mm
  if (on && lo == 0) {
    SA.jwt[s] = nls;
    SA.negative[s] = 0u;
  }
  sync();
  // ---- ice and liquid volume fractions, the level above the water table ----
  if (on)
    for (int j = 1 + lo; j <= nls; j += nper) {
      const double ws = LVc(f.watsat, c, j, ld), dzj = LVc(f.dz, c, joff + j, ld);
      const double vol_ice = jl_min(ws, jl_div(LVc(f.h2osoi_ice, c, joff + j, ld), dzj * DENICE));
      const double icef = jl_min(1.0, jl_div(vol_ice, ws));
      LV(f.icefrac, c, j, ld) = icef;
      A(Z_ICE, j) = icef;
      A(Z_VWC, j) = jl_div(jl_max(LV(f.h2osoi_liq, c, joff + j, ld), 1.0e-6), dzj * DENH2O);
      if (zwt_m <= LVc(f.zi, c, joff_zi + j, ld)) atomicMin(&SA.jwt[s], j - 1);
    }
  sync();
  const int jwt = on ? SA.jwt[s] : nls;
  // ---- equilibrium water content and matric potential; hydraulic conductivity, matric
  // potential and their derivatives ----
  if (on)
    for (int j = 1 + lo; j <= nls; j += nper) {
      const double ws = LVc(f.watsat, c, j, ld), suc = LVc(f.sucsat, c, j, ld), b = LVc(f.bsw, c, j, ld);
      const double z_jm1 = j == 1 ? 0.0 : LVc(f.zi, c, joff_zi + j - 1, ld) * 1.0e3;
      const double z_j = LVc(f.zi, c, joff_zi + j, ld) * 1.0e3;
      double ve;
      if (zwt <= z_jm1) {
        ve = ws;
      } else {
        const double onem1b = 1.0 - jl_div(1.0, b);
        const bool inside = zwt < z_j && zwt > z_jm1;
        const double tempi = inside ? 1.0 : cm_pow(jl_div(suc + zwt - z_j, suc), onem1b);
        const double temp0 = cm_pow(jl_div(suc + zwt - z_jm1, suc), onem1b);
        const double k = jl_div(-suc * ws, onem1b);
        if (inside) {
          const double above_wt = zwt - z_jm1;
          const double voleq1 = jl_div(k, above_wt) * (tempi - temp0);
          double v = jl_div(voleq1 * above_wt + ws * (z_j - zwt), z_j - z_jm1);
          v = jl_min(ws, v);
          ve = jl_max(v, 0.0);
        } else {
          double v = jl_div(k, z_j - z_jm1) * (tempi - temp0);
          v = jl_max(v, 0.0);
          ve = jl_min(ws, v);
        }
      }
      const double zqv = -suc * cm_pow(jl_max(jl_div(ve, ws), 0.01), -b);
      A(Z_ZQ, j) = jl_max(smpmin, zqv);
      const int jp1 = min(nls, j + 1);
      const double wsp = LVc(f.watsat, c, jp1, ld), vwc = A(Z_VWC, j);
      double s1 = jl_div(half_of(vwc + A(Z_VWC, jp1)), half_of(ws + wsp));
      s1 = jl_min(1.0, s1);
      const double s2 = LVc(f.hksat, c, j, ld) * cm_pow(s1, 2.0 * b + 2.0);
      const double imp = cm_pow(10.0, -e_ice * half_of(A(Z_ICE, j) + A(Z_ICE, jp1)));
      const double hk = imp * s1 * s2;
      double s_node = jl_max(jl_div(vwc, ws), 0.01);
      s_node = jl_min(1.0, s_node);
      double smpv = -suc * cm_pow(s_node, -b);
      smpv = jl_max(smpmin, smpv);
      A(Z_HK, j) = hk;
      A(Z_DHK, j) = imp * (2.0 * b + 3.0) * s2 * jl_div(1.0, ws + wsp);
      A(Z_SMP, j) = smpv;
      A(Z_DSM, j) = jl_div(-b * smpv, vwc);
      LV(f.smp_l, c, j, ld) = smpv;
      LV(f.hk_l, c, j, ld) = hk;
    }
  sync();
  // ---- the bottom level and the aquifer level, a thread per column; vwc_zwt only matters
  // with the water table below the soil column ----
  const bool deep = on && jwt == nls;
  double q_n = 0.0, d1_n = 0.0, d2_n = 0.0;               // outflow of the bottom level
  double zmm_n = 0.0, dz_aq = 0.0;
  if (on && lo == 0) {
    const int j = nls;
    zmm_n = LVc(f.z, c, joff + j, ld) * 1.0e3;
    if (deep) {
      const double suc = LVc(f.sucsat, c, j, ld), ws = LVc(f.watsat, c, j, ld), b = LVc(f.bsw, c, j, ld);
      double vwc_zwt = ws;
      // the level below the soil column, or the last one where the grid has none below
      if (LVc(f.t_soisno, c, joff + min(jwt + 1, nlevgrnd), ld) < TFRZ) {
        double v = A(Z_VWC, j);
        for (int k = nls; k <= nlevgrnd; k++) {
          if (zwt_m <= LVc(f.zi, c, joff_zi + k, ld)) {
            const double t = LVc(f.t_soisno, c, joff + k, ld);
            double smp1 = jl_div(HFUS * (TFRZ - t), GRAV * t) * 1000.0;
            smp1 = jl_max(suc, smp1);
            v = ws * cm_pow(jl_div(smp1, suc), jl_div(-1.0, b));
            v = jl_min(v, half_of(ws + LVc(f.h2osoi_vol, c, nls, ld)));
            break;
          }
        }
        vwc_zwt = v;
      }
      const double z_j = LVc(f.zi, c, joff_zi + j, ld) * 1.0e3;
      const double onem1b = 1.0 - jl_div(1.0, b);
      const double temp0 = cm_pow(jl_div(suc + zwt - z_j, suc), onem1b);
      double v = jl_div(jl_div(-suc * ws, onem1b), zwt - z_j) * (1.0 - temp0);
      v = jl_max(v, 0.0);
      v = jl_min(ws, v);
      const double zq_aq = jl_max(smpmin, -suc * cm_pow(jl_max(jl_div(v, ws), 0.01), -b));
      double s_node = jl_max(half_of(jl_div(vwc_zwt + A(Z_VWC, j), ws)), 0.01);
      s_node = jl_min(1.0, s_node);
      double smp1 = -suc * cm_pow(s_node, -b);
      smp1 = jl_max(smpmin, smp1);
      const double dsmpdw1 = jl_div(-b * smp1, s_node * ws);
      const double zmm_aq = half_of(1.0e3 * zwt_m + zmm_n);
      dz_aq = 1.0e3 * zwt_m - zmm_n;
      const double den = zmm_aq - zmm_n;
      const double num = (smp1 - A(Z_SMP, j)) - (zq_aq - A(Z_ZQ, j));
      const double hk = A(Z_HK, j), dhk = A(Z_DHK, j);
      q_n = jl_div(-hk * num, den);
      d1_n = jl_div(-(-hk * A(Z_DSM, j) + num * dhk), den);
      d2_n = jl_div(-(hk * dsmpdw1 + num * dhk), den);
    } else {
      dz_aq = LVc(f.dz, c, joff + j, ld) * 1.0e3;
    }
  }
  sync();                                                  // VWC and ICE are read
  // ---- the fluxes between levels j and j+1 and their derivatives ----
  if (on)
    for (int j = 1 + lo; j < nls; j += nper) {
      const double den = LVc(f.z, c, joff + j + 1, ld) * 1.0e3 - LVc(f.z, c, joff + j, ld) * 1.0e3;
      const double num = (A(Z_SMP, j + 1) - A(Z_SMP, j)) - (A(Z_ZQ, j + 1) - A(Z_ZQ, j));
      const double hk = A(Z_HK, j), dhk = A(Z_DHK, j), nd = num * dhk;
      A(Z_QO, j) = jl_div(-hk * num, den);
      A(Z_D1, j) = jl_div(-(-hk * A(Z_DSM, j) + nd), den);
      A(Z_D2, j) = jl_div(-(hk * A(Z_DSM, j + 1) + nd), den);
    }
  if (on && lo == 0) {
    A(Z_QO, nls) = q_n;
    A(Z_D1, nls) = d1_n;
    A(Z_D2, nls) = d2_n;
  }
  sync();                                                  // HK, DHK and DSM are read
  // ---- the tridiagonal system ----
  if (on)
    for (int j = 1 + lo; j <= nls; j += nper) {
      const double dzmm = LVc(f.dz, c, joff + j, ld) * 1.0e3, root = LVc(f.qflx_rootsoi, c, j, ld);
      if (j == 1) {
        A(Z_R, 1) = f.qflx_infl[c] - A(Z_QO, 1) - root;
        A(Z_A, 1) = 0.0;
        A(Z_B, 1) = dzmm * (0.0 + jl_div(1.0, dtime)) + A(Z_D1, 1);
      } else {
        A(Z_R, j) = A(Z_QO, j - 1) - A(Z_QO, j) - root;
        A(Z_A, j) = -A(Z_D1, j - 1);
        A(Z_B, j) = jl_div(dzmm, dtime) - A(Z_D2, j - 1) + A(Z_D1, j);
      }
    }
  if (on && lo == 0) {
    const double b = jl_div(dz_aq, dtime);
    A(Z_R, nls + 1) = deep ? q_n - 0.0 : 0.0;
    A(Z_A, nls + 1) = deep ? -d1_n : 0.0;
    A(Z_B, nls + 1) = deep ? b - d2_n + 0.0 : b;
    A(Z_C, nls + 1) = 0.0;
  }
  sync();
  // ---- tridiagonal_multi! over the soil levels and the aquifer level (jtop = 1) ----
  if (on && lo == 0) {
    const int n = nls + 1;
    double cp = 0.0, dp = 0.0;
    for (int j = 1; j <= n; j++) {
      double den = A(Z_B, j), num = A(Z_R, j);
      const double cj = A(Z_C, j);
      if (j == 1) {
        if (abs_lt(den, 1.0e-30)) den = 1.0e-30;
      } else {
        const double a = A(Z_A, j);
        den = den - a * cp;
        if (abs_lt(den, 1.0e-30)) den = copysign(1.0e-30, den == 0.0 ? 1.0 : den);
        num = num - a * dp;
      }
      div_pair(cj, num, den, cp, dp);
      A(Z_C, j) = cp;
      A(Z_R, j) = dp;
    }
    for (int j = n - 1; j >= 1; j--) {
      dp = A(Z_R, j) - A(Z_C, j) * dp;
      A(Z_R, j) = dp;
    }
  }
  sync();
  // ---- the new liquid water ----
  if (on)
    for (int j = 1 + lo; j <= nls; j += nper) {
      const double l = LV(f.h2osoi_liq, c, joff + j, ld) + A(Z_R, j) * (LVc(f.dz, c, joff + j, ld) * 1.0e3);
      LV(f.h2osoi_liq, c, joff + j, ld) = l;
      A(Z_A, j) = l;
      if (!(l >= 0.0)) atomicOr(&SA.negative[s], 1u << j);
    }
  sync();
  // ---- aquifer recharge, water deficit ----
  if (on && lo == 0) {
    double qc;
    if (jwt < nls) {
      const int jw = jwt, jn = jw + 1, jp1 = min(nls, jn + 1);
      const double s_node = jl_max(jl_div(LVc(f.h2osoi_vol, c, jn, ld), LVc(f.watsat, c, jn, ld)), 0.01);
      const double s1 = jl_min(1.0, s_node);
      const double imp = cm_pow(10.0, -e_ice * half_of(LV(f.icefrac, c, jn, ld) + LV(f.icefrac, c, jp1, ld)));
      const double ka = imp * LVc(f.hksat, c, jn, ld) * cm_pow(s1, 2.0 * LVc(f.bsw, c, jn, ld) + 3.0);
      const int jm = jw > 1 ? jw : 1;
      const double smp1 = jl_max(smpmin, A(Z_SMP, jm));
      const double wh = smp1 - A(Z_ZQ, jm);
      if (jw == 0) qc = jl_div(-ka * (0.0 - wh), (zwt_m + 1.0e-3) * 1000.0);
      else qc = jl_div(-ka * (0.0 - wh), (zwt_m - LVc(f.z, c, joff + jw, ld)) * 1000.0 * 2.0);
      qc = jl_max(jl_div(-10.0, dtime), qc);
      qc = jl_min(jl_div(10.0, dtime), qc);
    } else {
      qc = jl_div(A(Z_R, nls + 1) * dz_aq, dtime);
    }
    f.qcharge[c] = qc;
    double acc = 0.0;
    for (unsigned int m = SA.negative[s]; m; m &= m - 1) acc = acc + -A(Z_A, __ffs((int)m) - 1);
    f.qflx_deficit[c] = acc;
  }
}

template <bool BLOCK>
cudaError_t launch_form(const Dims& D, int64_t nc, const clmgb_zd09_fields& f, double e_ice, double dtime, int sh,
                        cudaStream_t s) {
  const size_t smem = BLOCK ? (size_t)zd_bytes<32>(32, D.nlevsoi + 1) : (size_t)ZWARPS * (size_t)zd_bytes<4>(1 << sh, D.nlevsoi + 1);
  const cudaError_t e = allow_dynamic_smem(k_zd09<BLOCK>, BLOCK ? (size_t)zd_bytes<32>(32, MAXSOI + 1)
                                                               : (size_t)ZWARPS * (size_t)zd_bytes<4>(4, MAXSOI + 1));
  if (e != cudaSuccess) return e;
  const int64_t cols = BLOCK ? 32 : (int64_t)ZWARPS << sh;
  k_zd09<BLOCK><<<(unsigned)((nc + cols - 1) / cols), ZD_BLOCK, smem, s>>>(D, nc, f, e_ice, dtime, sh);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_zd09(const Dims& D, int64_t nc, const clmgb_zd09_fields& f, double e_ice, double dtime,
                        cudaStream_t s) {
  int dev = 0, nsm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || (e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
    return e;
  // the warp form up to 48 columns per SM: at 6,000 columns (39 per SM) it took 89 us
  // against 105 of the block form, at 8,000 (53) 107 against 105, at 16,000 170 against 136
  if (nc > (int64_t)nsm * ZD_WARP_FORM) return launch_form<true>(D, nc, f, e_ice, dtime, 0, s);
  int sh = 0;
  while (sh < 2 && (nc >> sh) > (int64_t)nsm * 16) sh++;
  return launch_form<false>(D, nc, f, e_ice, dtime, sh, s);
}

}  // namespace clmgb
