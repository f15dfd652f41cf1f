// kernels.cu — CUDA kernels of the soil/snow column solve (one thread per column).
#include "clmgb_device.cuh"
#include "launch.h"
#include "work_order.cuh"
#include "richards_coop.cuh"

namespace clmgb {

constexpr int BLOCK = 128;

static inline unsigned grid_for(int64_t n) { return (unsigned)((n + BLOCK - 1) / BLOCK); }

__device__ __forceinline__ void report(uint32_t st, uint32_t* col_status, uint32_t* dev_status, int64_t c) {
  if (col_status) col_status[c] = st;
  if (st && dev_status) atomicOr(dev_status, st);
}

// a thread per column and level (a thread per column: 17 us at 1,024 columns, a chain of 20
// levels' divisions; this, 2.6)
__global__ void __launch_bounds__(BLOCK)
k_water_fractions(Dims D, int64_t nc, clmgb_soilwater_fields f) {
  const int64_t c = (int64_t)blockIdx.x * BLOCK + threadIdx.x;
  if (c >= nc) return;
  if (f.mask_hydrology[c]) water_fractions_level(D, f, c, 1 + (int)blockIdx.y);
}

__global__ void __launch_bounds__(BLOCK)
k_moisture_form(Dims D, int64_t nc, clmgb_soilwater_fields f, clmgb_swm_config cfg, double dtime,
                uint32_t* col_status, uint32_t* dev_status) {
  const int64_t c = (int64_t)blockIdx.x * BLOCK + threadIdx.x;
  if (c >= nc) return;
  uint32_t st = 0;
  if (f.mask_hydrology[c]) st = moisture_form_col(D, f, cfg, dtime, c);
  report(st, col_status, dev_status, c);
}

// soil_temperature! -> set_soil_water_fractions! -> soil_water! for one column, one launch.
__global__ void __launch_bounds__(BLOCK)
k_column_step(Dims D, int64_t nc, clmgb_soiltemp_fields ft, clmgb_soilwater_fields fw, clmgb_swm_config cfg,
              double dtime, int snow_method, double* t_ssbef, double* t_h2osfc_bef,
              uint32_t* col_status, uint32_t* dev_status) {
  const int64_t c = (int64_t)blockIdx.x * BLOCK + threadIdx.x;
  if (c >= nc) return;
  uint32_t st = 0;
  if (ft.mask_nolakec[c]) {
    if (t_ssbef) {
      const int L = D.nlevsno + D.nlevmax;
      for (int jj = 1; jj <= L; jj++) LV(t_ssbef, c, jj, D.ldc) = LV(ft.t_soisno, c, jj, D.ldc);
    }
    if (t_h2osfc_bef) t_h2osfc_bef[c] = ft.t_h2osfc[c];
    st |= soil_temperature_col(D, ft, c, dtime, snow_method);
  }
  if (fw.mask_hydrology[c]) {
    water_fractions_col(D, fw, c);
    st |= moisture_form_col(D, fw, cfg, dtime, c);
  }
  report(st, col_status, dev_status, c);
}

// soilwm_moisture_form_solve! as a persistent kernel fed by a device work queue.
// Each lane owns one column at a time and advances it one substep attempt per loop
// trip; when its column finishes it takes the next column index from the queue
// (one atomicAdd per warp for all lanes that need work).  Columns need from 1 to
// ~70 attempts, so lanes stay busy instead of waiting for the slowest column of
// the warp.  With `order` the queue hands out columns in that order (longest
// expected first) and the impedances come precomputed in imp_cache.  The
// per-column arithmetic is unchanged, so results do not depend on the schedule.
// `queue` must be zero at launch.
// With LOG the kernel also writes the substep log of every column it solves (the
// starting water of each accepted substep and the solve's outputs), for the step
// adjoint; the solve itself is unchanged.
// With qs.defer > 0 (never with LOG) a column that has made qs.defer attempts and
// is not done leaves the lane at its next accepted substep: the lane stores the
// column's state and takes new work, and warps that run out of queued columns
// finish the deferred ones one warp per column (coop_drain, richards_coop.cuh), so
// the few columns that need several times the mean number of attempts no longer
// hold the kernel's end with one useful lane per warp.
template <bool LOG>
__global__ void __launch_bounds__(BLOCK)
k_moisture_form_queue(Dims D, int64_t nc, clmgb_soilwater_fields f, clmgb_swm_config cfg, double dtime,
                      uint32_t* col_status, int or_status, uint32_t* dev_status, unsigned long long* queue,
                      const uint32_t* order, const unsigned int* nlisted_ptr, const double* imp_cache,
                      int64_t ld_imp, const double* dt_init, SubstepLogView lg, int fresh_batch, QueueScratch qs) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned long long nq = order ? (unsigned long long)(*(volatile const unsigned int*)nlisted_ptr)
                                      : (unsigned long long)nc;
  MfLane L;
  int nacc = 0;
  bool active = false, exhausted = false, kept = false;
  for (;;) {
    const bool need = !active && !exhausted;
    const unsigned m = __ballot_sync(FULL, need);
    if (m) {
      const int leader = __ffs(m) - 1;
      unsigned long long base = 0;
      if (lane == leader) base = atomicAdd(queue, (unsigned long long)__popc(m));
      base = __shfl_sync(FULL, base, leader);
      if (need) {
        const unsigned long long k = base + (unsigned long long)__popc(m & ((1u << lane) - 1u));
        if (k >= nq) {
          exhausted = true;
        } else {
          const int64_t c = order ? (int64_t)order[k] : (int64_t)k;
          if (order || f.mask_hydrology[c]) {
            if (mf_begin(L, D, f, cfg, dtime, c, imp_cache, ld_imp, dt_init)) {
              active = true;
              nacc = 0;
              kept = false;
            } else {
              const uint32_t st = L.status;
              if (col_status) col_status[c] = or_status ? (col_status[c] | st) : st;
              if (st && dev_status) atomicOr(dev_status, st);
            }
          } else if (col_status && !or_status) {
            col_status[c] = 0;
          }
        }
      }
    }
    if (!__any_sync(FULL, active)) {
      if (__all_sync(FULL, exhausted)) {
        // no queued column left for this warp: finish deferred ones, one warp each
        if (!LOG && qs.defer > 0) coop_drain(D, f, cfg, dtime, col_status, or_status, dev_status, qs);
        break;
      }
      continue;
    }
    // Batched refresh.  A lane whose substep was just accepted needs the hydraulic
    // block (mf_refresh, about 2.7 attempts' worth of FP64 work) before its next
    // attempt.  Run at once, it idles the other lanes of the warp; with
    // fresh_batch > 0 such lanes wait while the others attempt, until fresh_batch of
    // them need it or no lane can attempt, and then run it together.  Each column's
    // operations and their order are unchanged.
    bool can_try = active;
    if (fresh_batch > 0) {
      const bool want = active && L.fresh && L.nsub < D.attempt_cap;
      const unsigned wm = __ballot_sync(FULL, want);
      const unsigned tm = __ballot_sync(FULL, active && !want);
      if (wm && (__popc(wm) >= fresh_batch || tm == 0) && want) {
        if (LOG && nacc < lg.cap) {
          double* r0 = lg.rec + L.c * lg.stride + (int64_t)nacc * SUB_REC;
          for (int j = 1; j <= L.nlayers; j++) r0[j - 1] = L.liq[j];
        }
        FieldState<clmgb_soilwater_fields> X(f, L.c, D.ldc);
        mf_refresh(L, D, f, cfg, X);
      }
      can_try = active && !(L.fresh && L.nsub < D.attempt_cap);
    }
    if (!can_try) continue;
    double* rec = nullptr;
    double dts = 0.0, dtd = 0.0;
    if (LOG) {
      rec = lg.rec + L.c * lg.stride;
      if (L.fresh && nacc < lg.cap)
        for (int j = 1; j <= L.nlayers; j++) rec[(int64_t)nacc * SUB_REC + j - 1] = L.liq[j];
      dts = L.dtsub;
      dtd = L.dtdone;
    }
    const bool fin = mf_attempt(L, D, f, cfg, dtime);
    if (LOG && L.dtdone != dtd) {
      if (nacc < lg.cap) {
        rec[(int64_t)nacc * SUB_REC + MAXSOI] = dts;
        rec[(int64_t)nacc * SUB_REC + MAXSOI + 1] = dtd;
      }
      nacc++;
    }
    if (!LOG && !fin && qs.defer > 0 && L.fresh && L.nsub >= qs.defer && !kept) {
      // hand the column over; a slot the drain gave back leaves it with this lane
      if (coop_defer(L, qs)) {
        active = false;
        continue;
      }
      kept = true;
    }
    if (fin) {
      const uint32_t st = mf_end(L, D, f);
      if (LOG) {
        double* out = rec + (int64_t)lg.cap * SUB_REC;
        for (int j = 1; j <= L.nlayers; j++) {
          out[j - 1] = L.liq[j];
          out[MAXSOI + j - 1] = LV(f.smp_l, L.c, j, D.ldc);
          out[2 * MAXSOI + j - 1] = LV(f.hk_l, L.c, j, D.ldc);
        }
        out[3 * MAXSOI] = L.qc;
        out[3 * MAXSOI + 1] = (double)L.nsub;
        out[3 * MAXSOI + 2] = (double)st;
        lg.count[L.c] = nacc;
      }
      if (col_status) col_status[L.c] = or_status ? (col_status[L.c] | st) : st;
      if (st && dev_status) atomicOr(dev_status, st);
      active = false;
    }
  }
}

// compute_qcharge! after a moisture-form solve with the water-table lower boundary
// (soil_water_movement.jl:1575-1598): one thread per hydrology column the solve
// could take (nbedrock in range).
__global__ void __launch_bounds__(BLOCK)
k_compute_qcharge(Dims D, int64_t nc, clmgb_soilwater_fields f, double dtime) {
  const int64_t c = (int64_t)blockIdx.x * BLOCK + threadIdx.x;
  if (c >= nc || !f.mask_hydrology[c]) return;
  const int64_t nl = f.col_nbedrock[c];
  if (nl < 1 || nl > D.nlevsoi) return;
  compute_qcharge_col(D, f, dtime, c);
}

// The use_flexibleCN branch of soil_water! (soil_water_movement.jl:1812-1843) for one
// column: smooth_ifelse on Float64 is the exact branch x >= 0 ? a : b (smooth_ad.jl:253-257).
__global__ void __launch_bounds__(BLOCK)
k_flexible_cn(Dims D, int64_t nc, clmgb_flexcn_fields f) {
  const int64_t c = (int64_t)blockIdx.x * BLOCK + threadIdx.x;
  if (c >= nc || !f.mask_hydrology[c]) return;
  const int64_t ld = D.ldc;
  const int joff = D.nlevsno, nlevsoi = D.nlevsoi;
  const double watmin = 0.001;
  for (int j = 1; j <= nlevsoi - 1; j++) {
    double& lj = LV(f.h2osoi_liq, c, joff + j, ld);
    const double xs = lj >= 0.0 ? 0.0 : watmin - lj;
    lj = lj + xs;
    double& ln = LV(f.h2osoi_liq, c, joff + j + 1, ld);
    ln = ln - xs;
  }
  {
    double& lj = LV(f.h2osoi_liq, c, joff + nlevsoi, ld);
    const double xs = (lj - watmin) >= 0.0 ? 0.0 : watmin - lj;
    lj = lj + xs;
    f.wa[c] = f.wa[c] - xs;
  }
  for (int j = 1; j <= nlevsoi; j++) {
    const double dzv = LVc(f.dz, c, joff + j, ld);
    LV(f.h2osoi_vol, c, j, ld) =
        jl_div(LV(f.h2osoi_liq, c, joff + j, ld), dzv * DENH2O) + jl_div(LVc(f.h2osoi_ice, c, joff + j, ld), dzv * DENICE);
  }
}

// Ice impedances of every hydrology column, one thread per column, into imp_cache
// [nlevsoi][ld_imp] (uniform work: no lane waits on another column).
__global__ void __launch_bounds__(BLOCK)
k_impedance(Dims D, int64_t nc, clmgb_soilwater_fields f, double e_ice, double* imp_cache, int64_t ld_imp) {
  const int64_t c = (int64_t)blockIdx.x * BLOCK + threadIdx.x;
  if (c >= nc || !f.mask_hydrology[c]) return;
  const int64_t nl = f.col_nbedrock[c];
  if (nl < 1 || nl > D.nlevsoi) return;
  const int nlayers = (int)nl;
  for (int j = 1; j <= nlayers; j++) imp_cache[(int64_t)(j - 1) * ld_imp + c] = mf_impedance(D, f, e_ice, c, j, nlayers);
}

// Longest-expected-first order of the hydrology columns: the key is the previous call's
// substep count (num_substeps, the state field); NaN or non-positive counts are key 0.
struct SubstepKey {
  const uint8_t* mask;
  const double* num_substeps;
  uint32_t* col_status;
  int or_status;
  __device__ int operator()(int64_t c) const {
    if (!mask[c]) return -1;
    const double ns = num_substeps[c];
    if (!(ns > 0.0)) return 0;
    return ns >= (double)(ORDER_BINS - 1) ? ORDER_BINS - 1 : (int)ns;
  }
  __device__ void unlisted(int64_t c) const {
    if (col_status && !or_status) col_status[c] = 0;
  }
};

// Evaluates the shared transcendentals (clm_math.h) elementwise; op 0 log, 1 exp,
// 2 pow, 3 log10.  Used to check that GPU and CPU builds return identical bits.
__global__ void __launch_bounds__(BLOCK)
k_math_eval(int op, int64_t n, const double* x, const double* y, double* out) {
  const int64_t i = (int64_t)blockIdx.x * BLOCK + threadIdx.x;
  if (i >= n) return;
  const double a = x[i];
  double r;
  if (op == 0) r = cm_log(a);
  else if (op == 1) r = cm_exp(a);
  else if (op == 2) r = cm_pow(a, y[i]);
  else if (op == 3) r = cm_log10(a);
  else if (op == 4) r = cm_sin(a);
  else if (op == 5) r = cm_acos(a);
  else r = jl_div(a, y[i]);
  out[i] = r;
}

__global__ void __launch_bounds__(BLOCK)
k_phase_change(Dims D, int64_t nc, clmgb_soiltemp_fields f, double dtime, const double* dhsdT, int which) {
  const int64_t c = (int64_t)blockIdx.x * BLOCK + threadIdx.x;
  if (c >= nc || !f.mask_nolakec[c]) return;
  if (which == 0) phase_change_h2osfc_col(D, f, c, dtime, dhsdT[c]);
  else phase_change_beta_col(D, f, c, dtime, dhsdT[c]);
}

// batched_band_solve! (band_diagonal.jl:87-170), a thread per column: band_lu_solve's
// elimination with its window of KL+1 rows in registers, the rows entering it straight
// from the band matrix and the right-hand side; the thread keeps the rows of U, and
// tvector the eliminated right-hand side until the back substitution.  Row exchanges are
// decided on the bits.  65,537 systems of 26 to 38 rows with five full bands: 186 us,
// 342 with the band copied to a 2.5 KB stack first and FP64 comparisons.  28 FP64
// instructions a row, 65 cycles of the sub-partition's FP64 unit each, bound it (110 us).
template <int KL, int KU>
__global__ void __launch_bounds__(BLOCK)
k_band_solve(int64_t nc, int64_t ldc, int nlev, double* tvector, const double* __restrict__ bmatrix,
             const double* __restrict__ rvector, const int64_t* jtop, const int64_t* jbot,
             const uint8_t* mask, int nlevsno_off) {
  constexpr int R = KL + 1, C = KL + KU + 1;
  const int64_t c = (int64_t)blockIdx.x * BLOCK + threadIdx.x;
  if (c >= nc || !mask[c]) return;
  const int64_t jt = jtop[c] + nlevsno_off + 1;
  const int64_t n64 = jbot[c] - jtop[c] + 1;
  if (n64 <= 0 || jt < 1 || jt + n64 - 1 > nlev || n64 > MAXROWS + 1) return;
  const int n = (int)n64;
  const double* const bm = bmatrix + c + (jt - 1) * ldc * C;
  const double* const rv = rvector + c + (jt - 1) * ldc;
  double* const tv = tvector + c + (jt - 1) * ldc;
  // A[i, j] of the band (j = i - KL .. i + KU), 0 outside the system
  auto entry = [&](int i, int j) -> double {
    return j >= 0 && j < n ? bm[(int64_t)(i - j + KL) * ldc + (int64_t)i * ldc * C] : 0.0;
  };
  double u[(MAXROWS + 1) * C];
  double w[R][C], x[R];
#pragma unroll
  for (int i = 0; i < R; i++) {
#pragma unroll
    for (int k = 0; k < C; k++) w[i][k] = i < n && k - i <= KU ? entry(i, k) : 0.0;
    x[i] = i < n ? rv[i * ldc] : 0.0;
  }
  for (int k = 0; k < n; k++) {
    const int r = k + 1 + KL;                       // the row that enters below
    double nw[C], nx = 0.0;
#pragma unroll
    for (int i = 0; i < C; i++) nw[i] = r < n ? entry(r, k + 1 + i) : 0.0;
    if (r < n) nx = rv[(int64_t)r * ldc];
    int piv = 0;
    long long maxv = dbits(w[0][0]) & 0x7fffffffffffffffLL;
#pragma unroll
    for (int i = 1; i < R; i++) {
      const long long v = dbits(w[i][0]) & 0x7fffffffffffffffLL;
      if (k + i < n && v > maxv && v <= 0x7ff0000000000000LL) {
        maxv = v;
        piv = i;
      }
    }
#pragma unroll
    for (int i = 1; i < R; i++) {
      const bool sw = i == piv;
#pragma unroll
      for (int e = 0; e < C; e++) {
        const double t = w[0][e];
        w[0][e] = sw ? w[i][e] : t;
        w[i][e] = sw ? t : w[i][e];
      }
      const double t = x[0];
      x[0] = sw ? x[i] : t;
      x[i] = sw ? t : x[i];
    }
    double f[R];
    if (k + R - 1 < n) {
      if constexpr (R == 3) div_pair(w[1][0], w[2][0], w[0][0], f[1], f[2]);
      else f[1] = jl_div(w[1][0], w[0][0]);
    } else if (k + 1 < n) {
      f[1] = jl_div(w[1][0], w[0][0]);
    }
#pragma unroll
    for (int i = 1; i < R; i++) {
      if (k + i < n) {
#pragma unroll
        for (int e = 1; e < C; e++) w[i][e] = w[i][e] - f[i] * w[0][e];
        x[i] = x[i] - f[i] * x[0];
      }
    }
#pragma unroll
    for (int e = 0; e < C; e++) u[k * C + e] = w[0][e];
    tv[(int64_t)k * ldc] = x[0];
    // slide down a row and right a column
#pragma unroll
    for (int i = 0; i < R - 1; i++) {
#pragma unroll
      for (int e = 0; e < C - 1; e++) w[i][e] = w[i + 1][e + 1];
      w[i][C - 1] = 0.0;
      x[i] = x[i + 1];
    }
#pragma unroll
    for (int e = 0; e < C; e++) w[R - 1][e] = nw[e];
    x[R - 1] = nx;
  }
  double y[C];                                      // x of the rows below
#pragma unroll
  for (int e = 0; e < C; e++) y[e] = 0.0;
  for (int i = n - 1; i >= 0; i--) {
    double s = tv[(int64_t)i * ldc];
#pragma unroll
    for (int e = 1; e < C; e++)
      if (i + e < n) s = s - u[i * C + e] * y[e - 1];
    const double xi = jl_div(s, u[i * C]);
#pragma unroll
    for (int e = C - 1; e > 0; e--) y[e] = y[e - 1];
    y[0] = xi;
    tv[(int64_t)i * ldc] = xi;
  }
}

constexpr int MAXTRI = 64;

// tridiagonal_multi! (tridiagonal.jl:86-127), a thread per column.  The coefficients are
// loaded three levels ahead (one level ahead measured 72 us for the case below: a level's
// arithmetic is shorter than a load); of the sweep's two results per level one waits in
// shared memory ([level][thread], no bank conflicts), the other in u.  100,003 systems of
// 21 levels: 37 us, 113 with the hardware division, FP64 comparisons, loads in step and
// the results in local memory.  Six FP64 instructions a level (20 us) and 101 MB of memory
// traffic (15 us) bound it.
__global__ void __launch_bounds__(BLOCK)
k_tridiagonal_multi(int64_t ncols, int64_t ld, int nlevs, double* u, const double* __restrict__ a,
                    const double* __restrict__ b, const double* __restrict__ cc, const double* __restrict__ r,
                    const int64_t* jtop, const uint8_t* mask) {
  extern __shared__ double smem_tri[];
  const int nt = blockDim.x;
  const int64_t col = (int64_t)blockIdx.x * nt + threadIdx.x;
  if (col >= ncols || !mask[col]) return;
  const int64_t j64 = jtop[col];
  if (j64 < 1 || j64 > nlevs) return;
  const int j = (int)j64;
  double* const cp = smem_tri + threadIdx.x;
  const double tiny = 1e-30;
  struct Level { double a, b, c, r; };
  auto load = [&](int jj) -> Level {
    if (jj > nlevs) return Level{0.0, 0.0, 0.0, 0.0};
    return Level{LVc(a, col, jj, ld), LVc(b, col, jj, ld), LVc(cc, col, jj, ld), LVc(r, col, jj, ld)};
  };
  Level v = load(j), v1 = load(j + 1), v2 = load(j + 2);
  double cp_prev = 0.0, dp_prev = 0.0;
  for (int jj = j; jj <= nlevs; jj++) {
    const Level v3 = load(jj + 3);
    double denom = v.b, num = v.r;
    if (jj == j) {
      if (abs_lt(denom, tiny)) denom = tiny;
    } else {
      denom = v.b - v.a * cp_prev;
      if (abs_lt(denom, tiny)) denom = copysign(tiny, denom == 0.0 ? 1.0 : denom);
      num = v.r - v.a * dp_prev;
    }
    div_pair(v.c, num, denom, cp_prev, dp_prev);
    cp[(jj - 1) * nt] = cp_prev;
    LV(u, col, jj, ld) = dp_prev;
    v = v1;
    v1 = v2;
    v2 = v3;
  }
  double u_next = dp_prev, d = nlevs > j ? LV(u, col, nlevs - 1, ld) : 0.0;
  for (int jj = nlevs - 1; jj >= j; jj--) {
    const double dn = jj > j ? LV(u, col, jj - 1, ld) : 0.0;
    u_next = d - cp[(jj - 1) * nt] * u_next;
    LV(u, col, jj, ld) = u_next;
    d = dn;
  }
}

// The same systems by parallel cyclic reduction, one warp per column (CLMGB_TRIDIAG_PCR):
// lane l holds rows l and l+32 of the column's n = nlevs - jtop + 1 <= 64 unknowns in
// registers.  Each round with stride k eliminates the couplings to rows i-k and i+k
// (rows outside the system act as identity rows), so after ceil(log2 n) rounds every
// row stands alone and x_i = r_i / b_i.  The divisors get the reference's 1e-30
// pivot guard.  Without pivoting it is meant for the diagonally dominant systems of the
// soil-water and lake solves; its rounding differs from the sequential elimination's.
constexpr int PCR_WARPS = 4;
// row t (0..32*NH-1) of a value held as v[h] for rows lane + 32h
template <int NH>
__device__ __forceinline__ double pcr_row(const double* v, int t) {
  const double x0 = __shfl_sync(0xffffffffu, v[0], t & 31);
  if (NH == 1) return x0;
  const double x1 = __shfl_sync(0xffffffffu, v[NH - 1], t & 31);
  return (t >> 5) ? x1 : x0;
}
__device__ __forceinline__ double pcr_guard(double d) {
  return fabs(d) < 1e-30 ? copysign(1e-30, d == 0.0 ? 1.0 : d) : d;
}
// the system of one column, n <= 32*NH unknowns, rows lane + 32h of this lane
template <int NH>
__device__ __forceinline__ void pcr_solve(int64_t col, int64_t ld, int j0, int n, double* u,
                                          const double* __restrict__ a, const double* __restrict__ b,
                                          const double* __restrict__ cc, const double* __restrict__ r) {
  const int lane = threadIdx.x & 31;
  double A[NH], B[NH], C[NH], R[NH];
#pragma unroll
  for (int h = 0; h < NH; h++) {
    const int i = lane + 32 * h;
    if (i < n) {
      const int lev = j0 + i;
      A[h] = i == 0 ? 0.0 : LVc(a, col, lev, ld);
      B[h] = LVc(b, col, lev, ld);
      C[h] = i == n - 1 ? 0.0 : LVc(cc, col, lev, ld);
      R[h] = LVc(r, col, lev, ld);
    } else {
      A[h] = 0.0; B[h] = 1.0; C[h] = 0.0; R[h] = 0.0;
    }
  }
  for (int k = 1; k < n; k <<= 1) {
    double An[NH], Bn[NH], Cn[NH], Rn[NH];
#pragma unroll
    for (int h = 0; h < NH; h++) {
      const int i = lane + 32 * h;
      const int lo = i - k, hi = i + k;
      // rows i-k and i+k (identity rows outside 0..n-1); every lane joins every shuffle
      const int tl = lo < 0 ? 0 : lo, th = hi > 32 * NH - 1 ? 32 * NH - 1 : hi;
      double al = pcr_row<NH>(A, tl), bl = pcr_row<NH>(B, tl), cl = pcr_row<NH>(C, tl), rl = pcr_row<NH>(R, tl);
      double ah = pcr_row<NH>(A, th), bh = pcr_row<NH>(B, th), ch = pcr_row<NH>(C, th), rh = pcr_row<NH>(R, th);
      if (lo < 0) { al = 0.0; bl = 1.0; cl = 0.0; rl = 0.0; }
      if (hi >= n) { ah = 0.0; bh = 1.0; ch = 0.0; rh = 0.0; }
      const double alpha = -A[h] / pcr_guard(bl);
      const double gamma = -C[h] / pcr_guard(bh);
      An[h] = alpha * al;
      Cn[h] = gamma * ch;
      Bn[h] = B[h] + alpha * cl + gamma * ah;
      Rn[h] = R[h] + alpha * rl + gamma * rh;
    }
#pragma unroll
    for (int h = 0; h < NH; h++) {
      A[h] = An[h]; B[h] = Bn[h]; C[h] = Cn[h]; R[h] = Rn[h];
    }
  }
#pragma unroll
  for (int h = 0; h < NH; h++) {
    const int i = lane + 32 * h;
    if (i < n) LV(u, col, j0 + i, ld) = R[h] / pcr_guard(B[h]);
  }
}
__global__ void __launch_bounds__(32 * PCR_WARPS)
k_tridiagonal_multi_pcr(int64_t ncols, int64_t ld, int nlevs, double* u, const double* __restrict__ a,
                        const double* __restrict__ b, const double* __restrict__ cc,
                        const double* __restrict__ r, const int64_t* jtop, const uint8_t* mask) {
  const int64_t col = (int64_t)blockIdx.x * PCR_WARPS + (threadIdx.x >> 5);
  if (col >= ncols || !mask[col]) return;             // the whole warp leaves together
  const int64_t j64 = jtop[col];
  if (j64 < 1 || j64 > nlevs) return;
  const int j0 = (int)j64, n = nlevs - j0 + 1;
  if (n <= 32) pcr_solve<1>(col, ld, j0, n, u, a, b, cc, r);
  else pcr_solve<2>(col, ld, j0, n, u, a, b, cc, r);
}

// Synthetic per-step forcing (the upstream radiation / infiltration modules are out
// of scope): sabg = sabg_soil = sabg_snow = G, sabg_lyr = G on the top active layer
// and 0 elsewhere, forc_lwrad = SB*t_grnd^4, qflx_infl = I.
__global__ void __launch_bounds__(BLOCK)
k_synth_forcing(Dims D, int64_t nc, clmgb_soiltemp_fields ft, clmgb_soilwater_fields fw, const double* G,
                const double* I) {
  const int64_t c = (int64_t)blockIdx.x * BLOCK + threadIdx.x;
  if (c >= nc || !ft.mask_nolakec[c]) return;
  const double g = G[c];
  const int64_t snl = ft.col_snl[c];
  for (int64_t p1 = ft.col_patchi[c]; p1 <= ft.col_patchf[c]; p1++) {
    if (p1 < 1 || p1 > D.np) break;
    const int64_t p = p1 - 1;
    ((double*)ft.sabg)[p] = g;
    ((double*)ft.sabg_soil)[p] = g;
    ((double*)ft.sabg_snow)[p] = g;
    for (int k = 1; k <= D.nlevsno + 1; k++) LV((double*)ft.sabg_lyr, p, k, D.ldp) = 0.0;
    if (snl <= 0 && snl >= -D.nlevsno) LV((double*)ft.sabg_lyr, p, (int)snl + 1 + D.nlevsno, D.ldp) = g;
  }
  ((double*)ft.forc_lwrad)[c] = SB * jl_pow4(ft.t_grnd[c]);
  ((double*)fw.qflx_infl)[c] = I[c];
}

// ---------------------------------------------------------------------------
cudaError_t launch_water_fractions(const Dims& D, int64_t nc, const clmgb_soilwater_fields& f, cudaStream_t s) {
  k_water_fractions<<<dim3((unsigned)grid_for(nc), (unsigned)D.nlevsoi), BLOCK, 0, s>>>(D, nc, f);
  return cudaGetLastError();
}
cudaError_t launch_moisture_form(const Dims& D, int64_t nc, const clmgb_soilwater_fields& f,
                                 const clmgb_swm_config& cfg, double dtime, uint32_t* col_status,
                                 uint32_t* dev_status, cudaStream_t s) {
  k_moisture_form<<<grid_for(nc), BLOCK, 0, s>>>(D, nc, f, cfg, dtime, col_status, dev_status);
  return cudaGetLastError();
}
cudaError_t launch_column_step(const Dims& D, int64_t nc, const clmgb_soiltemp_fields& ft,
                               const clmgb_soilwater_fields& fw, const clmgb_swm_config& cfg, double dtime,
                               int snow_method, double* t_ssbef, double* t_h2osfc_bef, uint32_t* col_status,
                               uint32_t* dev_status, cudaStream_t s) {
  k_column_step<<<grid_for(nc), BLOCK, 0, s>>>(D, nc, ft, fw, cfg, dtime, snow_method, t_ssbef, t_h2osfc_bef,
                                               col_status, dev_status);
  return cudaGetLastError();
}
int queue_blocks_per_sm() {
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_moisture_form_queue<false>, BLOCK, 0) != cudaSuccess)
    nb = 1;
  return nb > 0 ? nb : 1;
}
cudaError_t launch_moisture_form_queue(const Dims& D, int64_t nc, const clmgb_soilwater_fields& f,
                                       const clmgb_swm_config& cfg, double dtime, uint32_t* col_status,
                                       int or_status, uint32_t* dev_status, unsigned long long* queue,
                                       int grid_blocks, const QueueScratch& qs, cudaStream_t s,
                                       const double* dt_init, const SubstepLogView* log) {
  cudaError_t e = cudaMemsetAsync(queue, 0, sizeof(unsigned long long), s);
  if (e != cudaSuccess) return e;
  if (log && (e = cudaMemsetAsync(log->count, 0xff, (size_t)nc * sizeof(int32_t), s)) != cudaSuccess) return e;
  const bool use = qs.capacity >= nc && qs.order && qs.bins && qs.imp;
  // the packed kernel hands no column over, so the late index that tests the hand-over's
  // bounded wait selects the per-lane kernel, which does; a limit of the polls alone has
  // nothing to act on and leaves the solve to the packed kernel (65,536 columns 1.65 ms,
  // the per-lane kernel 6.1)
  const bool packed = use && qs.packed && qs.pcache && qs.publish_delay == 0;
  if (use) {
    if (packed) {
      if ((e = launch_column_records(D, nc, f, cfg.e_ice, qs.pcache, qs.records_tma != 0,
                                     dev_status, s, qs.records_tma_used)) != cudaSuccess)
        return e;
    } else {
      k_impedance<<<grid_for(nc), BLOCK, 0, s>>>(D, nc, f, cfg.e_ice, qs.imp, qs.capacity);
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (qs.longest_first) {
      const SubstepKey key = {f.mask_hydrology, f.num_substeps, col_status, or_status};
      if ((e = launch_order(nc, key, qs.bins, qs.order, s)) != cudaSuccess) return e;
    }
  }
  const int64_t need = (nc + BLOCK - 1) / BLOCK;
  const int grid = (int)(need < grid_blocks ? need : grid_blocks);
  const bool listed = use && qs.longest_first;
  const uint32_t* ord = listed ? qs.order : nullptr;
  const unsigned int* nl = listed ? qs.bins + 2 * ORDER_BINS : nullptr;
  const double* imp = use ? qs.imp : nullptr;
  const int64_t ldi = use ? qs.capacity : 0;
  QueueScratch q = qs;
  if (!use || packed || log || !q.d_count) q.defer = 0;    // deferral needs the reserved scratch
  if (q.defer > 0) {                                       // empty list, zero claim/publish/consume counts
    if ((e = cudaMemsetAsync(q.d_count, 0, 3 * sizeof(unsigned long long), s)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(q.d_list, 0xff, (size_t)nc * sizeof(uint32_t), s)) != cudaSuccess) return e;
  }
  if (packed) {
    if ((e = launch_moisture_form_packed(D, nc, f, cfg, dtime, col_status, or_status, dev_status, queue, ord, nl,
                                         dt_init, log, grid_blocks, q, s)) != cudaSuccess)
      return e;
    // the solved columns' water, smp_l and hk_l from their records to the state
    if ((e = launch_column_outputs(D, nc, f, qs.pcache, s)) != cudaSuccess) return e;
  } else if (log)
    k_moisture_form_queue<true><<<grid > 0 ? grid : 1, BLOCK, 0, s>>>(D, nc, f, cfg, dtime, col_status, or_status,
                                                                      dev_status, queue, ord, nl, imp, ldi, dt_init,
                                                                      *log, qs.fresh_batch, q);
  else
    k_moisture_form_queue<false><<<grid > 0 ? grid : 1, BLOCK, 0, s>>>(D, nc, f, cfg, dtime, col_status, or_status,
                                                                       dev_status, queue, ord, nl, imp, ldi, dt_init,
                                                                       SubstepLogView{nullptr, nullptr, 0, 0},
                                                                       qs.fresh_batch, q);
  return cudaGetLastError();
}
cudaError_t launch_compute_qcharge(const Dims& D, int64_t nc, const clmgb_soilwater_fields& f,
                                  const clmgb_swm_config& cfg, double dtime, cudaStream_t s) {
  if (cfg.lower_boundary_condition != CLMGB_BC_WATERTABLE || nc <= 0) return cudaSuccess;
  k_compute_qcharge<<<grid_for(nc), BLOCK, 0, s>>>(D, nc, f, dtime);
  return cudaGetLastError();
}
cudaError_t launch_flexible_cn(const Dims& D, int64_t nc, const clmgb_flexcn_fields& f, cudaStream_t s) {
  k_flexible_cn<<<grid_for(nc), BLOCK, 0, s>>>(D, nc, f);
  return cudaGetLastError();
}
cudaError_t launch_math_eval(int op, int64_t n, const double* x, const double* y, double* out, cudaStream_t s) {
  k_math_eval<<<grid_for(n), BLOCK, 0, s>>>(op, n, x, y, out);
  return cudaGetLastError();
}
cudaError_t launch_phase_change(const Dims& D, int64_t nc, const clmgb_soiltemp_fields& f, double dtime,
                                const double* dhsdT, int which, cudaStream_t s) {
  k_phase_change<<<grid_for(nc), BLOCK, 0, s>>>(D, nc, f, dtime, dhsdT, which);
  return cudaGetLastError();
}
cudaError_t launch_band_solve(int64_t nc, int64_t ldc, int nlev, double* tvector, const double* bmatrix,
                              const double* rvector, const int64_t* jtop, const int64_t* jbot,
                              const uint8_t* mask, int kl, int ku, int nlevsno_off, cudaStream_t s) {
  if (kl == 2 && ku == 2)
    k_band_solve<2, 2><<<grid_for(nc), BLOCK, 0, s>>>(nc, ldc, nlev, tvector, bmatrix, rvector, jtop, jbot, mask,
                                                      nlevsno_off);
  else if (kl == 1 && ku == 1)
    k_band_solve<1, 1><<<grid_for(nc), BLOCK, 0, s>>>(nc, ldc, nlev, tvector, bmatrix, rvector, jtop, jbot, mask,
                                                      nlevsno_off);
  else
    return cudaErrorInvalidValue;
  return cudaGetLastError();
}
cudaError_t launch_tridiagonal_multi(int64_t ncols, int64_t ldc, int nlevs, double* u, const double* a,
                                     const double* b, const double* c, const double* r, const int64_t* jtop,
                                     const uint8_t* mask, cudaStream_t s, int method) {
  if (nlevs > MAXTRI) return cudaErrorInvalidValue;
  if (method == CLMGB_TRIDIAG_PCR)
    k_tridiagonal_multi_pcr<<<(unsigned)((ncols + PCR_WARPS - 1) / PCR_WARPS), 32 * PCR_WARPS, 0, s>>>(
        ncols, ldc, nlevs, u, a, b, c, r, jtop, mask);
  else {
    const int nt = BLOCK;          // 64 KB at MAXTRI levels: three blocks on an SM
    const size_t smem = (size_t)nlevs * nt * sizeof(double);
    const cudaError_t e = allow_dynamic_smem(k_tridiagonal_multi, (size_t)MAXTRI * nt * sizeof(double));
    if (e != cudaSuccess) return e;
    k_tridiagonal_multi<<<(unsigned)((ncols + nt - 1) / nt), nt, smem, s>>>(ncols, ldc, nlevs, u, a, b, c, r, jtop,
                                                                           mask);
  }
  return cudaGetLastError();
}
cudaError_t launch_synth_forcing(const Dims& D, int64_t nc, const clmgb_soiltemp_fields& ft,
                                 const clmgb_soilwater_fields& fw, const double* G, const double* I,
                                 cudaStream_t s) {
  k_synth_forcing<<<grid_for(nc), BLOCK, 0, s>>>(D, nc, ft, fw, G, I);
  return cudaGetLastError();
}

}  // namespace clmgb
