// richards_packed.cu — the work-queue Richards solve (soilwm_moisture_form_solve!,
// soil_water_movement.jl:1250-1489) with a warp's columns spread over its lanes.
//
// A warp owns up to KS = 8 columns at a time, its slots, and advances all of them by
// one substep attempt per loop trip; a slot whose column finishes takes the next column
// of the queue.  On GB300 an FP64 instruction holds its sub-partition's FP64 unit for
// about 65 cycles whatever the number of active lanes, so the work is laid out for few
// FP64 instructions and short serial chains, with few columns in the warp as well as
// with many:
//   * everything but the tridiagonal recurrences runs over (column, level) items, 32 at
//     a time: the water update and the saturations, the hydraulic properties, the fluxes
//     and their derivatives, the net fluxes (mf_refresh, after an accepted substep), the
//     matrix entries and the error estimate (mf_attempt);
//   * the forward sweep uses both half-warps: lane s carries column s's pivot
//     (gam_j = c_{j-1}/bet_{j-1}, bet_j = b_j - a_j gam_j) and lane s + 16 its
//     right-hand side one level behind (dwat_{j-1} = num_{j-1}/bet_{j-1}, num_j = r_j -
//     a_j dwat_{j-1}): the same quotient, product and difference, so a level costs one
//     division and two FP64 instructions for all the warp's columns;
//   * back substitution on the lower half-warp.
// A warp left with one long column therefore runs it at the latency of its own chain,
// and nothing is handed over between warps.
//
// The level arrays live in the warp's shared memory, [array][level][slot] with a slot
// stride of 9 doubles: items of consecutive levels and lanes of consecutive slots are
// both free of bank conflicts.  The soil parameters and the water stay in the columns'
// records (k_column_records, records.cu), which the resident columns keep in L2.
//
// Every value is formed by the reference's expression (mf_refresh, mf_attempt), so the
// results are the per-lane kernels' bits.
//
// Measured per call (scale workload, steps 5-24, ms), against the kernel with one column
// per lane and a warp-per-column finish it replaced: 61 columns 1.88 -> 0.29, 1,024 4.06
// -> 0.46, 16,384 6.27 -> 0.98, 65,536 6.90 -> 1.65, 262,144 9.94 -> 3.84.  What bounds
// it: at few columns the longest column's attempts, one after another (8 us each, half of it
// the forward sweep and the back substitution); at many the FP64 unit, and the latency of the
// divisions and powers.  Three or four level arrays in the L2-resident records instead, and
// 18 warps of 16 columns, took 3.90 ms at 262,144 columns and 1.68 at 65,536, for 27 % more
// scratch; exact quotients from 64-bit reciprocals kept there gained nothing.  The items'
// loops are not unrolled: 3.84 ms against 3.99, the code stays smaller (ncu at 262,144 columns
// with 18 warps: FP64 unit 70 % busy, issue slots 44 %, instruction fetch 1.7 of 9.8 cycles
// a warp waits per instruction).
#include "clmgb_device.cuh"
#include "launch.h"

namespace clmgb {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int KS = 8, SLD = KS + 1, HALF = 16;     // slots, their stride, lanes of a half-warp
// Up to FEW_SLOTS columns for each of FEW_WARPS warps a block the variant with an attempt's
// quotients and powers in line runs (FEW): a warp waits for its own chain, and independent
// ones overlap.  ms a call in line / through the shared functions with MANY_WARPS, scale
// workload: 61 columns 0.250 / 0.266, 1,024 0.457 / 0.480, 4,000 0.635 / 0.666, 8,000 0.800 /
// 0.825, 12,000 0.790 / 0.822; with warps in different phases the code is no longer found in
// the instruction cache: 16,000 1.003 / 0.995, 24,000 1.06 / 1.03, 65,536 1.83 / 1.57, 262,144
// 5.56 / 3.79.
constexpr int FEW_SLOTS = 8, FEW_WARPS = 5;
// Many columns: 2 blocks, 18 warps of 8 columns and 20 levels, in an SM's shared memory.  ms a
// call at 65,536 / 262,144 columns of the scale workload and at 262,144 of the snow workload:
// 16 columns and 10 warps 1.72 / 4.27 / 1.65, 12 and 12 1.65 / 4.15 / 1.57, 10 and 14 1.65 /
// 4.14 / 1.55, 8 and 18 1.65 / 4.03 / 1.42.  With 22 to 25 levels, or 20 and the expensive flux
// estimate, one such block fits: 25 levels 2.4 / 7.2 ms, the expensive estimate 2.1 / 6.1 (the
// kernel with a column per lane 6.4 / 18.7 and 5.6 / 12.8).
constexpr int MANY_WARPS = 9;

// level arrays: the flux derivatives dqodw1, dqodw2 and the net flux (kept from a
// refresh to the next), dt_dz, and four that the sweeps of an attempt and the passes of a
// refresh use in turn; the outflow, which only the expensive flux estimate reads again
enum LevelArray { LA_D1 = 0, LA_D2, LA_FN, LA_DT, LA_A, LA_B, LA_C, LA_R, LA_Q };

// per-slot values the items read
struct SlotArea {
  double dt[KS], dtc[KS];               // this attempt's substep; the one dt_dz was formed for
  double qb[KS], hb[KS], db[KS];        // bottom level: outflow, conductivity and its derivative
  int64_t c[KS];
  int nl[KS];
  int bad[KS];                          // a level's water is not finite
  int nacc[KS];                         // substep log: records written
  uint8_t list[KS];
};

__host__ __device__ constexpr int64_t level_doubles(int nls, bool expensive) {
  return (int64_t)(expensive ? 9 : 8) * nls * SLD;
}
__host__ __device__ constexpr int64_t warp_bytes(int nls, bool expensive) {
  return level_doubles(nls, expensive) * 8 + (int64_t)((sizeof(SlotArea) + 15) / 16 * 16);
}

// A quotient of a group: with FEW in line and without a branch, so that independent ones
// overlap (ok turns false where the group has to be formed again by jl_div); else jl_div.
template <bool FEW>
__device__ __forceinline__ double quotient(double x, double y, bool& ok) {
  if (!FEW) return jl_div(x, y);
  bool o;
  const double q = cm_div_fx(x, y, &o);
  ok = ok & o;
  return q;
}
// both powers of an item: with FEW in line, beside each other
template <bool FEW>
__device__ __forceinline__ void power_pair(double x1, double y1, double x2, double y2, double& p1, double& p2) {
  if (FEW) {
    const bool o1 = cm_pow_fx(x1, y1, &p1), o2 = cm_pow_fx(x2, y2, &p2);
    if (!o1) p1 = cm_pow_dd_call_(x1, y1);
    if (!o2) p2 = cm_pow_dd_call_(x2, y2);
  } else {
    p1 = cm_pow(x1, y1);
    p2 = cm_pow(x2, y2);
  }
}

// FEW: for warps of few columns, whose attempts wait for their own quotients and powers
template <bool LOG, bool EXPENSIVE, bool FEW>
__global__ void __launch_bounds__(32 * (FEW ? FEW_WARPS : MANY_WARPS), 2)
k_moisture_form_packed(Dims D, int64_t nc, clmgb_soilwater_fields f, clmgb_swm_config cfg, double dtime,
                       uint32_t* col_status, int or_status, uint32_t* dev_status, unsigned long long* queue,
                       const uint32_t* order, const unsigned int* nlisted_ptr, const double* dt_init,
                       SubstepLogView lg, int kslots, QueueScratch qs) {
  extern __shared__ __align__(16) unsigned char smem_packed[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int nls = D.nlevsoi, stride = PC_ALL * nls;
  double* const lev = reinterpret_cast<double*>(smem_packed + wib * warp_bytes(nls, EXPENSIVE));
  SlotArea& SA = *reinterpret_cast<SlotArea*>(lev + level_doubles(nls, EXPENSIVE));
  double* const pcache = qs.pcache;
  const int lower_bc = cfg.lower_boundary_condition;
  const unsigned long long nq = order ? (unsigned long long)(*(volatile const unsigned int*)nlisted_ptr)
                                      : (unsigned long long)nc;
  const unsigned long long nwarps = (unsigned long long)gridDim.x * (FEW ? FEW_WARPS : MANY_WARPS);
  const uint32_t magic = 65536u / (uint32_t)nls + 1u;       // t / nls for t < KS * 25
  // the tolerances as keys of non-negative doubles: e > upper and e < lower for e >= 0
  const long long key_up = cfg.xTolerUpper != cfg.xTolerUpper ? 0x7fffffffffffffffLL
                           : cfg.xTolerUpper < 0.0            ? -1LL
                                                              : (dbits(cfg.xTolerUpper) & 0x7fffffffffffffffLL);
  const long long key_lo = cfg.xTolerLower > 0.0 ? dbits(cfg.xTolerLower) : 0LL;
  auto A = [&](int a, int j, int s) -> double& { return lev[(a * nls + (j - 1)) * SLD + s]; };

  // the (column, level) items of the slots in a mask, 32 at a time
  struct Item { int s, j, nl; bool ok; };
  auto list_slots = [&](unsigned mask) -> int {
    __syncwarp();
    if (lane < KS && ((mask >> lane) & 1u)) SA.list[__popc(mask & ((1u << lane) - 1u))] = (uint8_t)lane;
    __syncwarp();
    return __popc(mask) * nls;
  };
  auto item = [&](int t, int T) -> Item {
    Item it;
    const int q = (int)(((uint32_t)t * magic) >> 16);
    it.ok = t < T;
    it.s = it.ok ? SA.list[q] : 0;
    it.j = t - q * nls + 1;
    it.nl = SA.nl[it.s];
    it.ok = it.ok && it.j <= it.nl;
    return it;
  };

  // the slot of lanes 0..KS-1
  int64_t c = 0;
  int n = 0, nsub = 0, nacc = 0;
  bool active = false, fresh = false, first = true;
  bool exhausted = lane >= kslots;
  uint32_t status = 0;
  double dtsub = 0.0, dtdone = 0.0, qc = 0.0;

  // The water of the slots in `mask`: the accepted substep's update where `upd` is set,
  // then the saturation of each level (:1283-1287, kept in LA_A) unless the column is
  // `done`.  With LOG the water is also written to the column's next record, or, when
  // done, with the other outputs behind the records.
  auto water_pass = [&](unsigned mask, unsigned upd, unsigned done) {
    const int T = list_slots(mask);
#pragma unroll 1
    for (int t0 = 0; t0 < T; t0 += 32) {
      const Item it = item(t0 + lane, T);
      if (!it.ok) continue;
      const int64_t cc = SA.c[it.s];
      double* rec = pcache + cc * (int64_t)stride + (it.j - 1);
      const double dzw = rec[PC_DZW * nls], ws = rec[PC_WS * nls];
      double liq = rec[PC_LIQ * nls];
      if ((upd >> it.s) & 1u) {
        liq = liq + A(LA_R, it.j, it.s) * dzw;
        rec[PC_LIQ * nls] = liq;
      }
      const bool dn = (done >> it.s) & 1u;
      if (LOG) {
        double* lrec = lg.rec + cc * lg.stride;
        if (dn) {
          double* out = lrec + (int64_t)lg.cap * SUB_REC + (it.j - 1);
          out[0] = liq;
          out[MAXSOI] = rec[PC_SMP * nls];
          out[2 * MAXSOI] = rec[PC_HK * nls];
        } else if (SA.nacc[it.s] < lg.cap) {
          lrec[(int64_t)SA.nacc[it.s] * SUB_REC + it.j - 1] = liq;
        }
      }
      if (dn) {
        if (!finite_bits(liq)) SA.bad[it.s] = 1;
      } else {
        const double lm = jl_max(liq, 1.0e-6);
        bool ok = true;
        double s = quotient<FEW>(quotient<FEW>(lm, dzw, ok), ws, ok);
        if (FEW && !ok) s = jl_div(jl_div(lm, dzw), ws);
        s = jl_min(s, 1.0);
        A(LA_A, it.j, it.s) = jl_max(0.01, s);
      }
    }
    __syncwarp();
  };
  // mf_end for the lanes whose slot is done (after water_pass)
  auto finish = [&](bool dn) {
    if (dn) {
      if (SA.bad[lane]) status |= CLMGB_COL_NONFINITE;
      f.qcharge[c] = qc;
      f.num_substeps[c] = (double)nsub;
      if (LOG) {
        double* out = lg.rec + c * lg.stride + (int64_t)lg.cap * SUB_REC;
        out[3 * MAXSOI] = qc;
        out[3 * MAXSOI + 1] = (double)nsub;
        out[3 * MAXSOI + 2] = (double)status;
        lg.count[c] = nacc;
      }
      if (col_status) col_status[c] = or_status ? (col_status[c] | status) : status;
      if (status && dev_status) atomicOr(dev_status, status);
      active = false;
    }
  };

  for (;;) {
    // ---- new columns for the empty slots ----
    const bool need = !active && !exhausted;
    const unsigned m = __ballot_sync(FULL, need);
    bool began = false;
    if (m) {
      unsigned long long k;
      if (first) {
        // slot s of warp w starts with column s * nwarps + w of the order: the longest
        // expected columns are spread over all warps, neighbours over all SMs
        k = (unsigned long long)lane * nwarps + (unsigned long long)wib * gridDim.x + blockIdx.x;
      } else {
        const int leader = __ffs(m) - 1;
        unsigned long long base = 0;
        if (lane == leader) base = atomicAdd(queue, (unsigned long long)__popc(m));
        base = __shfl_sync(FULL, base, leader);
        k = (unsigned long long)kslots * nwarps + base + (unsigned long long)__popc(m & ((1u << lane) - 1u));
      }
      if (need) {
        if (k >= nq) {
          exhausted = true;
        } else {
          c = order ? (int64_t)order[k] : (int64_t)k;
          if (order || f.mask_hydrology[c]) {
            const int64_t nl = f.col_nbedrock[c];
            if (nl >= 1 && nl <= nls) {
              n = (int)nl;
              nsub = 0;
              nacc = 0;
              status = 0;
              dtsub = dtime;
              if (dt_init) {
                const double d = dt_init[c];
                if (d == d) dtsub = jl_min(jl_max(d, cfg.dtmin), dtime);   // NaN keeps dtime
              }
              dtdone = 0.0;
              qc = 0.0;
              active = fresh = began = true;
              SA.c[lane] = c;
              SA.nl[lane] = n;
              SA.dtc[lane] = -1.0;
              SA.bad[lane] = 0;
              SA.nacc[lane] = 0;
            } else {
              const uint32_t st = CLMGB_COL_LEVEL_RANGE;
              if (col_status) col_status[c] = or_status ? (col_status[c] | st) : st;
              if (dev_status) atomicOr(dev_status, st);
            }
          } else if (col_status && !or_status) {
            col_status[c] = 0;
          }
        }
      }
      first = false;
      const unsigned bm = __ballot_sync(FULL, began);
      if (bm) water_pass(bm, 0u, 0u);
    }
    if (!__any_sync(FULL, active)) {
      if (__all_sync(FULL, exhausted)) break;
      continue;
    }
    // ---- columns that have used up their attempts ----
    const bool capped = active && nsub >= D.attempt_cap;
    const unsigned cm = __ballot_sync(FULL, capped);
    if (cm) {
      if (capped) {
        nsub += 1;
        status |= CLMGB_COL_SUBSTEP_CAP;
      }
      water_pass(cm, 0u, cm);
      finish(capped);
    }
    const unsigned am = __ballot_sync(FULL, active);
    if (!am) continue;
    // ---- refresh (mf_refresh, :1280-1378) of the columns with a new water state ----
    const unsigned fm = __ballot_sync(FULL, active && fresh);
    if (qs.work) {
      const unsigned la = __reduce_add_sync(FULL, active ? (unsigned)n : 0u);
      const unsigned lf = __reduce_add_sync(FULL, active && fresh ? (unsigned)n : 0u);
      if (lane == 0) {
        atomicAdd(qs.work, (unsigned long long)la);
        atomicAdd(qs.work + 1, (unsigned long long)lf);
      }
    }
    if (fm) {
      const int T = list_slots(fm);
      // hydraulic properties (:1288-1308): hk, dhkdw, smp, dsmpdw into LA_B, LA_C, LA_R, LA_FN
#pragma unroll 1
      for (int t0 = 0; t0 < T; t0 += 32) {
        const Item it = item(t0 + lane, T);
        if (it.ok) {
          const int j = it.j, s = it.s;
          double* rec = pcache + SA.c[s] * (int64_t)stride + (j - 1);
          const double b = rec[PC_BSW * nls], e = rec[PC_EXP * nls], ik = rec[PC_IK * nls];
          const double suc = rec[PC_SUC * nls], ws = rec[PC_WS * nls];
          const double sj = A(LA_A, j, s);
          double s1 = sj;
          if (j != it.nl) s1 = half_of(sj + A(LA_A, j + 1, s));
          s1 = jl_min(s1, 1.0);
          s1 = jl_max(0.01, s1);
          double p1, p2;
          power_pair<FEW>(s1, e, sj, -b, p1, p2);
          const double hkv = ik * p1;
          const double smpv = -suc * p2;
          A(LA_B, j, s) = hkv;
          A(LA_R, j, s) = smpv;
          bool ok = true;
          double dhk = quotient<FEW>(e * hkv, s1, ok), dsmp = quotient<FEW>(quotient<FEW>(-b * smpv, sj, ok), ws, ok);
          if (FEW && !ok) {
            dhk = jl_div(e * hkv, s1);
            dsmp = jl_div(jl_div(-b * smpv, sj), ws);
          }
          A(LA_C, j, s) = dhk;
          A(LA_FN, j, s) = dsmp;
          rec[PC_SMP * nls] = smpv;
          rec[PC_HK * nls] = hkv;
        }
      }
      __syncwarp();
      // fluxes and derivatives between levels (:1310-1345) and at the bottom (:1347-1370)
      constexpr int QO = EXPENSIVE ? LA_Q : LA_A;
#pragma unroll 1
      for (int t0 = 0; t0 < T; t0 += 32) {
        const Item it = item(t0 + lane, T);
        if (it.ok) {
          const int j = it.j, s = it.s;
          const int64_t cc = SA.c[s];
          const double* rec = pcache + cc * (int64_t)stride + (j - 1);
          const double hk = A(LA_B, j, s), dhkdw = A(LA_C, j, s), smp = A(LA_R, j, s), dsmpdw = A(LA_FN, j, s);
          const double ws = rec[PC_WS * nls];
          double qo = 0.0, d1 = 0.0, d2 = 0.0;
          if (j < it.nl) {
            const double hd = half_of(dhkdw);
            const double wsn = rec[PC_WS * nls + 1], den = rec[PC_DEN * nls];
            const double num = A(LA_R, j + 1, s) - smp;
            bool ok = true;
            double dhkds1 = quotient<FEW>(hd, ws, ok), dhkds2 = quotient<FEW>(hd, wsn, ok);
            qo = quotient<FEW>(-hk * num, den, ok) + hk;
            d1 = quotient<FEW>(hk * dsmpdw - dhkds1 * num, den, ok) + dhkds1;
            d2 = quotient<FEW>(-hk * A(LA_FN, j + 1, s) - dhkds2 * num, den, ok) + dhkds2;
            if (FEW && !ok) {
              dhkds1 = jl_div(hd, ws);
              dhkds2 = jl_div(hd, wsn);
              qo = jl_div(-hk * num, den) + hk;
              d1 = jl_div(hk * dsmpdw - dhkds1 * num, den) + dhkds1;
              d2 = jl_div(-hk * A(LA_FN, j + 1, s) - dhkds2 * num, den) + dhkds2;
            }
          } else {
            if (lower_bc == CLMGB_BC_WATERTABLE) {
              int jwt = nls;
              for (int jj = 1; jj <= nls; jj++) {
                if (f.zwt[cc] <= LVc(f.zi, cc, D.nlevsno + 1 + jj, D.ldc)) { jwt = jj - 1; break; }
              }
              if (j <= jwt) {
                const double dhkds1l = jl_div(dhkdw, ws);
                const double num = -smp;
                const double den = M_TO_MM * (f.zwt[cc] - LVc(f.z, cc, D.nlevsno + j, D.ldc));
                qo = jl_div(-hk * num, den) + hk;
                d1 = jl_div(hk * dsmpdw - dhkds1l * num, den) + dhkds1l;
              }
            } else if (lower_bc == CLMGB_BC_FLUX) {
              qo = hk;
              d1 = jl_div(dhkdw, ws);
            }
            SA.qb[s] = qo;
            SA.hb[s] = hk;
            SA.db[s] = dhkdw;
          }
          A(QO, j, s) = qo;
          A(LA_D1, j, s) = d1;
          A(LA_D2, j, s) = d2;
        }
      }
      __syncwarp();
      // net flux (:1372-1378); the inflow of level j > 1 is the outflow of level j-1
#pragma unroll 1
      for (int t0 = 0; t0 < T; t0 += 32) {
        const Item it = item(t0 + lane, T);
        if (it.ok) {
          const int64_t cc = SA.c[it.s];
          const double root = pcache[cc * (int64_t)stride + PC_ROOT * nls + (it.j - 1)];
          const double qin = it.j == 1 ? f.qflx_infl[cc] : A(QO, it.j - 1, it.s);
          A(LA_FN, it.j, it.s) = qin - A(QO, it.j, it.s) - root;
        }
      }
      fresh = false;
    }
    if (active) {
      nsub += 1;
      SA.dt[lane] = dtsub;
    }
    // ---- dt_dz and the matrix (:1380-1397) ----
    const int T = list_slots(am);
#pragma unroll 1
    for (int t0 = 0; t0 < T; t0 += 32) {
      const Item it = item(t0 + lane, T);
      if (it.ok) {
        const int j = it.j, s = it.s;
        const long long bd = dbits(SA.dt[s]), bc = dbits(SA.dtc[s]);
        double dt = A(LA_DT, j, s);
        if (bd != bc) {
          // a power of two times the previous substep scales the quotient by the same
          // power: through its exponent
          const long long v = dbits(dt);
          const int ed = (int)((bd >> 52) & 0x7ff), ec = (int)((bc >> 52) & 0x7ff), ev = (int)((v >> 52) & 0x7ff);
          if (bc > 0 && ((bd ^ bc) & 0x000fffffffffffffLL) == 0 && ed > 0 && ec > 0 && ed < 2047 && ec < 2047 &&
              ev > 0 && ev + (ed - ec) > 0 && ev + (ed - ec) < 2047)
            dt = __longlong_as_double(v + ((long long)(ed - ec) << 52));
          else
            dt = jl_div(SA.dt[s], pcache[SA.c[s] * (int64_t)stride + PC_DZW * nls + (j - 1)]);
          A(LA_DT, j, s) = dt;
        }
        const double d1 = A(LA_D1, j, s), d2 = A(LA_D2, j, s);
        double d1p = 0.0, x = d1;
        if (j > 1) {
          d1p = A(LA_D1, j - 1, s);
          x = d1 - A(LA_D2, j - 1, s);
        }
        A(LA_A, j, s) = d1p * dt;
        A(LA_B, j, s) = -1.0 - x * dt;
        A(LA_C, j, s) = j == it.nl ? 0.0 : -d2 * dt;
        A(LA_R, j, s) = -A(LA_FN, j, s) * dt;
      }
    }
    __syncwarp();
    // ---- Thomas forward sweep (:1421-1438) ----
    const int s = lane & (HALF - 1);                        // lanes of no slot have no levels
    const bool up = lane >= HALF;
    const int ns = ((am >> s) & 1u) ? SA.nl[s] : 0;
    const int nmax = (int)__reduce_max_sync(FULL, (unsigned)ns);
    {
      double bet = 1.0, num = 1.0, u = 1.0;
      if (ns) {
        bet = A(LA_B, 1, s);
        if (abs_lt(bet, 1.0e-30)) bet = 1.0e-30;
        num = A(LA_R, 1, s);
        u = up ? num : A(LA_C, 1, s);
      }
      for (int j = 2; j <= nmax + 1; j++) {
        double a = 0.0, w = 1.0, cn = 1.0;
        if (j <= ns) {
          a = A(LA_A, j, s);
          w = up ? A(LA_R, j, s) : A(LA_B, j, s);
          cn = A(LA_C, j, s);
        }
        const double q = div_chain(u, __shfl_sync(FULL, bet, s));
        const double v = w - a * q;
        if (j <= ns + 1 && ns) A(up ? LA_R : LA_C, j - 1, s) = q;     // dwat of level j-1, gam of level j
        if (j <= ns) {
          if (up) {
            u = v;
          } else {
            bet = v;
            if (abs_lt(bet, 1.0e-30)) bet = copysign(1.0e-30, bet == 0.0 ? 1.0 : bet);
            u = cn;
          }
        } else {
          u = 1.0;
          bet = 1.0;
        }
      }
    }
    __syncwarp();
    // ---- back substitution ----
    if (!up) {
      double x = ns ? A(LA_R, ns, s) : 0.0;
      for (int j = nmax - 1; j >= 1; j--) {
        if (j < ns) {
          x = A(LA_R, j, s) - A(LA_C, j, s) * x;
          A(LA_R, j, s) = x;
        }
      }
    }
    __syncwarp();
    // ---- error estimate (:1440-1457): per column, whether a level's error is above the
    // upper tolerance, not below the lower one, or NaN (which the maximum would be) ----
    bool e_up = false, e_nlo = false, e_nan = false;
    const int own0 = __popc(am & ((1u << lane) - 1u)) * nls;         // this slot's first item
#pragma unroll 1
    for (int t0 = 0; t0 < T; t0 += 32) {
      const Item it = item(t0 + lane, T);
      bool fu = false, fl = false, fn = false;
      if (it.ok) {
        const int j = it.j, si = it.s;
        const double dw = A(LA_R, j, si), fnet1 = A(LA_FN, j, si);
        double fnet0;
        if (EXPENSIVE) {
          const int64_t cc = SA.c[si];
          const double qin_test = j == 1 ? f.qflx_infl[cc] + 0.0 * dw
                                         : A(LA_Q, j - 1, si) + A(LA_D1, j - 1, si) * A(LA_R, j - 1, si) +
                                               A(LA_D2, j - 1, si) * dw;
          const double qout_test = j == it.nl ? A(LA_Q, j, si) + A(LA_D1, j, si) * dw
                                              : A(LA_Q, j, si) + A(LA_D1, j, si) * dw +
                                                    A(LA_D2, j, si) * A(LA_R, j + 1, si);
          fnet0 = qin_test - qout_test - pcache[cc * (int64_t)stride + PC_ROOT * nls + (j - 1)];
        } else {
          fnet0 = FEW ? div_chain(dw, A(LA_DT, j, si)) : jl_div(dw, A(LA_DT, j, si));
        }
        const long long ev = dbits(half_of(fabs(fnet1 - fnet0) * SA.dt[si])) & 0x7fffffffffffffffLL;
        fn = ev > 0x7ff0000000000000LL;
        fu = ev > key_up;
        fl = !(ev < key_lo);
      }
      const unsigned bu = __ballot_sync(FULL, fu), bl = __ballot_sync(FULL, fl), bn = __ballot_sync(FULL, fn);
      const int lo = own0 - t0, hi = lo + nls;                        // this slot's items: lanes lo..hi-1
      if (hi > 0 && lo < 32) {
        const unsigned mk = (hi >= 32 ? FULL : (1u << hi) - 1u) & (lo > 0 ? FULL << lo : FULL);
        e_up |= (bu & mk) != 0;
        e_nlo |= (bl & mk) != 0;
        e_nan |= (bn & mk) != 0;
      }
    }
    // ---- accept or reject (:1460-1483) ----
    bool acc = false, done = false;
    if (active) {
      SA.dtc[lane] = dtsub;
      if (e_up && !e_nan && dbits(dtsub) > dbits(cfg.dtmin)) {
        dtsub = jl_max(half_of(dtsub), cfg.dtmin);
      } else {
        acc = fresh = true;
        double qcTemp;
        const double dwn = A(LA_R, n, lane);
        if (lower_bc == CLMGB_BC_FLUX) qcTemp = SA.hb[lane] + SA.db[lane] * dwn;
        else if (lower_bc == CLMGB_BC_ZERO_FLUX) qcTemp = 0.0;
        else qcTemp = SA.qb[lane] + A(LA_D1, n, lane) * dwn;
        qc += qcTemp * jl_div(dtsub, dtime);
        if (LOG) {
          if (nacc < lg.cap) {
            double* lrec = lg.rec + c * lg.stride + (int64_t)nacc * SUB_REC;
            lrec[MAXSOI] = dtsub;
            lrec[MAXSOI + 1] = dtdone;
          }
          nacc++;
          SA.nacc[lane] = nacc;
        }
        dtdone += dtsub;
        const double left = dtime - dtdone;
        done = fabs(left) < cfg.verySmall;
        if (!done) {
          double nd = dtsub;
          if (!e_nlo) nd = dtsub * 2.0;
          dtsub = jl_min(nd, left);
        }
      }
    }
    const unsigned um = __ballot_sync(FULL, acc), dm = __ballot_sync(FULL, done);
    if (um) water_pass(um, um, dm);
    if (dm) finish(done);
  }
}

}  // namespace

cudaError_t launch_moisture_form_packed(const Dims& D, int64_t nc, const clmgb_soilwater_fields& f,
                                        const clmgb_swm_config& cfg, double dtime, uint32_t* col_status, int or_status,
                                        uint32_t* dev_status, unsigned long long* queue, const uint32_t* order,
                                        const unsigned int* nlisted, const double* dt_init, const SubstepLogView* log,
                                        int max_blocks, const QueueScratch& qs, cudaStream_t s) {
  const bool expensive = cfg.flux_calculation == 42;
  int dev = 0, nsm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  const bool few = !expensive && nc <= (int64_t)2 * nsm * FEW_WARPS * FEW_SLOTS;
  const int warps = few ? FEW_WARPS : MANY_WARPS;
  const size_t smem = (size_t)warps * (size_t)warp_bytes(D.nlevsoi, expensive);
  auto kern = log ? (few         ? k_moisture_form_packed<true, false, true>
                     : expensive ? k_moisture_form_packed<true, true, false>
                                 : k_moisture_form_packed<true, false, false>)
                  : (few         ? k_moisture_form_packed<false, false, true>
                     : expensive ? k_moisture_form_packed<false, true, false>
                                 : k_moisture_form_packed<false, false, false>);
  if ((e = allow_dynamic_smem(kern, (size_t)warps * (size_t)warp_bytes(MAXSOI, expensive))) != cudaSuccess) return e;
  int nb = 0;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, 32 * warps, smem)) != cudaSuccess) return e;
  if (nb < 1) return cudaErrorInvalidConfiguration;
  int64_t grid = (int64_t)nb * nsm;
  if (grid > max_blocks) grid = max_blocks > 0 ? max_blocks : 1;
  // as few columns per warp as the resident warps allow: a column alone in its warp
  // finishes soonest, and at most KS share one
  int64_t kslots = (nc + grid * warps - 1) / (grid * warps);
  if (kslots > KS) kslots = KS;
  if (kslots < 1) kslots = 1;
  kern<<<(unsigned)grid, 32 * warps, smem, s>>>(D, nc, f, cfg, dtime, col_status, or_status, dev_status, queue, order,
                                                nlisted, dt_init, log ? *log : SubstepLogView{nullptr, nullptr, 0, 0},
                                                (int)kslots, qs);
  return cudaGetLastError();
}

}  // namespace clmgb
