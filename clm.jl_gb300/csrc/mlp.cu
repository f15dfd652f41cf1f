// mlp.cu — the learned warm start of the moisture-form Richards solve.
//
// A 64 -> 128 -> 128 -> 21 multilayer perceptron (SiLU hidden layers, BF16 weights
// and activations, FP32 accumulation) proposes, for a column about to start a
// substep, how many times the remaining time must be halved before the solver's
// error test accepts the substep (output 0), together with the saturation increment
// of that substep on each of the 20 soil levels (outputs 1..20).  The solver takes
// the proposal as the size of its first attempt; its own accept/reject test
// (soil_water_movement.jl:1460-1463) still judges it and halves it if needed, so a
// result meets the same tolerance with or without the network.
//
// Kernels:
//   k_richards_samples    the plain solver, recording training pairs at the first R
//                         substep starts of every column: features, and the label
//                         found by trial attempts at remaining/2^k, k = 0, 1, ...
// The passes over all layers are in mlp_fused.cu; the per-layer kernels here serve the
// per-layer entry points.
//   k_linear<K, N>        Y = act(X W^T + b) with mma.sync m16n8k16 (bf16 x bf16 ->
//                         fp32); one warp owns 16 rows and all N outputs
//   k_linear_dw<N, K>     dW += dZ^T X, db += sum dZ over a chunk of rows (CUDA cores,
//                         fp32 accumulation, one atomic add per element per chunk)
//   k_silu_backward, k_mlp_loss, k_adam
//   k_mlp_features        the 64 inputs of every column at the start of a call
//   k_mlp_first_dt        proposal -> first substep size
#include <cuda_bf16.h>
#include "clmgb_device.cuh"
#include "launch.h"

namespace clmgb {

constexpr int MLP_IN = 64, MLP_HID = 128, MLP_OUT = 21, MLP_OUTP = 32;
constexpr int FEAT_LEVELS = 20;

__device__ __forceinline__ float silu(float z) { return z / (1.0f + expf(-z)); }

// ---------------------------------------------------------------------------
// Features of a column about to start a substep, in single precision (they are
// inputs to the network, not part of the solve):
//   0..19  saturation liq / (1000 dz watsat) of soil levels 1..20 (0 below the column)
//   20..39 ice fraction of the level (icefrac, set by set_soil_water_fractions!)
//   40..59 log10 of the hydraulic conductivity (mm/s): log10 ksat + (2b+3) log10 s1
//          - e_ice icefrac_interface, the logarithm of imp * ksat * s1^(2b+3)
//   60     infiltration into the top layer (1e3 mm/s units)
//   61     total transpiration sink (1e3 mm/s units)
//   62     remaining time of the step / dtime
//   63     log2(dtime / 60 s) / 6
// liq(j) gives the liquid water of soil level j.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float feature_saturation(double liq, double dz, double watsat) {
  return (float)liq / (1000.0f * (float)dz * (float)watsat);
}

// s, ice: the level's saturation and ice fraction; below, ice_below: those of the next
// level, not used at the lowest one
__device__ __forceinline__ float feature_log_conductivity(bool lowest, float s, float below, double ice,
                                                          double ice_below, double bsw, double hksat, float e_ice) {
  float s1 = lowest ? s : 0.5f * (s + below);
  s1 = fminf(fmaxf(s1, 0.01f), 1.0f);
  const float fi = lowest ? (float)ice : 0.5f * (float)(ice + ice_below);
  return log10f((float)hksat) + (2.0f * (float)bsw + 3.0f) * log10f(s1) - e_ice * fi;
}

template <class LiqF>
__device__ __forceinline__ void column_features(const Dims& D, const clmgb_soilwater_fields& f,
                                                const clmgb_swm_config& cfg, int64_t c, int nlayers, LiqF liq,
                                                double rem, double dtime, float* x) {
  const int64_t ld = D.ldc;
  float s[FEAT_LEVELS + 2] = {};
  float sink = 0.0f;
  for (int j = 1; j <= FEAT_LEVELS; j++) {
    const bool in = j <= nlayers;
    float sv = 0.0f;
    if (in) {
      sv = feature_saturation(liq(j), LVc(f.dz, c, D.nlevsno + j, ld), LVc(f.watsat, c, j, ld));
      sink += (float)LVc(f.qflx_rootsoi, c, j, ld);
    }
    s[j] = sv;
    x[j - 1] = sv;
    x[19 + j] = in ? (float)LV(f.icefrac, c, j, ld) : 0.0f;
  }
  constexpr int next = FEAT_LEVELS + 1;               // below the last level of the features
  if (nlayers >= next)
    s[next] = feature_saturation(liq(next), LVc(f.dz, c, D.nlevsno + next, ld), LVc(f.watsat, c, next, ld));
  for (int j = 1; j <= FEAT_LEVELS; j++)
    x[39 + j] = j > nlayers ? -30.0f
                            : feature_log_conductivity(j == nlayers, s[j], s[j + 1], LV(f.icefrac, c, j, ld),
                                                       j == nlayers ? 0.0 : LV(f.icefrac, c, j + 1, ld),
                                                       LVc(f.bsw, c, j, ld), LVc(f.hksat, c, j, ld), (float)cfg.e_ice);
  x[60] = (float)(f.qflx_infl[c] * 1.0e3);
  x[61] = sink * 1.0e3f;
  x[62] = (float)(rem / dtime);
  x[63] = log2f((float)(dtime / 60.0)) / 6.0f;
}

// The plain solve of one column, recording up to rmax training pairs (one per
// substep start).  The label of a substep start is the smallest k for which an
// attempt at remaining/2^k (at least dtmin) is accepted; the trials run on a copy of
// the lane and do not change the solve.
__global__ void __launch_bounds__(64)
k_richards_samples(Dims D, int64_t nc, clmgb_soilwater_fields f, clmgb_swm_config cfg, double dtime, int rmax,
                   float* feat, float* targ, unsigned int* count, int64_t capacity, uint32_t* col_status) {
  const int64_t c = (int64_t)blockIdx.x * 64 + threadIdx.x;
  if (c >= nc) return;
  if (!f.mask_hydrology[c]) return;
  MfLane L;
  if (!mf_begin(L, D, f, cfg, dtime, c)) {
    if (col_status) col_status[c] |= L.status;
    return;
  }
  const int64_t ld = D.ldc;
  int recorded = 0;
  bool done = false;
  while (!done) {
    if (L.fresh && recorded < rmax) {
      const double rem = dtime - L.dtdone;
      float x[MLP_IN];
      column_features(D, f, cfg, c, L.nlayers, [&](int j) { return L.liq[j]; }, rem, dtime, x);
      int k = 0;
      double incr[MAXSOI + 1];
      for (;; k++) {
        MfLane T = L;
        double dt = rem;
        for (int i = 0; i < k; i++) dt = jl_max(dt / 2.0, cfg.dtmin);
        T.dtsub = dt;
        const double before = T.dtdone;
        FieldState<clmgb_soilwater_fields> XT(f, c, ld);
        mf_attempt(T, D, f, cfg, dtime, XT);
        if (T.dtdone != before || dt <= cfg.dtmin || k >= 12) {
          for (int j = 1; j <= L.nlayers; j++)
            incr[j] = (T.liq[j] - L.liq[j]) / (M_TO_MM * L.dzv[j] * LVc(f.watsat, c, j, ld));
          break;
        }
      }
      const unsigned int slot = atomicAdd(count, 1u);
      if (slot < capacity) {
        for (int i = 0; i < MLP_IN; i++) feat[(int64_t)slot * MLP_IN + i] = x[i];
        float* t = targ + (int64_t)slot * MLP_OUTP;
        t[0] = (float)k;
        for (int j = 1; j <= FEAT_LEVELS; j++) t[j] = j <= L.nlayers ? (float)incr[j] : 0.0f;
        for (int j = FEAT_LEVELS + 1; j < MLP_OUTP; j++) t[j] = 0.0f;
      }
      recorded++;
    }
    FieldState<clmgb_soilwater_fields> X(f, c, ld);
    done = mf_attempt(L, D, f, cfg, dtime, X);
  }
  FieldState<clmgb_soilwater_fields> X(f, c, ld);
  const uint32_t st = mf_end(L, D, f, X);
  if (col_status) col_status[c] |= st;
}

// ---------------------------------------------------------------------------
// Y = act(X W^T + b): X [M x K] bf16 (row stride ldx), W [N x K] bf16, b [N] fp32;
// Z [M x N] fp32 pre-activation (optional), Y [M x N] bf16 (optional, row stride
// ldy).  64 rows per block of 4 warps.  mma.sync m16n8k16 fragments (PTX ISA):
// with g = lane/4 and t = lane%4, A regs hold rows g and g+8 at columns 2t, 2t+1
// and 2t+8, 2t+9; B regs hold columns 2t, 2t+1 and 2t+8, 2t+9 of row g of W (one
// output); C holds rows g, g+8 at outputs 2t, 2t+1.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void mma_bf16(float* d, const uint32_t* a, const uint32_t* b) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

template <int K, int N>
__global__ void __launch_bounds__(128)
k_linear(int64_t M, const __nv_bfloat16* __restrict__ X, int64_t ldx, const __nv_bfloat16* __restrict__ W,
         const float* __restrict__ bias, int act, float* Z, int64_t ldz, __nv_bfloat16* Y, int64_t ldy) {
  constexpr int KP = K + 8;   // padded smem row (bank spread)
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __nv_bfloat16* sW = (__nv_bfloat16*)smem_raw;
  __nv_bfloat16* sX = sW + N * KP;
  const int64_t row0 = (int64_t)blockIdx.x * 64;
  for (int i = threadIdx.x; i < N * K; i += 128) sW[(i / K) * KP + (i % K)] = W[i];
  for (int i = threadIdx.x; i < 64 * K; i += 128) {
    const int r = i / K, k = i % K;
    const int64_t gr = row0 + r;
    sX[r * KP + k] = gr < M ? X[gr * ldx + k] : __float2bfloat16(0.0f);
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int r0 = warp * 16;
  float acc[N / 8][4];
#pragma unroll
  for (int n = 0; n < N / 8; n++) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0f;
#pragma unroll
  for (int kk = 0; kk < K; kk += 16) {
    uint32_t a[4];
    a[0] = *(const uint32_t*)&sX[(r0 + g) * KP + kk + 2 * t];
    a[1] = *(const uint32_t*)&sX[(r0 + g + 8) * KP + kk + 2 * t];
    a[2] = *(const uint32_t*)&sX[(r0 + g) * KP + kk + 8 + 2 * t];
    a[3] = *(const uint32_t*)&sX[(r0 + g + 8) * KP + kk + 8 + 2 * t];
#pragma unroll
    for (int n = 0; n < N / 8; n++) {
      uint32_t b[2];
      b[0] = *(const uint32_t*)&sW[(n * 8 + g) * KP + kk + 2 * t];
      b[1] = *(const uint32_t*)&sW[(n * 8 + g) * KP + kk + 8 + 2 * t];
      mma_bf16(acc[n], a, b);
    }
  }
#pragma unroll
  for (int n = 0; n < N / 8; n++) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int64_t gr = row0 + r0 + g + 8 * h;
      if (gr >= M) continue;
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int col = n * 8 + 2 * t + e;
        const float z = acc[n][2 * h + e] + (bias ? bias[col] : 0.0f);
        if (Z) Z[gr * ldz + col] = z;
        if (Y) Y[gr * ldy + col] = __float2bfloat16(act ? silu(z) : z);
      }
    }
  }
}

// dW [N x K] += dZ^T X, db [N] += column sums of dZ, over rows [chunk*128, +128)
template <int N, int K>
__global__ void __launch_bounds__(256)
k_linear_dw(int64_t M, const __nv_bfloat16* __restrict__ dZ, int64_t lddz, const __nv_bfloat16* __restrict__ X,
            int64_t ldx, float* dW, float* db) {
  constexpr int CH = 128;
  constexpr int TN = (N >= 128) ? 8 : 2, TK = (N >= 128) ? ((K >= 128) ? 8 : 4) : 8;
  static_assert((N / TN) * (K / TK) == 256, "one tile per thread");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* sZ = (float*)smem_raw;            // [CH x N]
  float* sX = sZ + CH * N;                 // [CH x K]
  const int64_t r0 = (int64_t)blockIdx.x * CH;
  for (int i = threadIdx.x; i < CH * N; i += 256) {
    const int64_t r = r0 + i / N;
    sZ[i] = r < M ? __bfloat162float(dZ[r * lddz + i % N]) : 0.0f;
  }
  for (int i = threadIdx.x; i < CH * K; i += 256) {
    const int64_t r = r0 + i / K;
    sX[i] = r < M ? __bfloat162float(X[r * ldx + i % K]) : 0.0f;
  }
  __syncthreads();
  const int tn = threadIdx.x / (K / TK), tk = threadIdx.x % (K / TK);
  float acc[TN][TK];
  for (int a = 0; a < TN; a++)
    for (int b = 0; b < TK; b++) acc[a][b] = 0.0f;
  for (int m = 0; m < CH; m++) {
    float zn[TN], xk[TK];
    for (int a = 0; a < TN; a++) zn[a] = sZ[m * N + tn * TN + a];
    for (int b = 0; b < TK; b++) xk[b] = sX[m * K + tk * TK + b];
    for (int a = 0; a < TN; a++)
      for (int b = 0; b < TK; b++) acc[a][b] = fmaf(zn[a], xk[b], acc[a][b]);
  }
  for (int a = 0; a < TN; a++)
    for (int b = 0; b < TK; b++) atomicAdd(&dW[(tn * TN + a) * K + tk * TK + b], acc[a][b]);
  if (db && threadIdx.x < N) {
    float s = 0.0f;
    for (int m = 0; m < CH; m++) s += sZ[m * N + threadIdx.x];
    atomicAdd(&db[threadIdx.x], s);
  }
}

// dZ = dY * silu'(Z), silu'(z) = s (1 + z (1 - s)), s = 1/(1+e^-z); bf16 out
__global__ void k_silu_backward(int64_t n, const float* Z, const __nv_bfloat16* dY, __nv_bfloat16* dZ) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float z = Z[i];
  const float s = 1.0f / (1.0f + expf(-z));
  dZ[i] = __float2bfloat16(__bfloat162float(dY[i]) * s * (1.0f + z * (1.0f - s)));
}

// loss = sum_m [w0 (y0 - t0)^2 + w1/20 sum_{j=1..20} (yj - tj)^2] / M ; dY bf16 [M x 32].
// A lane is an output, a warp takes LOSS_ROWS rows: coalesced rows and one atomic per block
// (a thread per row took 12 us at 4,096 rows: strided rows and 4,096 atomics; this, 3 us).
constexpr int LOSS_WARPS = 8, LOSS_ROWS = 4;
__global__ void __launch_bounds__(32 * LOSS_WARPS)
k_mlp_loss(int64_t M, const float* Y, const float* T, float w0, float w1, float* loss, __nv_bfloat16* dY) {
  static_assert(MLP_OUTP == 32, "a lane per output");
  __shared__ float part[LOSS_WARPS];
  const int warp = threadIdx.x >> 5, j = threadIdx.x & 31;
  const int64_t m0 = ((int64_t)blockIdx.x * LOSS_WARPS + warp) * LOSS_ROWS;
  const float inv = 1.0f / (float)M, w = j == 0 ? w0 : w1 / FEAT_LEVELS;
  float l = 0.0f;
#pragma unroll
  for (int i = 0; i < LOSS_ROWS; i++) {
    const int64_t m = m0 + i;
    if (m >= M) break;
    float d = 0.0f;
    if (j <= FEAT_LEVELS) {
      const float e = Y[m * MLP_OUTP + j] - T[m * MLP_OUTP + j];
      l += w * e * e;
      d = 2.0f * w * e * inv;
    }
    dY[m * MLP_OUTP + j] = __float2bfloat16(d);
  }
  for (int o = 16; o; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
  if (j == 0) part[warp] = l;
  __syncthreads();
  if (threadIdx.x == 0) {
    l = 0.0f;
    for (int i = 0; i < LOSS_WARPS; i++) l += part[i];
    atomicAdd(loss, l * inv);
  }
}

// Adam on fp32 master weights [rows x cols]; writes the bf16 copy and its transpose
__global__ void k_adam(int64_t rows, int64_t cols, float* w, const float* g, float* m, float* v, float lr,
                       float b1, float b2, float eps, float c1, float c2, __nv_bfloat16* wb, __nv_bfloat16* wbt) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows * cols) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.0f - b1) * gi;
  const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  w[i] = wi;
  if (wb) wb[i] = __float2bfloat16(wi);
  if (wbt) wbt[(i % cols) * rows + i / cols] = __float2bfloat16(wi);
}

// Normalised bf16 features of every column at the start of a solve (first substep); zeros
// before the normalisation where a column has no solve.  A block takes FT_COLS columns as
// (level, column) items, column fastest, so that the level arrays are read in rows, and
// writes its rows of X as one range.  A thread per column read the
// same bytes in 225 us at 131,072 columns (one level's chain of loads after another, 64
// scattered 2-byte stores); this takes 51 us, bound by the FP64 unit that the
// double-to-float conversions go through (85 % busy).  In integer instructions the
// conversions took the same 51 us, then bound by instructions issued.
constexpr int FT_COLS = 32, FT_PARTS = 10, FT_LD = MLP_IN + 2;   // FT_LD: an odd number of words
constexpr int FT_PER = FEAT_LEVELS / FT_PARTS;                    // levels of a thread
static_assert(FEAT_LEVELS % FT_PARTS == 0, "the levels split evenly");
__global__ void __launch_bounds__(FT_COLS * FT_PARTS)
k_mlp_features(Dims D, int64_t nc, clmgb_soilwater_fields f, float e_ice, float remaining, float minutes,
               const float* __restrict__ mean, const float* __restrict__ istd, __nv_bfloat16* X, int words) {
  __shared__ float sat[FEAT_LEVELS + 2][FT_COLS], root[FEAT_LEVELS + 1][FT_COLS], norm[2][MLP_IN];
  __shared__ __align__(16) __nv_bfloat16 out[FT_COLS][FT_LD];
  const int64_t ld = D.ldc, c0 = (int64_t)blockIdx.x * FT_COLS;
  const int col = threadIdx.x % FT_COLS, part = threadIdx.x / FT_COLS;
  const int64_t c = c0 + col;
  if (threadIdx.x < MLP_IN) {
    norm[0][threadIdx.x] = mean[threadIdx.x];
    norm[1][threadIdx.x] = istd[threadIdx.x];
  }
  // every load of the thread before any of them is used, those of columns without a solve
  // and of levels below a column's lowest included: whether they count is itself a load
  uint8_t live = 0;
  int64_t bed = 0;
  if (c < nc) {
    live = f.mask_hydrology[c];
    bed = f.col_nbedrock[c];
  }
  double liq[FT_PER], dz[FT_PER], ws[FT_PER], rt[FT_PER], ice[FT_PER], below[FT_PER], bsw[FT_PER], hksat[FT_PER];
#pragma unroll
  for (int i = 0; i < FT_PER; i++) {
    const int j = 1 + part + i * FT_PARTS;
    liq[i] = dz[i] = ws[i] = rt[i] = ice[i] = below[i] = bsw[i] = hksat[i] = 0.0;
    if (c < nc && j <= D.nlevsoi) {
      liq[i] = LV(f.h2osoi_liq, c, D.nlevsno + j, ld);
      dz[i] = LVc(f.dz, c, D.nlevsno + j, ld);
      ws[i] = LVc(f.watsat, c, j, ld);
      rt[i] = LVc(f.qflx_rootsoi, c, j, ld);
      ice[i] = LV(f.icefrac, c, j, ld);
      if (j < D.nlevsoi) below[i] = LV(f.icefrac, c, j + 1, ld);
      bsw[i] = LVc(f.bsw, c, j, ld);
      hksat[i] = LVc(f.hksat, c, j, ld);
    }
  }
  const int nl = live && bed >= 1 && bed <= D.nlevsoi ? (int)bed : 0;
  float sv[FT_PER], xi[FT_PER];
#pragma unroll
  for (int i = 0; i < FT_PER; i++) {
    const int j = 1 + part + i * FT_PARTS;
    const bool in = j <= nl;
    sv[i] = in ? feature_saturation(liq[i], dz[i], ws[i]) : 0.0f;
    xi[i] = in ? (float)ice[i] : 0.0f;
    sat[j][col] = sv[i];
    root[j][col] = in ? (float)rt[i] : 0.0f;
  }
  constexpr int next = FEAT_LEVELS + 1;               // a level below those of the features
  if (part == 0)
    sat[next][col] = nl >= next ? feature_saturation(LV(f.h2osoi_liq, c, D.nlevsno + next, ld),
                                                     LVc(f.dz, c, D.nlevsno + next, ld), LVc(f.watsat, c, next, ld))
                                : 0.0f;
  __syncthreads();
  auto put = [&](int i, float x) { out[col][i] = __float2bfloat16((x - norm[0][i]) * norm[1][i]); };
#pragma unroll
  for (int i = 0; i < FT_PER; i++) {
    const int j = 1 + part + i * FT_PARTS;
    float xc = nl ? -30.0f : 0.0f;
    if (j <= nl)
      xc = feature_log_conductivity(j == nl, sv[i], sat[j + 1][col], ice[i], below[i], bsw[i], hksat[i], e_ice);
    put(j - 1, sv[i]);
    put(19 + j, xi[i]);
    put(39 + j, xc);
  }
  if (part == 0) {
    float sink = 0.0f;
    for (int j = 1; j <= FEAT_LEVELS && j <= nl; j++) sink += root[j][col];
    put(60, nl ? (float)(f.qflx_infl[c] * 1.0e3) : 0.0f);
    put(61, nl ? sink * 1.0e3f : 0.0f);
    put(62, nl ? remaining : 0.0f);
    put(63, nl ? log2f(minutes) / 6.0f : 0.0f);
  }
  __syncthreads();
  const int rows = (int)(nc - c0 < FT_COLS ? nc - c0 : FT_COLS);
  if (words) {                                      // X on a 4-byte boundary
    uint32_t* X32 = reinterpret_cast<uint32_t*>(X + c0 * MLP_IN);
    for (int i = threadIdx.x; i < rows * MLP_IN / 2; i += FT_COLS * FT_PARTS)
      X32[i] = *reinterpret_cast<const uint32_t*>(&out[i / (MLP_IN / 2)][i % (MLP_IN / 2) * 2]);
  } else {
    for (int i = threadIdx.x; i < rows * MLP_IN; i += FT_COLS * FT_PARTS)
      X[c0 * MLP_IN + i] = out[i / MLP_IN][i % MLP_IN];
  }
}

// first substep = dtime / 2^k, k = clamp(ceil(y0 - margin), 0, kmax)
__global__ void k_mlp_first_dt(int64_t nc, const float* Y, double dtime, float margin, int kmax, double* dt_first) {
  const int64_t c = (int64_t)blockIdx.x * 128 + threadIdx.x;
  if (c >= nc) return;
  const float y = Y[c * MLP_OUTP];
  int k = (int)ceilf(y - margin);
  if (!(y == y)) k = 0;
  k = k < 0 ? 0 : (k > kmax ? kmax : k);
  double dt = dtime;
  for (int i = 0; i < k; i++) dt = dt / 2.0;
  dt_first[c] = dt;
}

// ---------------------------------------------------------------------------
template <int K, int N>
static cudaError_t linear_launch(int64_t M, const void* X, int64_t ldx, const void* W, const float* b, int act,
                                 float* Z, int64_t ldz, void* Y, int64_t ldy, cudaStream_t s) {
  const size_t smem = (size_t)(N + 64) * (K + 8) * sizeof(__nv_bfloat16);
  cudaError_t e = cudaFuncSetAttribute(k_linear<K, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const unsigned int grid = (unsigned int)((M + 63) / 64);
  if (grid == 0) return cudaSuccess;
  k_linear<K, N><<<grid, 128, smem, s>>>(M, (const __nv_bfloat16*)X, ldx, (const __nv_bfloat16*)W, b, act, Z, ldz,
                                         (__nv_bfloat16*)Y, ldy);
  return cudaGetLastError();
}

cudaError_t launch_mlp_linear(int64_t M, int N, int K, const void* X, int64_t ldx, const void* W, const float* b,
                              int act, float* Z, int64_t ldz, void* Y, int64_t ldy, cudaStream_t s) {
  if (K == 64 && N == 128) return linear_launch<64, 128>(M, X, ldx, W, b, act, Z, ldz, Y, ldy, s);
  if (K == 128 && N == 128) return linear_launch<128, 128>(M, X, ldx, W, b, act, Z, ldz, Y, ldy, s);
  if (K == 128 && N == 32) return linear_launch<128, 32>(M, X, ldx, W, b, act, Z, ldz, Y, ldy, s);
  if (K == 32 && N == 128) return linear_launch<32, 128>(M, X, ldx, W, b, act, Z, ldz, Y, ldy, s);
  return cudaErrorInvalidValue;
}

template <int N, int K>
static cudaError_t dw_launch(int64_t M, const void* dZ, int64_t lddz, const void* X, int64_t ldx, float* dW,
                             float* db, cudaStream_t s) {
  const size_t smem = (size_t)128 * (N + K) * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(k_linear_dw<N, K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const unsigned int grid = (unsigned int)((M + 127) / 128);
  if (grid == 0) return cudaSuccess;
  k_linear_dw<N, K><<<grid, 256, smem, s>>>(M, (const __nv_bfloat16*)dZ, lddz, (const __nv_bfloat16*)X, ldx, dW,
                                            db);
  return cudaGetLastError();
}

cudaError_t launch_mlp_linear_dw(int64_t M, int N, int K, const void* dZ, int64_t lddz, const void* X, int64_t ldx,
                                 float* dW, float* db, cudaStream_t s) {
  if (N == 128 && K == 64) return dw_launch<128, 64>(M, dZ, lddz, X, ldx, dW, db, s);
  if (N == 128 && K == 128) return dw_launch<128, 128>(M, dZ, lddz, X, ldx, dW, db, s);
  if (N == 32 && K == 128) return dw_launch<32, 128>(M, dZ, lddz, X, ldx, dW, db, s);
  return cudaErrorInvalidValue;
}

cudaError_t launch_mlp_silu_backward(int64_t n, const float* Z, const void* dY, void* dZ, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_silu_backward<<<(unsigned int)((n + 255) / 256), 256, 0, s>>>(n, Z, (const __nv_bfloat16*)dY,
                                                                 (__nv_bfloat16*)dZ);
  return cudaGetLastError();
}

cudaError_t launch_mlp_loss(int64_t M, const float* Y, const float* T, float w0, float w1, float* loss, void* dY,
                            cudaStream_t s) {
  if (M <= 0) return cudaSuccess;
  constexpr int rows = LOSS_WARPS * LOSS_ROWS;
  k_mlp_loss<<<(unsigned int)((M + rows - 1) / rows), 32 * LOSS_WARPS, 0, s>>>(M, Y, T, w0, w1, loss, (__nv_bfloat16*)dY);
  return cudaGetLastError();
}

cudaError_t launch_mlp_adam(int64_t rows, int64_t cols, float* w, const float* g, float* m, float* v, float lr,
                            float b1, float b2, float eps, int step, void* wb, void* wbt, cudaStream_t s) {
  const int64_t n = rows * cols;
  if (n <= 0) return cudaSuccess;
  const float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
  k_adam<<<(unsigned int)((n + 255) / 256), 256, 0, s>>>(rows, cols, w, g, m, v, lr, b1, b2, eps, c1, c2,
                                                        (__nv_bfloat16*)wb, (__nv_bfloat16*)wbt);
  return cudaGetLastError();
}

cudaError_t launch_richards_samples(const Dims& D, int64_t nc, const clmgb_soilwater_fields& f,
                                    const clmgb_swm_config& cfg, double dtime, int rmax, float* feat, float* targ,
                                    unsigned int* count, int64_t capacity, uint32_t* col_status, cudaStream_t s) {
  k_richards_samples<<<(unsigned int)((nc + 63) / 64), 64, 0, s>>>(D, nc, f, cfg, dtime, rmax, feat, targ, count,
                                                                   capacity, col_status);
  return cudaGetLastError();
}

cudaError_t launch_mlp_features(const Dims& D, int64_t nc, const clmgb_soilwater_fields& f,
                                const clmgb_swm_config& cfg, double dtime, const float* mean, const float* istd,
                                void* X, cudaStream_t s) {
  k_mlp_features<<<(unsigned int)((nc + FT_COLS - 1) / FT_COLS), FT_COLS * FT_PARTS, 0, s>>>(
      D, nc, f, (float)cfg.e_ice, (float)(dtime / dtime), (float)(dtime / 60.0), mean, istd, (__nv_bfloat16*)X,
      ((uintptr_t)X & 3) == 0);
  return cudaGetLastError();
}

cudaError_t launch_mlp_first_dt(int64_t nc, const float* Y, double dtime, float margin, int kmax, double* dt_first,
                                cudaStream_t s) {
  k_mlp_first_dt<<<(unsigned int)((nc + 127) / 128), 128, 0, s>>>(nc, Y, dtime, margin, kmax, dt_first);
  return cudaGetLastError();
}

}  // namespace clmgb
