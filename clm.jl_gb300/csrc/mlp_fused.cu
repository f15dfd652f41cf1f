// mlp_fused.cu — the warm-start perceptron's passes as one launch each: the three layers
// forward, the three layers backward with their weight gradients, and the optimiser step
// over all parameters.
//
// The layers are narrow (64 -> 128 -> 128 -> 32), so a pass is bound by what it moves and by
// launches, not by its products: layer by layer each kernel read its weights and its input
// element by element and the next one read back what it wrote.  Here the weights stay in
// shared memory, a warp takes its rows through all layers with the activations in shared
// memory, and operands come in 16-byte loads and ldmatrix.  The layers' products are mma.sync
// m16n8k16 (BF16 x BF16 -> FP32) in the same order as in mlp.cu, and activations round to
// BF16 at the same places, so the forward pass and the backward signals are the same bits; the
// weight gradients sum their rows on the CUDA cores as there, 128 rows a block and an atomic
// addition a block.
//
// Device time of a training step of 4,096 rows: about 175 -> 53 us (forward 14, loss 4,
// backward 32, optimiser 3); the step is the host's (eight allocations and four calls,
// 155 us against 225 us with one call per layer).  Forward of 131,072 rows without
// activations kept: 257 -> 64 us, the warps waiting on shared memory and on the exponentials
// and divisions of SiLU (tensor pipe 18 % active, issue 41 %).
#include <cuda_bf16.h>
#include "clmgb_device.cuh"
#include "launch.h"

namespace clmgb {

namespace {

typedef __nv_bfloat16 bf16;
constexpr int NI = 64, NH = 128, NO = 32;           // inputs, hidden units, padded outputs
constexpr int LDI = NI + 8, LDH = NH + 8, LDO = NO + 8;   // padded rows: ldmatrix without bank conflicts

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldsm(uint32_t* r, uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void mma(float* d, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack2(float x, float y) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
  uint32_t u;
  memcpy(&u, &v, 4);
  return u;
}
__device__ __forceinline__ float silu(float z) { return z / (1.0f + expf(-z)); }

// A [rows x cols] BF16 array (rows contiguous) into shared memory rows of ld elements;
// rows from `valid` on are zeros.
template <int COLS>
__device__ __forceinline__ void stage(bf16* dst, int ld, const bf16* src, int rows, int64_t valid, int tid, int nt) {
  constexpr int CH = COLS / 8;
  for (int i = tid; i < rows * CH; i += nt) {
    const int r = i / CH, q = i % CH;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (r < valid) v = *reinterpret_cast<const uint4*>(src + (int64_t)r * COLS + q * 8);
    *reinterpret_cast<uint4*>(dst + r * ld + q * 8) = v;
  }
}

// acc[N/8][4] = the 16 rows at x (ldx) times W [N x K] (ldw) transposed
template <int K, int N>
__device__ __forceinline__ void tile_product(float (*acc)[4], const bf16* x, int ldx, const bf16* w, int ldw) {
  const int lane = threadIdx.x & 31;
  const uint32_t xa = smem_addr(x + ((lane & 7) + ((lane >> 3) & 1) * 8) * ldx + (lane >> 4) * 8);
  const uint32_t wa = smem_addr(w + ((lane & 7) + (lane >> 4) * 8) * ldw + ((lane >> 3) & 1) * 8);
#pragma unroll
  for (int n = 0; n < N / 8; n++) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0f;
#pragma unroll
  for (int k = 0; k < K; k += 16) {
    uint32_t a[4];
    ldsm(a, xa + k * 2);
#pragma unroll
    for (int n = 0; n < N / 16; n++) {
      uint32_t b[4];
      ldsm(b, wa + (n * 16 * ldw + k) * 2);
      mma(acc[2 * n], a, b[0], b[1]);
      mma(acc[2 * n + 1], a, b[2], b[3]);
    }
  }
}

// A hidden layer of a warp's 16 rows: z = acc + bias, h = silu(z) into the warp's rows hs of
// shared memory; with Z also z and h to global memory (rows below `valid`).
template <bool KEEP>
__device__ __forceinline__ void hidden_layer(float (*acc)[4], const float* bias, bf16* hs, float* Z, bf16* H,
                                             int64_t valid) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  __syncwarp();                                     // the layer's input rows are read
#pragma unroll
  for (int n = 0; n < NH / 8; n++) {
    const int col = n * 8 + 2 * t;
    const float b0 = bias[col], b1 = bias[col + 1];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int r = g + 8 * h;
      const float z0 = acc[n][2 * h] + b0, z1 = acc[n][2 * h + 1] + b1;
      if (KEEP && r < valid) *reinterpret_cast<float2*>(Z + (int64_t)r * NH + col) = make_float2(z0, z1);
      *reinterpret_cast<uint32_t*>(hs + r * LDH + col) = pack2(silu(z0), silu(z1));
    }
  }
  __syncwarp();
  if (KEEP) {
#pragma unroll
    for (int i = lane; i < 16 * NH / 8; i += 32) {
      const int r = i / (NH / 8), q = i % (NH / 8);
      if (r < valid)
        *reinterpret_cast<uint4*>(H + (int64_t)r * NH + q * 8) = *reinterpret_cast<const uint4*>(hs + r * LDH + q * 8);
    }
  }
}

constexpr int FW_WARPS = 8;
constexpr size_t FW_SMEM = sizeof(bf16) * (size_t)(NH * LDI + NH * LDH + NO * LDH + FW_WARPS * 16 * LDH) +
                           sizeof(float) * (size_t)(2 * NH + NO);

// Y = the network's outputs of X's rows; with KEEP also the pre-activations and activations
// the backward pass reads.  A warp takes 16 rows at a time through the three layers, its
// rows of shared memory holding each layer's input in turn, so that two blocks of 8 warps
// fit an SM beside their weights (4 warps with rows of their own for X: 73 us for 64).
template <bool KEEP>
__global__ void __launch_bounds__(32 * FW_WARPS, 2)
k_mlp_forward(int64_t M, const bf16* __restrict__ X, const bf16* __restrict__ W1, const float* __restrict__ b1,
              const bf16* __restrict__ W2, const float* __restrict__ b2, const bf16* __restrict__ W3,
              const float* __restrict__ b3, float* Z1, bf16* H1, float* Z2, bf16* H2, float* Y) {
  extern __shared__ __align__(16) unsigned char smem_fw[];
  bf16* const s1 = reinterpret_cast<bf16*>(smem_fw);
  bf16* const s2 = s1 + NH * LDI;
  bf16* const s3 = s2 + NH * LDH;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  bf16* const hs = s3 + NO * LDH + warp * 16 * LDH;     // the rows of X, then of H1, then of H2
  float* const bias = reinterpret_cast<float*>(s3 + NO * LDH + FW_WARPS * 16 * LDH);
  for (int i = tid; i < 2 * NH + NO; i += 32 * FW_WARPS)
    bias[i] = i < NH ? b1[i] : (i < 2 * NH ? b2[i - NH] : b3[i - 2 * NH]);
  stage<NI>(s1, LDI, W1, NH, NH, tid, 32 * FW_WARPS);
  stage<NH>(s2, LDH, W2, NH, NH, tid, 32 * FW_WARPS);
  stage<NH>(s3, LDH, W3, NO, NO, tid, 32 * FW_WARPS);
  __syncthreads();
  const int g = lane >> 2, t = lane & 3;
  const int64_t tiles = (M + 15) / 16;
  for (int64_t tile = (int64_t)warp * gridDim.x + blockIdx.x; tile < tiles; tile += (int64_t)gridDim.x * FW_WARPS) {
    const int64_t r0 = tile * 16, valid = M - r0;
    __syncwarp();
    stage<NI>(hs, LDI, X + r0 * NI, 16, valid, lane, 32);
    __syncwarp();
    float acc[NH / 8][4];
    tile_product<NI, NH>(acc, hs, LDI, s1, LDI);
    hidden_layer<KEEP>(acc, bias, hs, KEEP ? Z1 + r0 * NH : nullptr, KEEP ? H1 + r0 * NH : nullptr, valid);
    tile_product<NH, NH>(acc, hs, LDH, s2, LDH);
    hidden_layer<KEEP>(acc, bias + NH, hs, KEEP ? Z2 + r0 * NH : nullptr, KEEP ? H2 + r0 * NH : nullptr, valid);
    tile_product<NH, NO>(acc, hs, LDH, s3, LDH);
#pragma unroll
    for (int n = 0; n < NO / 8; n++) {
      const int col = n * 8 + 2 * t;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int r = g + 8 * h;
        if (r < valid)
          *reinterpret_cast<float2*>(Y + (r0 + r) * NO + col) =
              make_float2(acc[n][2 * h] + bias[2 * NH + col], acc[n][2 * h + 1] + bias[2 * NH + col + 1]);
      }
    }
  }
}

// T consecutive BF16 values on a boundary of their size, as floats
template <int T>
__device__ __forceinline__ void load_floats(const bf16* p, float* v) {
  uint32_t u[(T + 1) / 2];
  if constexpr (T == 1) u[0] = *reinterpret_cast<const uint16_t*>(p);
  else if constexpr (T == 2) u[0] = *reinterpret_cast<const uint32_t*>(p);
  else if constexpr (T == 4) *reinterpret_cast<uint2*>(u) = *reinterpret_cast<const uint2*>(p);
  else *reinterpret_cast<uint4*>(u) = *reinterpret_cast<const uint4*>(p);
#pragma unroll
  for (int i = 0; i < T; i++) v[i] = __uint_as_float(i & 1 ? u[i / 2] & 0xffff0000u : u[i / 2] << 16);
}

// dW [N x K] += the block's rows of dz^T x, rows `part` of S parts of dW: a tile of TN x TK
// for each thread, its sums in FP32 rounded to nearest, row after row, then one atomic
// addition: the additions of k_linear_dw (mlp.cu), whose partial sums these are bit for bit.
// (On the tensor cores, whose sums of 16 products are truncated, and by 64 rows, which
// doubles the atomic additions, the error against 64-bit sums was 1.1 times this at 16 rows
// and 1.4 to 1.6 times from 1,000 rows on.)
constexpr int BR = 128, BW = 16;                    // rows and warps of a backward block
template <int N, int K, int S>
__device__ __forceinline__ void weight_gradient(const bf16* dz, int ldz, const bf16* x, int ldx, float* dW, int part) {
  constexpr int PER = N / S * K / (32 * BW), TK = PER < 4 ? PER : 4, TN = PER / TK;
  static_assert(TN * TK * 32 * BW == N / S * K && K % TK == 0, "a tile per thread");
  const int n0 = part * (N / S) + threadIdx.x / (K / TK) * TN, k0 = threadIdx.x % (K / TK) * TK;
  float acc[TN][TK];
#pragma unroll
  for (int a = 0; a < TN; a++)
#pragma unroll
    for (int b = 0; b < TK; b++) acc[a][b] = 0.0f;
#pragma unroll 4
  for (int m = 0; m < BR; m++) {
    float zn[TN], xk[TK];
    load_floats<TN>(dz + m * ldz + n0, zn);
    load_floats<TK>(x + m * ldx + k0, xk);
#pragma unroll
    for (int a = 0; a < TN; a++)
#pragma unroll
      for (int b = 0; b < TK; b++) acc[a][b] = fmaf(zn[a], xk[b], acc[a][b]);
  }
#pragma unroll
  for (int a = 0; a < TN; a++) {
    float* p = dW + (n0 + a) * K + k0;
    if constexpr (TK == 4)
      asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(acc[a][0]), "f"(acc[a][1]),
                   "f"(acc[a][2]), "f"(acc[a][3])
                   : "memory");
    else
      asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(acc[a][0]), "f"(acc[a][1]) : "memory");
  }
}

// db += the columns' sums over the block's rows
template <int N>
__device__ __forceinline__ void bias_gradient(const bf16* dz, int ldz, float* db) {
  if (threadIdx.x < N) {
    float s = 0.0f;
#pragma unroll 16
    for (int m = 0; m < BR; m++) s += __bfloat162float(dz[m * ldz + threadIdx.x]);
    atomicAdd(&db[threadIdx.x], s);
  }
}

// dz = silu'(z) * bf16(dx): the warp's 16 rows and N columns of a layer's backward signal
template <int N>
__device__ __forceinline__ void signal(float (*acc)[4], const float* Z, int64_t valid, bf16* dz) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int n = 0; n < N / 8; n++) {
    const int col = n * 8 + 2 * t;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int r = g + 8 * h;
      float v[2] = {0.0f, 0.0f};
      if (r < valid) {
        const float2 z2 = *reinterpret_cast<const float2*>(Z + (int64_t)r * NH + col);
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const float z = e ? z2.y : z2.x;
          const float s = 1.0f / (1.0f + expf(-z));
          v[e] = __bfloat162float(__float2bfloat16(acc[n][2 * h + e])) * s * (1.0f + z * (1.0f - s));
        }
      }
      *reinterpret_cast<uint32_t*>(dz + r * LDH + col) = pack2(v[0], v[1]);
    }
  }
}

constexpr size_t BW_SMEM = sizeof(bf16) * (size_t)(NH * LDO + NH * LDH + BR * (LDO + 3 * LDH + LDI));

// The backward pass over BR rows per block: dZ2 = silu'(Z2) (dY W3), dZ1 = silu'(Z1) (dZ2
// W2) in shared memory, and the block's share of the three weight and bias gradients.  S
// blocks share the rows' weight gradients, each with the signals formed again.
// w3t, w2t: the transposed weights [in x out].
template <int S>
__global__ void __launch_bounds__(32 * BW)
k_mlp_backward(int64_t M, const bf16* __restrict__ X, const float* __restrict__ Z1, const bf16* __restrict__ H1,
               const float* __restrict__ Z2, const bf16* __restrict__ H2, const bf16* __restrict__ dY,
               const bf16* __restrict__ w2t, const bf16* __restrict__ w3t, float* dW1, float* dW2, float* dW3,
               float* db1, float* db2, float* db3) {
  extern __shared__ __align__(16) unsigned char smem_bw[];
  bf16* const s3 = reinterpret_cast<bf16*>(smem_bw);           // [NH][LDO]
  bf16* const s2 = s3 + NH * LDO;                              // [NH][LDH]
  bf16* const dy = s2 + NH * LDH;                              // [BR][LDO]
  bf16* const dz2 = dy + BR * LDO;                             // [BR][LDH]
  bf16* const dz1 = dz2 + BR * LDH;
  bf16* const act = dz1 + BR * LDH;                            // H2, then H1
  bf16* const xs = act + BR * LDH;                             // [BR][LDI]
  const int tid = threadIdx.x, warp = tid >> 5;
  const int64_t r0 = (int64_t)blockIdx.x * BR, valid = M - r0;
  stage<NO>(s3, LDO, w3t, NH, NH, tid, 32 * BW);
  stage<NO>(dy, LDO, dY + r0 * NO, BR, valid, tid, 32 * BW);
  stage<NH>(s2, LDH, w2t, NH, NH, tid, 32 * BW);
  stage<NH>(act, LDH, H2 + r0 * NH, BR, valid, tid, 32 * BW);
  stage<NI>(xs, LDI, X + r0 * NI, BR, valid, tid, 32 * BW);
  __syncthreads();
  // warp w: rows 16 (w / 2) .. and columns 64 (w % 2) .. of the backward signals
  const int row = (warp >> 1) * 16, half = (warp & 1) * (NH / 2);
  float acc[NH / 16][4];
  const int part = S > 1 ? (int)blockIdx.y : 0;
  tile_product<NO, NH / 2>(acc, dy + row * LDO, LDO, s3 + half * LDO, LDO);
  signal<NH / 2>(acc, Z2 + (r0 + row) * NH + half, valid - row, dz2 + row * LDH + half);
  weight_gradient<NO, NH, S>(dy, LDO, act, LDH, dW3, part);
  if (part == 0) bias_gradient<NO>(dy, LDO, db3);
  __syncthreads();                                             // dz2 is written, H2 read
  stage<NH>(act, LDH, H1 + r0 * NH, BR, valid, tid, 32 * BW);
  tile_product<NH, NH / 2>(acc, dz2 + row * LDH, LDH, s2 + half * LDH, LDH);
  signal<NH / 2>(acc, Z1 + (r0 + row) * NH + half, valid - row, dz1 + row * LDH + half);
  __syncthreads();
  weight_gradient<NH, NH, S>(dz2, LDH, act, LDH, dW2, part);
  if (part == 0) bias_gradient<NH>(dz2, LDH, db2);
  weight_gradient<NH, NI, S>(dz1, LDH, xs, LDI, dW1, part);
  if (part == S - 1) bias_gradient<NH>(dz1, LDH, db1);
}

// One Adam step over the six parameter arrays (the expressions of k_adam)
struct AdamArrays {
  float *w[6], *m[6], *v[6];
  const float* g[6];
  bf16 *wb[6], *wt[6];
  int rows[6], cols[6];
};
__global__ void __launch_bounds__(256)
k_mlp_adam_net(const __grid_constant__ AdamArrays a, float lr, float b1, float b2, float eps, float c1, float c2) {
  const int p = blockIdx.y, n = a.rows[p] * a.cols[p];
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  const float gi = a.g[p][i];
  const float mi = b1 * a.m[p][i] + (1.0f - b1) * gi;
  const float vi = b2 * a.v[p][i] + (1.0f - b2) * gi * gi;
  a.m[p][i] = mi;
  a.v[p][i] = vi;
  const float wi = a.w[p][i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  a.w[p][i] = wi;
  if (a.wb[p]) a.wb[p][i] = __float2bfloat16(wi);
  if (a.wt[p]) a.wt[p][(i % a.cols[p]) * a.rows[p] + i / a.cols[p]] = __float2bfloat16(wi);
}

}  // namespace

cudaError_t launch_mlp_forward(int64_t M, const void* X, const clmgb_mlp_net& net, float* Z1, void* H1, float* Z2,
                               void* H2, float* Y, int num_sms, cudaStream_t s) {
  if (M <= 0) return cudaSuccess;
  const bool keep = Z1 != nullptr;
  auto kern = keep ? k_mlp_forward<true> : k_mlp_forward<false>;
  const cudaError_t e = allow_dynamic_smem(kern, FW_SMEM);
  if (e != cudaSuccess) return e;
  // two blocks fit an SM's shared memory; tiles go to blocks first, so that few of them
  // still spread over the SMs
  const int64_t tiles = (M + 15) / 16, most = 2 * (int64_t)num_sms;
  kern<<<(unsigned)(tiles < most ? tiles : most), 32 * FW_WARPS, FW_SMEM, s>>>(
      M, (const bf16*)X, (const bf16*)net.wb[0], net.b[0], (const bf16*)net.wb[1], net.b[1], (const bf16*)net.wb[2],
      net.b[2], Z1, (bf16*)H1, Z2, (bf16*)H2, Y);
  return cudaGetLastError();
}

cudaError_t launch_mlp_gradients(int64_t M, const void* X, const float* Z1, const void* H1, const float* Z2,
                                 const void* H2, const void* dY, const clmgb_mlp_net& net, const clmgb_mlp_grad& g,
                                 int num_sms, cudaStream_t s) {
  static const size_t wn[3] = {(size_t)NH * NI, (size_t)NH * NH, (size_t)NO * NH}, bn[3] = {NH, NH, NO};
  cudaError_t e;
  // one clear where the six arrays are one range, as the caller of this library lays them out
  bool one = true;
  const float* at = g.dw[0];
  for (int i = 0; i < 3; i++) {
    one = one && g.dw[i] == at;
    at += wn[i];
  }
  for (int i = 0; i < 3; i++) {
    one = one && g.db[i] == at;
    at += bn[i];
  }
  if (one) {
    if ((e = cudaMemsetAsync(g.dw[0], 0, (size_t)(at - g.dw[0]) * sizeof(float), s)) != cudaSuccess) return e;
  } else {
    for (int i = 0; i < 3; i++) {
      if ((e = cudaMemsetAsync(g.dw[i], 0, wn[i] * sizeof(float), s)) != cudaSuccess) return e;
      if ((e = cudaMemsetAsync(g.db[i], 0, bn[i] * sizeof(float), s)) != cudaSuccess) return e;
    }
  }
  if (M <= 0) return cudaSuccess;
  // as many blocks to the rows as keep all of them resident at once (a block fills an SM); us
  // for 1, 2 and 4: 4,096 rows 49 / 38 / 32, 9,000 50 / 38 / 61, 16,384 50 / 74 / 117
  const int64_t blocks = (M + BR - 1) / BR;
  const int split = blocks * 4 <= num_sms ? 4 : blocks * 2 <= num_sms ? 2 : 1;
  auto kern = split == 4 ? k_mlp_backward<4> : split == 2 ? k_mlp_backward<2> : k_mlp_backward<1>;
  if ((e = allow_dynamic_smem(kern, BW_SMEM)) != cudaSuccess) return e;
  kern<<<dim3((unsigned)blocks, (unsigned)split), 32 * BW, BW_SMEM, s>>>(
      M, (const bf16*)X, Z1, (const bf16*)H1, Z2, (const bf16*)H2, (const bf16*)dY, (const bf16*)net.wt[1],
      (const bf16*)net.wt[2], g.dw[0], g.dw[1], g.dw[2], g.db[0], g.db[1], g.db[2]);
  return cudaGetLastError();
}

cudaError_t launch_mlp_adam_net(const clmgb_mlp_net& net, const clmgb_mlp_grad& g, float lr, float b1, float b2,
                                float eps, int step, cudaStream_t s) {
  const float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
  static const int out[3] = {NH, NH, NO}, in[3] = {NI, NH, NH};
  AdamArrays a;
  for (int i = 0; i < 3; i++) {
    a.w[i] = net.w[i]; a.m[i] = net.mw[i]; a.v[i] = net.vw[i]; a.g[i] = g.dw[i];
    a.wb[i] = (bf16*)net.wb[i]; a.wt[i] = (bf16*)net.wt[i]; a.rows[i] = out[i]; a.cols[i] = in[i];
    a.w[3 + i] = net.b[i]; a.m[3 + i] = net.mb[i]; a.v[3 + i] = net.vb[i]; a.g[3 + i] = g.db[i];
    a.wb[3 + i] = a.wt[3 + i] = nullptr; a.rows[3 + i] = 1; a.cols[3 + i] = out[i];
  }
  k_mlp_adam_net<<<dim3((unsigned)(NH * NH + 255) / 256, 6), 256, 0, s>>>(a, lr, b1, b2, eps, c1, c2);
  return cudaGetLastError();
}

}  // namespace clmgb
