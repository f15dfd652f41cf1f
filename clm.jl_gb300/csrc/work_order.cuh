// work_order.cuh — the order in which columns are handed out: a counting sort by a small
// key, largest first, so that columns of like work run side by side and the long ones start
// first.  The order within a key is arbitrary and does not affect any result.
//
// Key: a functor with `int operator()(int64_t c) const` (0..ORDER_BINS - 1, or -1 for a
// column not listed) and `void unlisted(int64_t c) const`.  bins: [ORDER_BINS] counts,
// [ORDER_BINS] places handed out, [1] the number listed.
//
// The lanes of a warp with the same key take their places together (__match_any_sync),
// and a block reserves its places per key with one atomic: with a global atomic per column
// the scatter alone took 43 us at 65,536 columns, most of them on two or three keys, now 4.
// Up to ORDER_ONE_MAX columns one block does all of it, its keys in registers (3.4 us and
// one launch at 1,024 columns; 6.3 us and four with the count and the places apart); beyond,
// its passes over the columns are longer than two kernels (19 us against 9 at 10,007).
#pragma once
#include <stdint.h>
#include <cuda_runtime.h>

namespace clmgb {

constexpr int ORDER_BINS = 64;
constexpr int ORDER_WORDS = 2 * ORDER_BINS + 1;
constexpr int ORDER_THREADS = 256, ORDER_PER = 4;      // columns of a thread, many columns
constexpr int ORDER_ONE_THREADS = 1024;
constexpr int ORDER_ONE_PER = 4;
constexpr int64_t ORDER_ONE_MAX = ORDER_ONE_THREADS * ORDER_ONE_PER;   // columns that one block lists

// adds the warp's lanes with key b >= 0 to sh[b]; returns the lane's place among all added
__device__ __forceinline__ unsigned int order_add(unsigned int* sh, int b) {
  const unsigned int same = __match_any_sync(0xffffffffu, b);
  const int lane = threadIdx.x & 31, leader = __ffs(same) - 1;
  unsigned int first = 0;
  if (b >= 0 && lane == leader) first = atomicAdd(&sh[b], (unsigned)__popc(same));
  return __shfl_sync(0xffffffffu, first, leader) + __popc(same & ((1u << lane) - 1u));
}
// base[b] = the number of columns with larger keys; returns their total in thread 0
__device__ __forceinline__ unsigned int order_bases(const unsigned int* count, unsigned int* base) {
  if (threadIdx.x < ORDER_BINS) {
    unsigned int s = 0;
    for (int b = threadIdx.x + 1; b < ORDER_BINS; b++) s += count[b];
    base[threadIdx.x] = s;
    return s + count[threadIdx.x];
  }
  return 0;
}

template <class Key>
__global__ void __launch_bounds__(ORDER_ONE_THREADS)
k_order_one(int64_t nc, Key key, unsigned int* bins, uint32_t* order) {
  __shared__ unsigned int count[ORDER_BINS], base[ORDER_BINS];
  if (threadIdx.x < ORDER_BINS) count[threadIdx.x] = 0;
  __syncthreads();
  int b[ORDER_ONE_PER];
  unsigned int place[ORDER_ONE_PER];
#pragma unroll
  for (int i = 0; i < ORDER_ONE_PER; i++) {
    const int64_t c = i * ORDER_ONE_THREADS + threadIdx.x;
    b[i] = c < nc ? key(c) : -1;
  }
#pragma unroll
  for (int i = 0; i < ORDER_ONE_PER; i++) {
    const int64_t c = i * ORDER_ONE_THREADS + threadIdx.x;
    place[i] = order_add(count, b[i]);
    if (b[i] < 0 && c < nc) key.unlisted(c);
  }
  __syncthreads();
  const unsigned int n = order_bases(count, base);
  if (threadIdx.x == 0) bins[2 * ORDER_BINS] = n;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < ORDER_ONE_PER; i++)
    if (b[i] >= 0) order[base[b[i]] + place[i]] = (uint32_t)(i * ORDER_ONE_THREADS + threadIdx.x);
}

template <class Key>
__global__ void __launch_bounds__(ORDER_THREADS)
k_order_count(int64_t nc, Key key, unsigned int* bins) {
  __shared__ unsigned int count[ORDER_BINS];
  if (threadIdx.x < ORDER_BINS) count[threadIdx.x] = 0;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < ORDER_PER; i++) {
    const int64_t c = ((int64_t)blockIdx.x * ORDER_PER + i) * ORDER_THREADS + threadIdx.x;
    order_add(count, c < nc ? key(c) : -1);
  }
  __syncthreads();
  if (threadIdx.x < ORDER_BINS && count[threadIdx.x]) atomicAdd(&bins[threadIdx.x], count[threadIdx.x]);
}

template <class Key>
__global__ void __launch_bounds__(ORDER_THREADS)
k_order_place(int64_t nc, Key key, unsigned int* bins, uint32_t* order) {
  __shared__ unsigned int all[ORDER_BINS], count[ORDER_BINS], base[ORDER_BINS];
  if (threadIdx.x < ORDER_BINS) {
    all[threadIdx.x] = bins[threadIdx.x];
    count[threadIdx.x] = 0;
  }
  __syncthreads();
  const unsigned int n = order_bases(all, base);
  if (threadIdx.x == 0 && blockIdx.x == 0) bins[2 * ORDER_BINS] = n;
  int b[ORDER_PER];
  unsigned int place[ORDER_PER];
#pragma unroll
  for (int i = 0; i < ORDER_PER; i++) {
    const int64_t c = ((int64_t)blockIdx.x * ORDER_PER + i) * ORDER_THREADS + threadIdx.x;
    b[i] = c < nc ? key(c) : -1;
    place[i] = order_add(count, b[i]);
    if (b[i] < 0 && c < nc) key.unlisted(c);
  }
  __syncthreads();
  if (threadIdx.x < ORDER_BINS && count[threadIdx.x])
    base[threadIdx.x] += atomicAdd(&bins[ORDER_BINS + threadIdx.x], count[threadIdx.x]);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < ORDER_PER; i++) {
    const int64_t c = ((int64_t)blockIdx.x * ORDER_PER + i) * ORDER_THREADS + threadIdx.x;
    if (b[i] >= 0) order[base[b[i]] + place[i]] = (uint32_t)c;
  }
}

// order[0 .. bins[2 ORDER_BINS]) = the listed columns, largest key first
template <class Key>
cudaError_t launch_order(int64_t nc, const Key& key, unsigned int* bins, uint32_t* order, cudaStream_t s) {
  if (nc <= ORDER_ONE_MAX) {
    k_order_one<<<1, ORDER_ONE_THREADS, 0, s>>>(nc, key, bins, order);
    return cudaGetLastError();
  }
  const cudaError_t e = cudaMemsetAsync(bins, 0, ORDER_WORDS * sizeof(unsigned int), s);
  if (e != cudaSuccess) return e;
  const unsigned grid = (unsigned)((nc + ORDER_THREADS * ORDER_PER - 1) / (ORDER_THREADS * ORDER_PER));
  k_order_count<<<grid, ORDER_THREADS, 0, s>>>(nc, key, bins);
  k_order_place<<<grid, ORDER_THREADS, 0, s>>>(nc, key, bins, order);
  return cudaGetLastError();
}

}  // namespace clmgb
