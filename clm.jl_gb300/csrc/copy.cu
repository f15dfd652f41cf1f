// copy.cu — many device arrays copied in one launch.
//
// A trajectory's reverse copies states of some 70 arrays of 16 KB to a few MB; a copy each is
// bound by launching them (16,384 columns: 64 copies of 2.2 us on the device and twice that
// on the host; this launch 29 us).  A block takes COPY_TILE bytes of one array, found in the
// table of the arrays' first tiles; 16 bytes a load where both ends allow it, single bytes
// otherwise.
#include "clmgb_device.cuh"
#include "launch.h"

namespace clmgb {

namespace {

constexpr int COPY_THREADS = 256, COPY_UNROLL = 4;
constexpr int64_t COPY_TILE = (int64_t)COPY_THREADS * COPY_UNROLL * 16;

struct CopyTable {
  unsigned char* dst[COPY_MAX];
  const unsigned char* src[COPY_MAX];
  int64_t bytes[COPY_MAX];
  uint32_t first[COPY_MAX + 1];                     // an array's first tile
  int n;
};

__global__ void __launch_bounds__(COPY_THREADS)
k_copy_arrays(const __grid_constant__ CopyTable t) {
  int lo = 0, hi = t.n;                             // first[lo] <= blockIdx.x < first[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) / 2;
    if (t.first[mid] <= blockIdx.x) lo = mid;
    else hi = mid;
  }
  const int64_t at = (int64_t)(blockIdx.x - t.first[lo]) * COPY_TILE;
  unsigned char* const dst = t.dst[lo] + at;
  const unsigned char* const src = t.src[lo] + at;
  const int64_t left = t.bytes[lo] - at, len = left < COPY_TILE ? left : COPY_TILE;
  int64_t done = 0;
  if ((((uintptr_t)dst | (uintptr_t)src) & 15) == 0) {
    const int words = (int)(len / 16);
    uint4 v[COPY_UNROLL];
#pragma unroll
    for (int i = 0; i < COPY_UNROLL; i++) {
      const int w = i * COPY_THREADS + threadIdx.x;
      if (w < words) v[i] = reinterpret_cast<const uint4*>(src)[w];
    }
#pragma unroll
    for (int i = 0; i < COPY_UNROLL; i++) {
      const int w = i * COPY_THREADS + threadIdx.x;
      if (w < words) reinterpret_cast<uint4*>(dst)[w] = v[i];
    }
    done = (int64_t)words * 16;
  }
  for (int64_t b = done + threadIdx.x; b < len; b += COPY_THREADS) dst[b] = src[b];
}

}  // namespace

cudaError_t launch_copy_arrays(int n, void* const* dst, const void* const* src, const int64_t* bytes, cudaStream_t s) {
  for (int at = 0; at < n;) {
    CopyTable t;
    uint64_t tiles = 0;
    for (t.n = 0; at < n && t.n < COPY_MAX; at++) {
      const uint64_t more = (uint64_t)((bytes[at] + COPY_TILE - 1) / COPY_TILE);
      if (tiles + more > 0x7fffffffu) {
        if (t.n == 0) return cudaErrorInvalidValue;
        break;
      }
      if (more == 0 || dst[at] == src[at]) continue;
      t.dst[t.n] = (unsigned char*)dst[at];
      t.src[t.n] = (const unsigned char*)src[at];
      t.bytes[t.n] = bytes[at];
      t.first[t.n++] = (uint32_t)tiles;
      tiles += more;
    }
    if (t.n == 0) continue;
    t.first[t.n] = (uint32_t)tiles;
    k_copy_arrays<<<(unsigned)tiles, COPY_THREADS, 0, s>>>(t);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace clmgb
