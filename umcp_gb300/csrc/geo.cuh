// Helpers shared by the area and volume kernels (surface_kernels.cu, geo32.cu).
#pragma once
#include "launch.h"

namespace umcp {
namespace dev {

template <typename T>
__device__ __forceinline__ void cross3(const T a[3], const T b[3], T o[3]) {
  o[0] = a[1] * b[2] - a[2] * b[1];
  o[1] = a[2] * b[0] - a[0] * b[2];
  o[2] = a[0] * b[1] - a[1] * b[0];
}

// The block's sums (red[q][0], word q) to its row; the last block to finish sums
// the rows (in a fixed order) and forms E_r, dE_r/dA, dE_r/dV and dE_r/dalpha.
__device__ inline void geo_finish_rows(const GeoArgs &G, double (*red)[kGeoThreads]) {
  __shared__ bool last;
  if (threadIdx.x < kGeoWords) G.block[(size_t)blockIdx.x * kGeoWords + threadIdx.x] = red[threadIdx.x][0];
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = (atomicAdd(G.done, 1u) == gridDim.x - 1);
  __syncthreads();
  if (!last) return;
  __threadfence();
  // Fixed-order sum of the block rows by the whole block: thread (i, q) sums word q
  // of rows i, i + 16, ..., and the 16 sums of a word are added in order. (One
  // thread a word is a chain of loads from L2: 27 us for 640 rows, a restrained evaluation
  // of a 40,962-vertex vesicle alone 206 -> 179 us.)
  static_assert(kGeoThreads % kGeoWords == 0, "a thread per word and row class");
  constexpr int kClasses = kGeoThreads / kGeoWords;
  const int q = threadIdx.x % kGeoWords, i = threadIdx.x / kGeoWords;
  double t = 0;
#pragma unroll 8
  for (unsigned b = i; b < gridDim.x; b += kClasses) t += __ldcg(&G.block[(size_t)b * kGeoWords + q]);
  red[q][i] = t;
  __syncthreads();
  if (i == 0) {
    for (int k = 1; k < kClasses; ++k) t += red[q][k];
    red[q][0] = t;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const double A = red[0][0], V = red[1][0];
    const double cA = G.A0 > 0 ? G.KA * (A - G.A0) / G.A0 : 0.0, cV = G.KV * (V - G.V0);
    G.gterm[kGeoA] = A;
    G.gterm[kGeoV] = V;
    G.gterm[kGeoE] = (G.A0 > 0 ? 0.5 * G.KA * (A - G.A0) * (A - G.A0) / G.A0 : 0.0) + 0.5 * G.KV * (V - G.V0) * (V - G.V0);
    G.gterm[kGeoCA] = cA;
    G.gterm[kGeoCV] = cV;
    for (int k = 0; k < 3; ++k) G.gterm[kGeoDAlpha + k] = cA * red[2 + k][0] + cV * red[5 + k][0];
    *G.done = 0u;
  }
}

// Block sums of the per-thread accumulators in a fixed order, then the rows.
__device__ inline void geo_finish(const GeoArgs &G, const double acc[kGeoWords], double (*red)[kGeoThreads]) {
#pragma unroll
  for (int q = 0; q < kGeoWords; ++q) red[q][threadIdx.x] = acc[q];
  __syncthreads();
  for (int w = kGeoThreads / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w)
#pragma unroll
      for (int q = 0; q < kGeoWords; ++q) red[q][threadIdx.x] += red[q][threadIdx.x + w];
    __syncthreads();
  }
  geo_finish_rows(G, red);
}
}  // namespace dev
}  // namespace umcp
