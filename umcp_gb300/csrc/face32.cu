// Kernels of the precision form's half-warp face pass (face32.cuh) and their
// launches: any of a mesh's patch types in one launch, and a batch's tiles of
// one irregular patch type.
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_common.cuh"
#include "face32.cuh"
#include "launch.h"
#include "launch_host.h"

namespace umcp {
namespace dev {
namespace f32 {

constexpr size_t kSmemBytes = sizeof(Smem<13, 16>);
static_assert(kSmemBytes >= sizeof(Smem<12, 15>) && kSmemBytes >= sizeof(Smem<11, 16>), "largest patch type");
constexpr int kMinBlocks = 4;

// Faces [first, end) by this block's warps, two at a time, from pair `pair` in
// strides of `stride` pairs.
template <int NCP, int NPT, bool KG_REG, bool GEO>
__device__ __forceinline__ void faces(Smem<NCP, NPT> &sm, const FaceSrc &S, const SurfaceParams &P, int first, int end,
                                      int pair, int stride, double w, double dudv, bool want_da,
                                      float *__restrict__ partial, KahanSums<6> &sums) {
  const int hw = threadIdx.x >> 4, lane = threadIdx.x & 15, half = hw & 1;
  const double *r = S.r + 3 * (size_t)P.nv;
  const float alpha[3] = {(float)r[0], (float)r[1], (float)r[2]};
  const float am1[3] = {(float)(r[0] - 1.0), (float)(r[1] - 1.0), (float)(r[2] - 1.0)};
  const Coef M = point_coef(P, w, dudv);
  const float k_reg = (float)P.k_reg;
  const bool reg_alpha = KG_REG && NCP != 12 && P.k_reg != 0.0;
  Ahead cur, nxt;
  int f = first + 2 * pair;  // the pair's first face (uniform over the warp)
  if (f < end) load<NCP, NPT, KG_REG>(S, f + half, end, lane, cur);
  for (; f < end; f += 2 * stride) {
    const int fn = f + 2 * stride;
    if (fn < end) load<NCP, NPT, KG_REG>(S, fn + half, end, lane, nxt);
    face<NCP, NPT, KG_REG, GEO>(sm, hw, lane, cur, P, alpha, am1, M, k_reg, reg_alpha, want_da, partial, sums);
    cur = nxt;
  }
}

// Block sums of n per-lane sums in a fixed order into out[n]: energies times e_scale
// (SurfaceParams), box-scale derivatives over alpha.
__device__ __forceinline__ void block_row(double (*red)[6], const KahanSums<6> &sums, const double *e_scale,
                                          const double *alpha, int n, double *out) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    if (q >= n) break;
    const double s = warp_sum(sums.s[q], sums.c[q]);
    if (lane == 0) red[warp][q] = s;
  }
  __syncthreads();
  if ((int)threadIdx.x < n) {
    double s = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) s += red[w][threadIdx.x];
    out[threadIdx.x] = threadIdx.x < 3 ? s * e_scale[threadIdx.x] : s / alpha[threadIdx.x - 3];
  }
}

template <int NCP, int NPT>
__device__ __forceinline__ void group(void *raw, const FaceGroup32 &G, int block, const SurfaceParams &P,
                                      const double *__restrict__ r, const F32View &f, float *__restrict__ partial,
                                      double *__restrict__ row, bool want_da, const double *__restrict__ gterm) {
  Smem<NCP, NPT> &sm = *reinterpret_cast<Smem<NCP, NPT> *>(raw);
  const double w = stage(sm, G.table);
  if (gterm)  // restraints
    for (int i = threadIdx.x; i < NCP * F32Table<NCP, NPT>::NC4; i += kThreads)
      (&sm.M[0][0])[i] = __ldg(reinterpret_cast<const float4 *>(G.table + F32Table<NCP, NPT>::kCorner) + i);
  __syncthreads();
  grid_dependency_wait();  // the state comes from the kernels before
  grid_dependents(kFewFaceBlocks);
  FaceSrc S{};
  S.cp = G.cp; S.g0f = G.g0; S.rr0f = G.rr0; S.compf = G.comp; S.dest = G.dest;
  S.r = r; S.rhi = f.hi; S.rlo = f.lo; S.dsp = f.dsp;
  KahanSums<6> sums;
  const int pair = block * kWarps + (threadIdx.x >> 5), stride = G.nblocks * kWarps;
  const bool kg_reg = P.kg != 0.0 || P.k_reg != 0.0;
  if (gterm) {  // restraints: their coefficients come from the sums kernel
    if (threadIdx.x < NPT) sm.geo[threadIdx.x] = geo_coef(gterm, w, G.dudv);
    if (threadIdx.x == 0) sm.cV = (float)gterm[kGeoCV];
    __syncthreads();
    if (kg_reg) faces<NCP, NPT, true, true>(sm, S, P, 0, G.nfaces, pair, stride, w, G.dudv, want_da, partial, sums);
    else faces<NCP, NPT, false, true>(sm, S, P, 0, G.nfaces, pair, stride, w, G.dudv, want_da, partial, sums);
  } else {
    if (kg_reg) faces<NCP, NPT, true, false>(sm, S, P, 0, G.nfaces, pair, stride, w, G.dudv, want_da, partial, sums);
    else faces<NCP, NPT, false, false>(sm, S, P, 0, G.nfaces, pair, stride, w, G.dudv, want_da, partial, sums);
  }
  block_row(sm.red, sums, P.e_scale[NCP != 12], r + 3 * (size_t)P.nv, want_da ? 6 : 3, row);
}

}  // namespace f32

// Block b of the launch takes the group whose blocks include b, counted from
// the launch's end, so that the few irregular faces start first; it writes the
// block-partial row of its place in its group.
__global__ void __launch_bounds__(f32::kThreads, f32::kMinBlocks)
    face32_kernel(const __grid_constant__ FaceSet32 F, const __grid_constant__ SurfaceParams P,
                  const double *__restrict__ r, F32View f, float *__restrict__ partial, double *__restrict__ blockpart,
                  FinishArgs fin) {
  __shared__ alignas(16) unsigned char raw[f32::kSmemBytes];
  int b = gridDim.x - 1 - blockIdx.x, k = 0;
  while (k + 1 < F.ngroups && b >= F.g[k].nblocks) b -= F.g[k++].nblocks;
  const FaceGroup32 &G = F.g[k];
  double *row = blockpart + 6 * (size_t)(G.block_base + b);
  const bool want_da = fin.galpha != nullptr;  // a run's steps leave the box scales alone
  const double *gterm = F.geo ? fin.gterm : nullptr;
  if (G.ncp == 12) f32::group<12, 15>(raw, G, b, P, r, f, partial, row, want_da, gterm);
  else if (G.ncp == 11) f32::group<11, 16>(raw, G, b, P, r, f, partial, row, want_da, gterm);
  else f32::group<13, 16>(raw, G, b, P, r, f, partial, row, want_da, gterm);
  count_and_finish<f32::kThreads>(fin, blockpart);
}

// Batch: a block takes tiles of one patch type in turn (persistent grid) and
// writes each tile's three energy sums.
template <int NCP, int NPT>
__global__ void __launch_bounds__(f32::kThreads, f32::kMinBlocks)
    batch_face32_kernel(const BatchJob *__restrict__ jobs, int group, const BatchTile *__restrict__ tiles,
                        const int *__restrict__ counts, const float *__restrict__ table, double dudv,
                        double *__restrict__ tile_sums) {
  using namespace f32;
  __shared__ Smem<NCP, NPT> sm;
  __shared__ BatchFaceJob sj;
  __shared__ int s_active;
  const int ntiles = counts[group], tile_base = counts[3 + group];
  if ((int)blockIdx.x >= ntiles) return;
  const double w = stage(sm, table);
  int job = -1;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const BatchTile tile = tiles[tile_base + t];
    __syncthreads();  // the previous tile's readers of sj and sm.red are done
    if (tile.job != job) {
      const int *src = reinterpret_cast<const int *>(&jobs[tile.job].f);
      int *dst = reinterpret_cast<int *>(&sj);
      for (int i = threadIdx.x; i < (int)(sizeof(BatchFaceJob) / sizeof(int)); i += kThreads) dst[i] = src[i];
      if (threadIdx.x == 0) s_active = job_active(jobs[tile.job].f);
      job = tile.job;
      __syncthreads();
    }
    KahanSums<6> sums;
    if (s_active) {
      const FaceSrc &src = sj.src[group];
      const int pair = threadIdx.x >> 5, end = tile.first + tile.count;
      if (sj.P.kg != 0.0 || sj.P.k_reg != 0.0)
        faces<NCP, NPT, true, false>(sm, src, sj.P, tile.first, end, pair, kWarps, w, dudv, false, (float *)sj.partial, sums);
      else
        faces<NCP, NPT, false, false>(sm, src, sj.P, tile.first, end, pair, kWarps, w, dudv, false, (float *)sj.partial, sums);
    }
    block_row(sm.red, sums, sj.P.e_scale[1], nullptr, 3, tile_sums + 3 * (size_t)(tile_base + t));
  }
}

}  // namespace dev

int face_blocks32(int nfaces) {
  if (nfaces <= 0) return 0;
  // A group's persistent grid: at most as many blocks as fit on the device at once (a
  // fixed number per device, so the face-to-block assignment and the sums' order are
  // fixed). A launch takes the groups' grids together: on a mesh whose regular group
  // fills the device, the irregular groups' few blocks make a second wave.
  static PerDevice pd;
  const int cached = per_device(pd, [] {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, dev::face32_kernel, dev::f32::kThreads, 0);
    return sm_count() * (per_sm > 0 ? per_sm : 1);
  });
  const int need = grid_for(nfaces, dev::f32::kHW);
  return need < cached ? need : cached;
}

cudaError_t launch_faces32(const FaceSet32 &F, const dev::SurfaceParams &P, const double *r, const F32Pos &f,
                           float *partial, double *blockpart, const FinishArgs &fin, cudaStream_t s, bool chained) {
  int grid = 0;
  for (int k = 0; k < F.ngroups; ++k) {
    if (F.g[k].nfaces > 0 && F.g[k].ncp != 11 && F.g[k].ncp != 12 && F.g[k].ncp != 13) return cudaErrorInvalidValue;
    grid += F.g[k].nblocks;
  }
  if (!grid) return cudaSuccess;
  if (!f.hi || !f.lo || !f.dsp) return cudaErrorInvalidValue;
  const F32View view{f.hi, f.lo, f.dsp};
  if (chained) return launch_after(dev::face32_kernel, grid, dev::f32::kThreads, 0, s, F, P, r, view, partial, blockpart, fin);
  dev::face32_kernel<<<grid, dev::f32::kThreads, 0, s>>>(F, P, r, view, partial, blockpart, fin);
  return cudaGetLastError();
}

int batch_face_blocks32(int ncp) {
  static PerDevice pd[2];
  auto blocks = [](auto kernel) {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, dev::f32::kThreads, 0);
    return sm_count() * (per_sm > 0 ? per_sm : 1);
  };
  if (ncp == 11) return per_device(pd[0], [&] { return blocks(dev::batch_face32_kernel<11, 16>); });
  return per_device(pd[1], [&] { return blocks(dev::batch_face32_kernel<13, 16>); });
}

cudaError_t launch_batch_faces32(const BatchJob *jobs, int group, const BatchTile *tiles, const int *counts,
                                 const float *table, int ncp, double dudv, double *tile_sums, int grid,
                                 cudaStream_t s) {
  constexpr int NT = dev::f32::kThreads;
  if (ncp == 11)
    dev::batch_face32_kernel<11, 16><<<grid, NT, 0, s>>>(jobs, group, tiles, counts, table, dudv, tile_sums);
  else if (ncp == 13)
    dev::batch_face32_kernel<13, 16><<<grid, NT, 0, s>>>(jobs, group, tiles, counts, table, dudv, tile_sums);
  else
    return cudaErrorInvalidValue;
  return cudaGetLastError();
}

}  // namespace umcp
