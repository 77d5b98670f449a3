// Kernels of the FP64 face pass (face64.cuh) and their launches: a single
// mesh's faces of every patch type in one launch, and a batch's tiles.
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_common.cuh"
#include "face64.cuh"
#include "launch.h"
#include "launch_host.h"

namespace umcp {
namespace dev {
namespace f64 {

// Bytes of the largest patch type's shared memory.
constexpr size_t kSmemBytes = sizeof(Smem<13, 16>);
static_assert(kSmemBytes >= sizeof(Smem<12, 15>) && kSmemBytes >= sizeof(Smem<11, 16>), "largest patch type");
// Blocks per SM the registers are capped for (168 a thread): three warps a
// scheduler, so that one warp's integer contractions run beside another's FP64.
// (Four spill.)
constexpr int kMinBlocks = 3;

// Sum of q over each warp's lanes into red[warp][i], then over the block into out.
__device__ __forceinline__ void block_row(double (*red)[6], const double *v, int n, double *out) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int q = 0; q < n; ++q) {
    const double s = warp_sum(v[q]);
    if (lane == 0) red[warp][q] = s;
  }
  __syncthreads();
  if ((int)threadIdx.x < n) {
    double s = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) s += red[w][threadIdx.x];
    out[threadIdx.x] = s;
  }
}

// Faces [first, end) by this block's warps, two at a time, from pair `pair` in
// strides of `stride` pairs.
template <int NCP, int NPT, bool KG_REG>
__device__ __forceinline__ void faces(Smem<NCP, NPT> &sm, const FaceSrc &S, const SurfaceParams &P, int first, int end,
                                      int pair, int stride, const int eb[5], double weight, double dudv, bool irregular,
                                      bool want_da, double *__restrict__ partial, Sums &sums) {
  const int hw = threadIdx.x >> 4, lane = threadIdx.x & 15, half = hw & 1;
  const double *r = S.r;
  const double alpha[3] = {r[3 * P.nv], r[3 * P.nv + 1], r[3 * P.nv + 2]};
  const bool unit = alpha[0] == 1.0 && alpha[1] == 1.0 && alpha[2] == 1.0;
  const double am1[3] = {alpha[0] - 1.0, alpha[1] - 1.0, alpha[2] - 1.0};
  const PointCoef C(P, weight, dudv);
  const bool reg_alpha = KG_REG && irregular && P.k_reg != 0.0 && want_da;
  Ahead cur, nxt;
  int f = first + 2 * pair;  // the pair's first face (uniform over the warp)
  if (f < end) load<NCP, NPT, KG_REG>(S, P, f + half, end, lane, cur);
  for (; f < end; f += 2 * stride) {
    const int fn = f + 2 * stride;
    if (fn < end) load<NCP, NPT, KG_REG>(S, P, fn + half, end, lane, nxt);
    face<NCP, NPT, KG_REG>(sm, hw, lane, eb, cur, alpha, am1, unit, C, reg_alpha, want_da, partial, sums);
    cur = nxt;
  }
  if (want_da)
#pragma unroll
    for (int c = 0; c < 3; ++c) sums.da[c] /= alpha[c];
}

template <int NCP, int NPT>
__device__ __forceinline__ void group(void *raw, const FaceGroup64 &G, int block, const SurfaceParams &P,
                                      const double *__restrict__ r, double *__restrict__ partial,
                                      double *__restrict__ row, bool want_da, bool chain) {
  Smem<NCP, NPT> &sm = *reinterpret_cast<Smem<NCP, NPT> *>(raw);
  int eb[5];
  stage(sm, G.table, eb);
  const int lane = threadIdx.x & 15;
  const double w = lane < NPT ? __ldg(G.weight + lane) : 0.0;
  __syncthreads();
  grid_dependency_wait();  // the state comes from the kernels before
  if (chain) grid_dependents(kFewFaceBlocks);
  FaceSrc S{};
  S.cp = G.cp; S.g0 = G.g0; S.rr0 = G.rr0; S.comp = G.comp; S.dest = G.dest; S.r = r;
  Sums sums;
  const int pair = block * kWarps + (threadIdx.x >> 5), stride = G.nblocks * kWarps;
  if (P.kg != 0.0 || P.k_reg != 0.0)
    faces<NCP, NPT, true>(sm, S, P, 0, G.nfaces, pair, stride, eb, w, G.dudv, NCP != 12, want_da, partial, sums);
  else
    faces<NCP, NPT, false>(sm, S, P, 0, G.nfaces, pair, stride, eb, w, G.dudv, NCP != 12, want_da, partial, sums);
  const double v[6] = {sums.ea, sums.ec, sums.er, sums.da[0], sums.da[1], sums.da[2]};
  block_row(sm.red, v, want_da ? 6 : 3, row);
}

}  // namespace f64

// Single mesh, FP64: every patch type's faces in one launch. Block b writes the
// block-partial row b; the groups' blocks follow one another in reverse, so
// that the few irregular ones start first.
__global__ void __launch_bounds__(f64::kThreads, f64::kMinBlocks)
    face64_kernel(const __grid_constant__ FaceSet64 F, const __grid_constant__ SurfaceParams P,
                  const double *__restrict__ r, double *__restrict__ partial, double *__restrict__ blockpart,
                  FinishArgs fin) {
  __shared__ alignas(16) unsigned char raw[f64::kSmemBytes];
  const int b = gridDim.x - 1 - blockIdx.x;
  int k = 0;
  while (k + 1 < F.ngroups && b >= F.g[k + 1].block_base) ++k;
  const FaceGroup64 &G = F.g[k];
  double *row = blockpart + 6 * (size_t)b;
  const bool want_da = fin.galpha != nullptr;  // a run's steps leave the box scales alone
  // With restraints the next kernel is their gradient pass, which the FP64 pipe bounds
  // too: started early its blocks gather on the SMs that this one's leave first (a
  // restrained evaluation of a 642-vertex vesicle 437 us, 139 without).
  const bool chain = fin.gterm == nullptr;
  if (G.ncp == 12) f64::group<12, 15>(raw, G, b - G.block_base, P, r, partial, row, want_da, chain);
  else if (G.ncp == 11) f64::group<11, 16>(raw, G, b - G.block_base, P, r, partial, row, want_da, chain);
  else f64::group<13, 16>(raw, G, b - G.block_base, P, r, partial, row, want_da, chain);
  count_and_finish<f64::kThreads>(fin, blockpart);
}

// Batch, FP64, one patch type: a block takes tiles in turn (persistent grid)
// and writes each tile's three energy sums.
template <int NCP, int NPT>
__global__ void __launch_bounds__(f64::kThreads, f64::kMinBlocks)
    batch_face64_kernel(const BatchJob *__restrict__ jobs, int group, const BatchTile *__restrict__ tiles,
                        const int *__restrict__ counts, const int *__restrict__ table,
                        const double *__restrict__ weight, double dudv, double *__restrict__ tile_sums) {
  using namespace f64;
  __shared__ Smem<NCP, NPT> sm;
  __shared__ BatchFaceJob sj;
  __shared__ int s_active;
  const int ntiles = counts[group], tile_base = counts[3 + group];
  if ((int)blockIdx.x >= ntiles) return;
  int eb[5];
  stage(sm, table, eb);
  const int lane = threadIdx.x & 15;
  const double w = lane < NPT ? __ldg(weight + lane) : 0.0;
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
    Sums sums;
    if (s_active) {
      const FaceSrc &src = sj.src[group];
      const int pair = threadIdx.x >> 5, end = tile.first + tile.count;
      if (sj.P.kg != 0.0 || sj.P.k_reg != 0.0)
        faces<NCP, NPT, true>(sm, src, sj.P, tile.first, end, pair, kWarps, eb, w, dudv, NCP != 12, false,
                              (double *)sj.partial, sums);
      else
        faces<NCP, NPT, false>(sm, src, sj.P, tile.first, end, pair, kWarps, eb, w, dudv, NCP != 12, false,
                               (double *)sj.partial, sums);
    }
    const double v[3] = {sums.ea, sums.ec, sums.er};
    block_row(sm.red, v, 3, tile_sums + 3 * (size_t)(tile_base + t));
  }
}

}  // namespace dev

int face_blocks64(int nfaces) {
  if (nfaces <= 0) return 0;
  // A group's persistent grid: at most as many blocks as fit on the device at once (a
  // fixed number per device, so the face-to-block assignment and the sums' order are
  // fixed). A launch takes the groups' grids together: on a mesh whose regular group
  // fills the device, the irregular groups' few blocks make a second wave.
  static PerDevice pd;
  const int cached = per_device(pd, [] {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, dev::face64_kernel, dev::f64::kThreads, 0);
    return sm_count() * (per_sm > 0 ? per_sm : 1);
  });
  const int need = grid_for(nfaces, dev::f64::kHW);
  return need < cached ? need : cached;
}

cudaError_t launch_faces64(const FaceSet64 &F, const dev::SurfaceParams &P, const double *r, double *partial,
                           double *blockpart, const FinishArgs &fin, cudaStream_t s) {
  int grid = 0;
  for (int k = 0; k < F.ngroups; ++k) {
    if (F.g[k].nfaces > 0 && F.g[k].ncp != 11 && F.g[k].ncp != 12 && F.g[k].ncp != 13) return cudaErrorInvalidValue;
    grid += F.g[k].nblocks;
  }
  if (!grid) return cudaSuccess;
  return launch_after(dev::face64_kernel, grid, dev::f64::kThreads, 0, s, F, P, r, partial, blockpart, fin);
}

int batch_face_blocks64(int ncp) {
  static PerDevice pd[3];
  auto blocks = [](auto kernel) {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, dev::f64::kThreads, 0);
    return sm_count() * (per_sm > 0 ? per_sm : 1);
  };
  if (ncp == 12) return per_device(pd[0], [&] { return blocks(dev::batch_face64_kernel<12, 15>); });
  if (ncp == 11) return per_device(pd[1], [&] { return blocks(dev::batch_face64_kernel<11, 16>); });
  return per_device(pd[2], [&] { return blocks(dev::batch_face64_kernel<13, 16>); });
}

cudaError_t launch_batch_faces64(const BatchJob *jobs, int group, const BatchTile *tiles, const int *counts,
                                 const int *table, const double *weight, int ncp, double dudv, double *tile_sums,
                                 int grid, cudaStream_t s) {
  constexpr int NT = dev::f64::kThreads;
  if (ncp == 12)
    dev::batch_face64_kernel<12, 15><<<grid, NT, 0, s>>>(jobs, group, tiles, counts, table, weight, dudv, tile_sums);
  else if (ncp == 11)
    dev::batch_face64_kernel<11, 16><<<grid, NT, 0, s>>>(jobs, group, tiles, counts, table, weight, dudv, tile_sums);
  else if (ncp == 13)
    dev::batch_face64_kernel<13, 16><<<grid, NT, 0, s>>>(jobs, group, tiles, counts, table, weight, dudv, tile_sums);
  else
    return cudaErrorInvalidValue;
  return cudaGetLastError();
}

}  // namespace umcp
