// Device helpers shared by the kernels' translation units.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "convert.h"
#include "launch.h"

namespace umcp {
namespace dev {

// Programmatic dependent launch: a kernel launched with programmatic stream
// serialization may start while the kernel before it on the stream runs; it
// waits here, before its first read of that kernel's results (a no-op when it
// was launched without the attribute).
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Lets the kernel after this one be scheduled once every block has come this
// far; it then waits for this kernel's end in grid_dependency_wait. A kernel
// calls it right after its own wait, so that the next one's blocks are up when it
// drains, but only where its grid is small (few_blocks: the most it may have).
// With a large one the next kernel's blocks go wherever this one's leave room
// first: its own blocks end up uneven over the SMs, and other streams' kernels
// lose their place. BD step with / without: 1,280 faces 11.3 / 12.5 us, 16,000
// faces 24.8 / 23.4, 131,072 faces 81 / 64.
constexpr unsigned kFewFaceBlocks = 320, kFewGatherBlocks = 96;
__device__ __forceinline__ void grid_dependents(unsigned few_blocks) {
  if (gridDim.x <= few_blocks) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// A job takes the step when it has neither stopped nor reached its limit.
__device__ __forceinline__ bool job_active(const BatchFaceJob &J) { return !*J.status && J.cnt[1] < J.limit; }

// The precision form's FP32 copies of one position coordinate x = r[i]:
// x = hi + lo to about 2^-48 relative, and dsp = x - r0[i] (the displacement
// from the reference state, rounded once from FP64).
__device__ __forceinline__ void store_f32_position(size_t i, double x, float *__restrict__ hi,
                                                   float *__restrict__ lo, const double *__restrict__ r0,
                                                   float *__restrict__ dsp) {
  const size_t at = pos_at(i);
  convert::to_f32_pair(x, hi[at], lo[at]);
  dsp[at] = convert::to_f32(__dsub_rn(x, r0[i]));
}

// The same for a vertex whose three coordinates one thread has, in the two
// 16-byte stores and the 4-byte one that load_vertex reads (hi: F32Pos::hi).
__device__ __forceinline__ void store_f32_vertex(int v, const double x[3], float *__restrict__ hi,
                                                 const double *__restrict__ r0) {
  float h[3], l[3], d[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    convert::to_f32_pair(x[c], h[c], l[c]);
    d[c] = convert::to_f32(__dsub_rn(x[c], r0[3 * (size_t)v + c]));
  }
  float *q = hi + kPosStride * (size_t)v;
  reinterpret_cast<float4 *>(q)[0] = make_float4(h[0], h[1], h[2], l[0]);
  reinterpret_cast<float4 *>(q)[1] = make_float4(l[1], l[2], d[0], d[1]);
  q[8] = d[2];
}

// Second half of a leapfrog step with M^-1 for coordinate i: r += qdot AK (and
// p reset for BD), and the precision form's FP32 copies (rhi NULL: none).
__device__ __forceinline__ void drift(const StepArgs &a, size_t i, double qdot, double *__restrict__ r,
                                      double *__restrict__ p, float *__restrict__ rhi, float *__restrict__ rlo,
                                      const double *__restrict__ r0, float *__restrict__ dsp) {
  const double x = __dadd_rn(r[i], __dmul_rn(qdot, a.AK));
  r[i] = x;
  if (a.kind == 1) p[i] = 0.0;
  if (rhi) store_f32_position(i, x, rhi, rlo, r0, dsp);
}

// Sum of q over the warp in a fixed (xor-tree) order.
__device__ __forceinline__ double warp_sum(double q) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) q += __shfl_xor_sync(0xFFFFFFFFu, q, off);
  return q;
}

// Fixed-order sum of the block partials, done by one block of NT threads: each
// warp takes a quantity at a time, its lanes every 32nd row, then an xor tree.
// (With a thread per row and a shared-memory tree over the block, every FP64
// add of the tree cost a warp instruction for a few active lanes.) Writes E,
// its parts and dE/dalpha; in a run also records E, flags non-finite or
// diverging energies (src/hd.C:1280-1305) and advances the run index. The
// box-scale sums are formed only where the caller takes them.
template <int NT>
__device__ void finish_sums(const FinishArgs &F, const double *__restrict__ blockpart) {
  __shared__ double tot[6];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nq = F.galpha ? 6 : 3;
  for (int q = warp; q < nq; q += NT / 32) {
    double a = 0;
    for (int b = lane; b < F.nblk; b += 32) a += __ldcg(&blockpart[6 * (size_t)b + q]);
    a = warp_sum(a);
    if (lane == 0) tot[q] = a;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double e = tot[0] + tot[1] + tot[2];
    if (F.gterm) e += F.gterm[kGeoE];  // the global restraints, summed before the face pass
    if (F.E) F.E[0] = e;
    if (F.parts) { F.parts[0] = tot[0]; F.parts[1] = tot[1]; F.parts[2] = tot[2]; }
    if (F.galpha)
      for (int c = 0; c < 3; ++c) {
        const double d = tot[3 + c] + (F.gterm ? F.gterm[kGeoDAlpha + c] : 0.0);
        F.galpha[c] = F.store_galpha ? d : F.galpha[c] + d;
      }
    if (!isfinite(e)) atomicOr(F.status, kStatusNonFinite);
    if (F.host_status) *F.host_status = atomicOr(F.status, 0);
    if (F.energies) {
      const uint64_t idx = F.cnt[1];
      F.energies[idx] = e;
      if (F.threshold > 0 && idx > 0 && e - F.energies[idx - 1] > F.threshold) atomicOr(F.status, kStatusDiverged);
      F.cnt[1] = idx + 1;
    }
  }
}

// The end of a face launch's block that has written its row of block partials:
// it counts on F.done, and the block that completes the pass's count sums the
// rows (the order of that sum does not depend on which block it is).
template <int NT>
__device__ __forceinline__ void count_and_finish(const FinishArgs &F, const double *__restrict__ blockpart) {
  if (!F.done) return;
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = (atomicAdd(F.done, 1u) == (unsigned)F.nblk - 1u);
  __syncthreads();
  if (!last) return;
  __threadfence();
  finish_sums<NT>(F, blockpart);
  if (threadIdx.x == 0) *F.done = 0u;
}

}  // namespace dev
}  // namespace umcp
