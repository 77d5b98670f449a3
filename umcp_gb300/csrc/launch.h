// Launch wrappers of the device kernels (surface_kernels.cu). Plain pointers;
// all work is queued on the given stream.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "face32_table.h"
#include "geo32_table.h"
#include "kernels.cuh"

namespace umcp {

// Status bits written by kernels into the mesh's device status word.
enum : int { kStatusNonFinite = 1, kStatusDiverged = 2, kStatusTimeout = 4 };

// Where and how the block partials of a face pass are summed (dev::count_and_finish).
// done: device counter of finished blocks, zero between launches; when non-null,
// the last block of the pass's face launches does the sum.
struct FinishArgs {
  int nblk;            // block-partial rows to sum: every block of every face launch of the pass, each of
                       // which counts on `done`; the block that brings it to nblk sums the rows
  double *E, *parts, *galpha;
  double *energies;    // run only: energies[cnt[1]] = E, cnt[1] += 1
  uint64_t *cnt;
  double threshold;    // energy rise that flags divergence (<= 0: off)
  int *status;
  unsigned *done;
  const double *gterm; // global restraint terms to add (NULL: none), see GeoArgs
  int *host_status;    // page-locked host word that receives the status (NULL: none)
  int store_galpha;    // galpha is overwritten instead of added to
};

// Global area and volume of the limit surface and their restraint, over every patch
// type (the plain path in FP64, a half-warp per face: geo_sums_kernel; the precision
// form with V beyond FP32, four warps per 32 faces: geo32.cu):
//   A = sum dudv w |Ru x Rv|,  V = 1/3 sum dudv w R.(Ru x Rv)
//   E_r = 1/2 K_A (A-A0)^2/A0 + 1/2 K_V (V-V0)^2
// gterm receives {A, V, E_r, dE_r/dA, dE_r/dV, dE_r/dalpha_xyz}.
struct GeoGroup {
  const uint32_t *cp;      // [nfaces][ncp] packed control points
  const int *dest;         // [nfaces][ncp] gradient-partial slots
  const double *basis;     // [npt][5][ncpp] rows u,v,uu,uv,vv
  const double *basis_w;   // [npt][ncp] value rows
  const double *weight;    // [npt]
  const void *tab;         // the precision form's rows: GeoRows<geo_padded(ncp)> (geo32_table.h)
  int ncp, npt, ncpp, nfaces, face_base;
  double dudv;
};
enum : int { kGeoA = 0, kGeoV, kGeoE, kGeoCA, kGeoCV, kGeoDAlpha, kGeoWords = 8 };
struct GeoArgs {
  GeoGroup g[3];
  int ngroups, nfaces, nv;
  const double *r;
  const float *rhi, *rlo;  // r = hi + lo (precision form)
  double box[3][3];
  float box_hi[3][3], box_lo[3][3];
  double KA, A0, KV, V0;
  double *block;           // [blocks][8] partial sums
  double *gterm;           // kGeoWords
  unsigned *done;          // finished-block counter (zero between launches)
};
constexpr int kGeoThreads = 128;
// Fixed grid (a function of the face count only, so every sum has a fixed order).
inline int geo_blocks(int nfaces) {
  const int b = nfaces > 0 ? (nfaces + 4 * (kGeoThreads / 16) - 1) / (4 * (kGeoThreads / 16)) : 1;  // >= 4 faces per half-warp
  return b < 152 * 8 ? b : 152 * 8;
}
// Sums A, V and their alpha derivatives; the last block writes gterm. The plain
// path, in FP64 throughout. staged: launch_stage_in comes before (a host call).
cudaError_t launch_geo_sums(const GeoArgs &G, bool staged, cudaStream_t s);
// The precision form (geo32.cu). fused: the face launches form the restraints' gradient (and with it dE_r/dalpha, which gterm then
// has as zero): its SIMT kernels.
cudaError_t launch_geo_sums32(const GeoArgs &G, bool fused, cudaStream_t s);
// partial[slot] += alpha * (dE_r/dA dA/dX + dE_r/dV dV/dX) for every (face, control point).
template <typename T>
cudaError_t launch_geo_grad(const GeoArgs &G, T *partial, cudaStream_t s);

// The precision form's FP32 copies of the positions (all NULL in the plain
// path): r = hi + lo to about 2^-48 relative, and dsp = r - r0, the
// displacement from the reference state r0 (setg0's state), rounded once.
// The face kernels form the area strain from dsp (f32::point).
struct F32Pos {
  float *hi = nullptr, *lo = nullptr;
  const double *r0 = nullptr;
  float *dsp = nullptr;
};

// The FP64 face pass (face64.cu): every patch type of a mesh in one launch. A
// group's blocks write the block-partial rows [block_base, block_base + nblocks),
// the groups' rows following one another from 0.
struct FaceGroup64 {
  const uint32_t *cp;
  const double *g0, *rr0, *comp, *weight;
  const int *dest, *table;  // gradient-partial slots; the patch type's fixed-point rows (fixed64.h)
  double dudv;
  int nfaces, ncp, nblocks, block_base;
};
struct FaceSet64 {
  FaceGroup64 g[3];
  int ngroups;
};
int face_blocks64(int nfaces);
cudaError_t launch_faces64(const FaceSet64 &F, const dev::SurfaceParams &P, const double *r, double *partial,
                           double *blockpart, const FinishArgs &fin, cudaStream_t s);

// The precision form's half-warp face pass (face32.cu): any of a mesh's patch
// types in one launch. partial[dest[f*ncp+x]] receives the alpha-scaled gradient
// of control point x of face f; blockpart[block_base + b] the sums of block b of
// the group, {E_area, E_curvature, E_angle, dE/dalpha_xyz}.
struct FaceGroup32 {
  const uint32_t *cp;
  const float *g0, *rr0, *comp, *table;  // table: face32_table.h
  const int *dest;
  double dudv;
  int nfaces, ncp, nblocks, block_base;
};
struct FaceSet32 {
  FaceGroup32 g[3];
  int ngroups;
  int geo;  // the restraints' gradient goes along (coefficients at FinishArgs::gterm)
};
struct F32View {
  const float *hi, *lo, *dsp;
};
int face_blocks32(int nfaces);
// chained: s's previous kernel is the one whose results it reads (the launch may
// then start while that one drains).
cudaError_t launch_faces32(const FaceSet32 &F, const dev::SurfaceParams &P, const double *r, const F32Pos &f,
                           float *partial, double *blockpart, const FinishArgs &fin, cudaStream_t s, bool chained);

// Regular faces (ncp 12, npt 15) of the precision form, one per thread
// (face_tpf_kernel): the same outputs; the same gradient bits.
// From kTpfFaces faces on. With fewer, a thread per face leaves the schedulers
// one warp each or none, and a face's serial chain (about 14 us) is the pass; a
// half-warp per face shortens it to about 3 us but issues 1.6 times the
// instructions per face. BD step, half-warps against a thread per face: 320
// faces 10.0 / 25 us, 8,192 18.4 / 22.1, 16,000 23.5 / 22.5, 20,400 26.7 / 25.6,
// 32,768 34 / 26.3, 131,072 103 / 65. In between the line lies on the half-warps'
// side of the crossing: with irregular patches beside and three evaluations in
// flight on separate streams, 20,480 faces take 43 against 49 us.
constexpr int kTpfFaces = 24000;
int face_blocks_tpf(int nfaces);
cudaError_t launch_faces_tpf(const TpfRows &rows, const dev::FaceLaunch &L, const int *dest,
                             const dev::SurfaceParams &P, const double *r, const F32Pos &f, float *partial,
                             double *blockpart, int *status, int grid, const FinishArgs &fin, int geo, cudaStream_t s);

// The regular faces of the precision form on the tensor cores (face_tc_kernel):
// the same outputs as launch_faces_tpf, in 128-face tiles; grid from
// face_blocks_tc.
int face_blocks_tc(int nfaces);
cudaError_t launch_faces_tc(const dev::FaceLaunch &L, const int *dest, const dev::SurfaceParams &P, const double *r,
                            const float *rhi, const float *rlo, const float *dsp, float *partial, double *blockpart,
                            int *status, int grid, const FinishArgs &fin, cudaStream_t s);

// The precision form's FP32 positions of r: f.hi[i] + f.lo[i] = r[i] to about
// 2^-48 relative, f.dsp[i] = r[i] - f.r0[i].
cudaError_t launch_split_positions(int n, const double *r, const F32Pos &f, cudaStream_t s);

// *dst |= *src on the device (one thread).
cudaError_t launch_status_merge(const int *src, int *dst, cudaStream_t s);

// Per vertex: g[3v+c] += (store: =) sum of its partial slots off[2v] + 32 k, k <
// off[2v+1] (32 vertices interleaved per group, see interleave_slots).
template <typename T>
cudaError_t launch_gather(int nv, const T *partial, const int *off, double *g, int store, cudaStream_t s);

// A host call's state from page-locked host memory (n doubles) into r, without
// a copy command; the status word cleared (status may be NULL); f.hi given: the
// FP32 positions of the first n - 3, as launch_split_positions.
cudaError_t launch_stage_in(int n, const double *host_r, double *r, const F32Pos &f, int *status, cudaStream_t s);

// Integrator kernels. r, p: 3*nv doubles. Noise from Philox4x32-10 keyed by
// seed, counter (vertex, step, stream) with step = cnt[0] + cnt[1] - 1.
struct StepArgs {
  int kind;            // 0 overdamped BD, 1 BD membrane, 2 Langevin
  double mob_dt;       // kind 0: D dt / kT
  double sigma;        // kind 0: sqrt(2 D dt); kinds 1,2: sqrt(2 gamma kT AK)
  double AK;           // AKMA_TIME * time_step
  double gamma;
  uint64_t seed;
  uint32_t stream;
  float mob_dt_f, sigma_f;  // kind 0: mob_dt and sigma rounded to FP32 (the precision form's increment)
};
// Gather fused with the vertex-local update (kind 0; kinds 1/2 with identity mass).
// f (all NULL in the plain path) receives the FP32 positions of the new state.
template <typename T>
cudaError_t launch_gather_step(int nv, const T *partial, const int *off, const StepArgs &a, const uint64_t *cnt,
                               double *r, double *p, const F32Pos &f, const int *status, cudaStream_t s);
// Kinds 1/2 with a mass matrix: gather the gradient and kick p (friction, kicks,
// noise), with p's FP32 copy for the apply (see launch_mass_input32; NULL in the
// plain path); then qdot = M^-1 p; then r += qdot AK (and p reset for BD).
template <typename T>
cudaError_t launch_gather_kick(int nv, const T *partial, const int *off, const StepArgs &a, const uint64_t *cnt,
                               double *p, float *x32, int ld, const int *status, cudaStream_t s);
cudaError_t launch_drift(int nv, const StepArgs &a, double *r, double *p, const double *qdot, const F32Pos &f,
                         const int *status, cudaStream_t s);

// One mesh of a batch (device pointers into the mesh's own buffers). The
// face kernel stages the leading part, BatchFaceJob, in shared memory.
struct BatchFaceJob {
  dev::FaceSrc src[3];     // patch types: regular, irregular valence 5, irregular valence 7
  dev::SurfaceParams P;
  void *partial;           // the mesh's gradient-partial slots
  uint64_t *cnt;           // {first step of the run, steps done}
  uint64_t limit;          // steps in the run
  int *status;
  int pad;
};
struct BatchJob {
  BatchFaceJob f;
  const int *off;          // vertex slot locations {first slot, count} (interleaved numbering)
  double *r, *p;           // state
  float *rhi, *rlo;        // FP32 hi/lo pairs of r (precision form), else NULL
  const double *r0;        // reference state (precision form)
  float *dsp;              // r - r0 in FP32 (precision form)
  double *E, *parts;       // energy (and parts) of the latest step
  double *energies;        // the run's recorded energies, indexed by steps done
  double threshold;        // energy rise that flags divergence (<= 0: off)
  StepArgs a;              // the job's integrator
};
// Faces [first, first+count) of one patch type of one job, or vertices
// [first, first+count) of one job.
struct BatchTile {
  int job, first, count;
};
// Layout of the batch's device count array.
enum : int { kCountTiles = 0, kCountTileBase = 3, kCountJobs = 6, kCountVertexTiles = 7, kCountWords = 8 };
constexpr int kVertexTile = 256;  // vertices per vertex tile (one thread each)

// Face launches of patch type `group` over its tiles (counts[group] of them,
// from counts[3 + group] in tiles); tile_sums[3 * global tile] receives each
// tile's energy terms. Persistent grids; tiles of stopped or finished jobs are
// skipped. Regular faces of the precision form (tpf; next_tile: {tiles handed
// out, blocks done}, which the launch leaves zero), its irregular ones (32), and
// FP64 (64); table: the patch type's (face32_table.h, fixed64.h).
cudaError_t launch_batch_faces_tpf(const TpfRows &rows, const BatchJob *jobs, int group, const BatchTile *tiles,
                                   const int *counts, const float *table, double dudv, double *tile_sums, int grid,
                                   int *next_tile, cudaStream_t s);
cudaError_t launch_batch_faces32(const BatchJob *jobs, int group, const BatchTile *tiles, const int *counts,
                                 const float *table, int ncp, double dudv, double *tile_sums, int grid, cudaStream_t s);
cudaError_t launch_batch_faces64(const BatchJob *jobs, int group, const BatchTile *tiles, const int *counts,
                                 const int *table, const double *weight, int ncp, double dudv, double *tile_sums,
                                 int grid, cudaStream_t s);
// Per job: tile sums in listed order (tile_idx[tile_off[j] .. tile_off[j+1])),
// energy record, flags, steps done; live[j] and prog[j] = {done, status}.
cudaError_t launch_batch_reduce(const BatchJob *jobs, const int *counts, int max_jobs, const int *tile_off,
                                const int *tile_idx, const double *tile_sums, int *live, unsigned long long *prog,
                                cudaStream_t s);
// Gather fused with the update, for live jobs (kinds 0, and 1/2 with identity mass).
template <typename T>
cudaError_t launch_batch_gather_step(const BatchJob *jobs, const BatchTile *vtiles, const int *counts,
                                     const int *live, int grid, cudaStream_t s);
// Run start of the jobs with start[j] != 0: counters {step0[j], 0}, status 0, hi/lo split.
cudaError_t launch_batch_start(const BatchJob *jobs, const BatchTile *vtiles, const int *counts, const int *start,
                               const unsigned long long *step0, int grid, cudaStream_t s);
// Host-driven steps: jobs' states packed in job order at pack + off[j] (3 nv + 3
// doubles each). unpack: into the jobs' resident states (and FP32 copies);
// pack: back out, with each job's latest energy in E[j].
cudaError_t launch_batch_unpack(const BatchJob *jobs, const BatchTile *vtiles, const int *counts,
                                const long long *off, const double *pack, int grid, cudaStream_t s);
cudaError_t launch_batch_pack(const BatchJob *jobs, const BatchTile *vtiles, const int *counts, const long long *off,
                              double *pack, double *E, int grid, cudaStream_t s);
// Device-filling grids of the batch face launches.
int batch_face_blocks_tpf();
int batch_face_blocks32(int ncp);
int batch_face_blocks64(int ncp);
// Faces in flight per block of the half-warp kernels: the unit of a batch's tile sizes.
constexpr int kHalfWarps = 8;

// Factors of an M^-1 apply per component, scale / alpha_c^2.
struct MassScale {
  double f[3];
};
// out[3i+c] (+)= f_c (scalev ? scalev[c*nrow+i] : 1) * sum_k val[k] in[3 col[k]+c].
// accumulate=0 overwrites out.
cudaError_t launch_spmv(int nrow, const int *row_ptr, const int *col, const double *val, const double *scalev,
                        const MassScale &f, const double *in, double *out, int accumulate, cudaStream_t s);
// The same on FP32 values and an FP32 input packed as float4 {x, y, z, 0} per
// row (spmv32_kernel).
cudaError_t launch_spmv32(int nrow, const int *row_ptr, const void *col, bool col16, const float *val,
                          const double *scalev, const MassScale &f, const float4 *in, double *out, int accumulate,
                          cudaStream_t s);
// The same on a dense FP32 matrix, rows padded with zeros to dense32_ld(n)
// floats, and the input as three vectors x[c][dense32_ld(n)], padded with zeros.
inline int dense32_ld(int n) { return (n + 31) / 32 * 32; }
size_t dense32_scratch_doubles(int n);
cudaError_t launch_dense_apply32(int n, const float *A, const float *x, double *scratch, const MassScale &f,
                                 const double *scalev, double *out, int accumulate, cudaStream_t s);
// A leapfrog step's apply and drift: as launch_dense_apply32 into qdot, then
// launch_drift, with the drift done where the product is formed.
cudaError_t launch_dense_drift32(int n, const float *A, const float *x, double *scratch, const StepArgs &a, double *r,
                                 double *p, const F32Pos &f, const int *status, cudaStream_t s);
// The FP32 input of those: out4[i] = {in[3i], in[3i+1], in[3i+2], 0}, or (ld > 0)
// out[c ld + i] = in[3i+c].
cudaError_t launch_mass_input32(int n, const double *in, float *out, int ld, cudaStream_t s);

}  // namespace umcp
