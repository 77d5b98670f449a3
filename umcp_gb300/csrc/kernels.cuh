// Device kernels of the membrane-surface hot path (sm_103a).
//
// The face kernels write per-face gradient partials and per-block energy sums; no
// float atomics. Which takes a face:
//   face_tpf_kernel, batch_face_tpf_kernel (surface_kernels.cu)  the precision
//       form's regular faces of large meshes and of batches, one thread per face;
//   face32_kernel, batch_face32_kernel (face32.cu, face32.cuh)  its irregular
//       faces, and the regular ones of smaller meshes, a half-warp per face;
//   face_tc_kernel (surface_kernels.cu)  its regular faces on the tensor cores
//       (an option);
//   face64_kernel, batch_face64_kernel (face64.cu, face64.cuh)  FP64, a
//       half-warp per face, contractions in fixed point.
// The gather kernels sum each vertex's partials in a fixed order (slots
// interleaved by groups of 32 vertices), most of them fused with an integrator
// update. The last block of a pass sums the block sums (count_and_finish).
//
// The energy model is the reference's surface::fenergy/ifenergy with
// FIXED_A and LOCAL_LIPID_ENERGY (src/interpLib.C:3426-3881); the gradient
// is its exact derivative (src/grad.C:65-942, 6445-7457), written here in
// closed form: with m = Ru x Rv, W = |m|^2, l = m.Suu, k = m.Suv, n = m.Svv,
//   H = c1 + c2 = -(l Rv.Rv - 2 k Ru.Rv + n Ru.Ru) / W^(3/2)
//   K = c1 c2   = (l n - k^2) / W^2 - SAFETY/4
// which the reference reaches through the shape-operator eigenvalues.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace umcp {
namespace dev {

constexpr int kMaxCpDev = 13;   // control points of the largest patch (valence 7 + 6)
constexpr int kVertexBits = 27;  // packed control point: vertex | image_code << 27
constexpr uint32_t kVertexMask = (1u << kVertexBits) - 1u;
constexpr double kSafety = 1e-12;  // SAFETY, src/interp.h:14

// Elements of a gradient-partial slot. The precision form pads its slots to 16
// bytes: a face kernel writes each with one store instead of three 4-byte ones
// (whose 32 scattered sectors per warp instruction were 16% of the 256-vesicle
// face pass), and the gather reads them with 16-byte loads. FP64 slots stay at
// 24 bytes: that pass is bound by the FP64 pipe.
template <typename T>
constexpr int kSlot = sizeof(T) == 8 ? 3 : 4;

// The precision form's FP32 positions of a vertex lie together, 12 floats on a
// 16-byte boundary: hi.xyz, lo.xyz, dsp.xyz and three of padding, so a face
// kernel fetches a control point with two 16-byte loads and a 4-byte one instead
// of nine 4-byte ones from three arrays. F32Pos::hi, lo and dsp point at the first
// vertex's hi, lo and dsp.
constexpr int kPosStride = 12;
// Offset of coordinate i = 3 v + c from those pointers.
__host__ __device__ constexpr size_t pos_at(size_t i) { return kPosStride * (i / 3) + i % 3; }

struct SurfaceParams {
  double kc, KA, kg, k_reg;
  double box[3][3];
  float box_hi[3][3], box_lo[3][3];  // box = hi + lo, for the precision form
  // Precision form, [regular, irregular patches][area, curvature, angle]: the points'
  // coefficients over the same rounded to FP32. One relative error of every face
  // alike, which no sum over faces averages out (all 15 weights of the regular rule
  // are 1/15), so each block's or tile's energy sums are scaled by it, in FP64.
  double e_scale[2][3];
  int nv;
};

// Per-mesh view for a face launch of the precision form.
struct FaceLaunch {
  int nfaces;              // faces in this launch
  int block_base;          // first block-partial row of this launch
  const uint32_t *cp;      // [nfaces][ncp] packed control points
  const float *g0f, *rr0f, *compf;  // [nfaces][npt], [nfaces][npt], [nfaces][3]: P2, Hbar, Pres
  const float *table;      // the patch type's staged table (face32_table.h)
  const double *basis;     // [npt][5][ncp rounded up to 4] rows u,v,uu,uv,vv (tensor-core kernel)
  const double *weight;    // [npt]
  double dudv;
};

// Where one face group's data and its mesh's state live.
struct FaceSrc {
  const uint32_t *cp;
  const double *g0, *rr0, *comp;
  const float *g0f, *rr0f, *compf;
  const int *dest;
  const double *r;
  const float *rhi, *rlo;
  const float *dsp;  // precision form: r - r0 per coordinate (displacement from the reference state); see kPosStride
  int nfaces;
};

template <typename T>
struct Vec3 {
  T x, y, z;
};

}  // namespace dev
}  // namespace umcp
