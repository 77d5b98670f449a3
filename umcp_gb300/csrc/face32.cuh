// The precision form's pointwise step and per-lane sums, shared by its face
// kernels (surface_kernels.cu).
#pragma once
#include <stddef.h>

#include "face32_table.h"
#include "kernels.cuh"
#include "launch.h"

namespace umcp {
namespace dev {

// Error-free sum: s + e == a + b exactly (Knuth's two-sum).
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e) {
  s = a + b;
  float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

// Kahan-compensated FP32 totals, which keep the FP64 pipe out of the face loop.
template <int N>
struct KahanSums {
  float s[N] = {}, c[N] = {};
  __device__ __forceinline__ void add(int q, float v) {
    const float y = v - c[q], t = s[q] + y;
    c[q] = (t - s[q]) - y;
    s[q] = t;
  }
  __device__ __forceinline__ double get(int q) const { return (double)s[q] - (double)c[q]; }
};

// Sum over the warp's lanes of the compensated total s - c, in a fixed (xor-tree)
// order, in pairs of FP32 (error-free sums): an FP64 tree costs the warp five
// instructions of 64 cycles for each quantity, which at a tile of eight faces
// was more than the faces.
__device__ __forceinline__ double warp_sum(float s, float c) {
  float hi = s, lo = -c;
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    const float oh = __shfl_xor_sync(0xFFFFFFFFu, hi, off), ol = __shfl_xor_sync(0xFFFFFFFFu, lo, off);
    float t, e;
    two_sum(hi, oh, t, e);
    lo = e + (lo + ol);
    hi = t;
  }
  return (double)hi + (double)lo;
}

namespace f32 {

__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ Vec3<float> cross(const Vec3<float> &x, const Vec3<float> &y) {
  return {fma(x.y, y.z, -mul(x.z, y.y)), fma(x.z, y.x, -mul(x.x, y.z)), fma(x.x, y.y, -mul(x.y, y.x))};
}
__device__ __forceinline__ float dot(const Vec3<float> &x, const Vec3<float> &y) {
  return fma(x.x, y.x, fma(x.y, y.y, mul(x.z, y.z)));
}
// 1/sqrt(x) and 1/x: the hardware estimates with one Newton step, about 1 ulp.
__device__ __forceinline__ float rsqrt(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return fma(mul(0.5f, y), fma(-mul(x, y), y, 1.f), y);
}
__device__ __forceinline__ float rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return fma(y, fma(-x, y, 1.f), y);
}

// A vertex's FP32 positions (hi: F32Pos::hi).
__device__ __forceinline__ void load_vertex(const float *__restrict__ hi, int v, float h[3], float l[3], float d[3]) {
  const float *q = hi + kPosStride * (size_t)v;
  const float4 a = __ldg(reinterpret_cast<const float4 *>(q)), b = __ldg(reinterpret_cast<const float4 *>(q) + 1);
  h[0] = a.x; h[1] = a.y; h[2] = a.z;
  l[0] = a.w; l[1] = b.x; l[2] = b.y;
  d[0] = b.z; d[1] = b.w; d[2] = __ldg(q + 8);
}

// Control point (hi + lo) in lattice image `code`, relative to the patch corner
// (ahi + alo, home image): error-free sums, so the local coordinates carry full
// FP32 precision even across periodic images.
__device__ __forceinline__ void local_position(const float hi[3], const float lo[3], int code, const float ahi[3],
                                               const float alo[3], const SurfaceParams &P, float l[3]) {
  if (code == 13) {  // the home image (every control point of a closed vesicle)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      float s2, e2;
      two_sum(hi[c], -ahi[c], s2, e2);
      l[c] = s2 + (e2 + (lo[c] - alo[c]));
    }
  } else {  // the lattice shift as hi + lo (each term exact: images are -1, 0 or +1)
    const int img[3] = {code % 3 - 1, (code / 3) % 3 - 1, code / 9 - 1};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      float sh = 0.f, she = 0.f, shl = 0.f;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        float t, e;
        two_sum(sh, mul((float)img[d], P.box_hi[d][c]), t, e);
        sh = t;
        she = add(she, e);
        shl = add(shl, mul((float)img[d], P.box_lo[d][c]));
      }
      float s1, e1, s2, e2;
      two_sum(hi[c], sh, s1, e1);
      two_sum(s1, -ahi[c], s2, e2);
      l[c] = s2 + ((e1 + e2) + ((lo[c] - alo[c]) + (she + shl)));
    }
  }
}

// The moduli times a quadrature point's weight, formed in FP64 once per launch
// or job and rounded once: kc w / 4, dudv w KA, dudv w kg. (The weights of a rule
// being equal, all faces share that rounding; SurfaceParams::e_scale takes it out of
// the energies.)
struct Coef {
  float curv, area, gauss;
};
__device__ __forceinline__ Coef point_coef(const SurfaceParams &P, double w, double dudv) {
  return {(float)(0.25 * P.kc * w), (float)(dudv * w * P.KA), (float)(dudv * w * P.kg)};
}

// The global restraints at a point: dE_r/dA and dE_r/dV times the point's area
// and volume weights (cA cw, cV cw / 3), and the limit point relative to the patch
// corner (GEO). The corner's own part of the volume gradient is formed once per face
// (GeoCorner; corner_entry in face32_table.h has the reason): with absolute limit points
// in the points' sums, the gradient of a 40,962-vertex vesicle under a volume restraint
// was off by 1.07e-6 of its norm, now 6.0e-7.
struct GeoPoint {
  float kA, kV;
  Vec3<float> R;
};
// The patch corner, absolute and box-scaled (it carries no image): x = hi + lo, times dE_r/dV.
struct GeoCorner {
  float x[3], hi[3], lo[3];
  __device__ __forceinline__ GeoCorner(const float alpha[3], const float ahi[3], const float alo[3], float cV) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float p = mul(alpha[c], ahi[c]), e = fma(alpha[c], alo[c], fma(alpha[c], ahi[c], -p));
      x[c] = add(p, e);
      hi[c] = mul(cV, p);
      lo[c] = fma(cV, e, fma(cV, p, -hi[c]));
    }
  }
  // its part of control point j's gradient, t x (hi + lo) with t = sum_i M[j][i] X_i
  __device__ __forceinline__ void gradient(const float t[3], float d[3]) const {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int a = (c + 1) % 3, b = (c + 2) % 3;
      d[c] = fma(t[a], hi[b], fma(-t[b], hi[a], fma(t[a], lo[b], -mul(t[b], lo[a]))));
    }
  }
};
__device__ __forceinline__ float2 geo_coef(const double *gterm, double w, double dudv) {
  return make_float2((float)(gterm[kGeoCA] * (dudv * w)), (float)(gterm[kGeoCV] * (dudv * w) / 3.0));
}

// One quadrature point's energy terms and adjoints.
struct Point {
  float ea, ec, er;       // area, curvature, angle
  Vec3<float> Ku, Kv, m;  // dE/dRu, dE/dRv, and the normal
  float lb, kb, nb;       // dE/dSuu = lb m, dE/dSuv = kb m, dE/dSvv = nb m
  float r11, r12, r22;    // the angle term's part of dE/dRu = r11 Ru + r12 Rv, dE/dRv = r22 Rv + r12 Ru (KG_REG)
};

// Pointwise energy and adjoint (the model of kernels.cuh) for K = {Ru, Rv, Suu,
// Suv, Svv} and quadrature weight w.
// dR = {Ru - Ru0, Rv - Rv0}, the tangents' change from the reference state,
// contracted from the control points' displacements. The area strain g - g0 is
// then formed without cancellation:
//   dm = m - m0 = (Ru - Ru0) x Rv0 + Ru x (Rv - Rv0),  W - W0 = dm . (2 m - dm),
//   g - g0 = (W - W0) / (g + g0)
// (exactly zero at the reference state). Subtracting g0 from an FP32 g would
// leave every tangent's rounding in the strain: at and near the reference
// state that rounding is the whole area force, on coarse patches up to 1e-5
// of the gradient.
// KG_REG = false: kg and k_reg are zero and their terms are left out.
// GEO: the restraints' gradient goes along, dE_r/dg = kA (g = |m|), dE_r/dm =
// kV R (R relative to the corner) and dE_r/dR = kV m (the last for the caller: one
// more coefficient of m beside lb, kb, nb, on the value row).
// Products and sums are rounded as written (no contraction is left to the
// compiler), so every kernel that inlines this rounds alike: a batch's job
// follows its single-mesh trajectory bit for bit whichever kernels run it.
template <bool KG_REG, bool GEO = false>
__device__ __forceinline__ Point point(const Vec3<float> K[5], const Vec3<float> dR[2], const Coef &M, float k_reg,
                                       float g0, float rr0, float P2, float Hbar, float Pres,
                                       const GeoPoint &geo = GeoPoint{}) {
  const Vec3<float> &Ru = K[0], &Rv = K[1], &Suu = K[2], &Suv = K[3], &Svv = K[4], &a = dR[0], &b = dR[1];
  Point o;
  const Vec3<float> m = cross(Ru, Rv);
  const float W = dot(m, m), E11 = dot(Ru, Ru), E12 = dot(Ru, Rv), E22 = dot(Rv, Rv);
  const float l = dot(m, Suu), k = dot(m, Suv), n = dot(m, Svv);
  const float ig = rsqrt(W), g = mul(W, ig), iW = mul(ig, ig), ig3 = mul(iW, ig);
  const float k2 = mul(-2.f, k);
  const float Tt = fma(l, E22, fma(k2, E12, mul(n, E11)));
  const float dH = fma(-Tt, ig3, -Hbar), aH = mul(P2, dH);  // H = -Tt W^-3/2
  const Vec3<float> v0 = {sub(Rv.x, b.x), sub(Rv.y, b.y), sub(Rv.z, b.z)};
  const Vec3<float> dm = {fma(a.y, v0.z, fma(-a.z, v0.y, fma(Ru.y, b.z, -mul(Ru.z, b.y)))),
                          fma(a.z, v0.x, fma(-a.x, v0.z, fma(Ru.z, b.x, -mul(Ru.x, b.z)))),
                          fma(a.x, v0.y, fma(-a.y, v0.x, fma(Ru.x, b.y, -mul(Ru.y, b.x))))};
  const Vec3<float> sm = {fma(2.f, m.x, -dm.x), fma(2.f, m.y, -dm.y), fma(2.f, m.z, -dm.z)};
  const float dg = mul(dot(dm, sm), rcp(add(g, g0)));
  const float ct = mul(mul(M.area, rcp(g0)), dg);
  o.ec = mul(M.curv, fma(aH, dH, Pres));
  o.ea = mul(ct, dg);
  o.er = 0.f;
  const float Tb = mul(mul(mul(-2.f, M.curv), aH), ig3), T2 = mul(-2.f, Tb);
  float W2 = fma(mul(2.f, ct), ig, mul(mul(-3.f, iW), mul(Tb, Tt)));  // 2 dE/dW
  o.lb = mul(Tb, E22);
  o.kb = mul(T2, E12);
  o.nb = mul(Tb, E11);
  float F11 = -mul(T2, n), F12 = mul(Tb, k2), F22 = -mul(T2, l);  // 2 dE/dE11, dE/dE12, 2 dE/dE22
  if constexpr (KG_REG) {
    const float Q = fma(l, n, -mul(k, k)), iW2 = mul(iW, iW), cg = mul(M.gauss, g0);
    o.ec = fma(cg, fma(Q, iW2, (float)(-0.25 * kSafety)), o.ec);
    const float Qb = mul(cg, iW2);
    W2 = fma(mul(mul(-4.f, Qb), Q), iW, W2);
    o.lb = fma(Qb, n, o.lb);
    o.kb = fma(Qb, k2, o.kb);
    o.nb = fma(Qb, l, o.nb);
    const float is = rsqrt(mul(E11, E22)), val = mul(E12, is), dv = sub(val, rr0), kdv = mul(k_reg, dv),
                vb = mul(2.f, kdv), vv = mul(mul(vb, val), mul(is, is));
    o.er = mul(kdv, dv);
    o.r11 = -mul(vv, E22);  // E22 / (E11 E22) = 1 / E11
    o.r12 = mul(vb, is);
    o.r22 = -mul(vv, E11);
    F11 = add(F11, o.r11);
    F12 = add(F12, o.r12);
    F22 = add(F22, o.r22);
  }
  if constexpr (GEO) W2 = fma(geo.kA, ig, W2);
  const float lb = o.lb, kb = o.kb, nb = o.nb;
  Vec3<float> mb = {fma(lb, Suu.x, fma(kb, Suv.x, fma(nb, Svv.x, mul(W2, m.x)))),
                    fma(lb, Suu.y, fma(kb, Suv.y, fma(nb, Svv.y, mul(W2, m.y)))),
                    fma(lb, Suu.z, fma(kb, Suv.z, fma(nb, Svv.z, mul(W2, m.z))))};
  if constexpr (GEO) mb = {fma(geo.kV, geo.R.x, mb.x), fma(geo.kV, geo.R.y, mb.y), fma(geo.kV, geo.R.z, mb.z)};
  // F11 Ru + F12 Rv + Rv x mb and F22 Rv + F12 Ru + mb x Ru
  o.Ku = {fma(Rv.y, mb.z, fma(-Rv.z, mb.y, fma(F11, Ru.x, mul(F12, Rv.x)))),
          fma(Rv.z, mb.x, fma(-Rv.x, mb.z, fma(F11, Ru.y, mul(F12, Rv.y)))),
          fma(Rv.x, mb.y, fma(-Rv.y, mb.x, fma(F11, Ru.z, mul(F12, Rv.z))))};
  o.Kv = {fma(mb.y, Ru.z, fma(-mb.z, Ru.y, fma(F22, Rv.x, mul(F12, Ru.x)))),
          fma(mb.z, Ru.x, fma(-mb.x, Ru.z, fma(F22, Rv.y, mul(F12, Ru.y)))),
          fma(mb.x, Ru.y, fma(-mb.y, Ru.x, fma(F22, Rv.z, mul(F12, Ru.z))))};
  o.m = m;
  return o;
}

// The point's part of alpha_c dE/dalpha_c, sum over the five rows of dE/dK . K,
// added to s (K is linear in the box-scaled coordinates).
__device__ __forceinline__ Vec3<float> scale_derivative(const Point &o, const Vec3<float> K[5], const Vec3<float> &s) {
  auto one = [&](float ku, float u, float kv, float v, float m, float uu, float uv, float vv, float s0) {
    return fma(ku, u, fma(kv, v, fma(m, fma(o.lb, uu, fma(o.kb, uv, mul(o.nb, vv))), s0)));
  };
  return {one(o.Ku.x, K[0].x, o.Kv.x, K[1].x, o.m.x, K[2].x, K[3].x, K[4].x, s.x),
          one(o.Ku.y, K[0].y, o.Kv.y, K[1].y, o.m.y, K[2].y, K[3].y, K[4].y, s.y),
          one(o.Ku.z, K[0].z, o.Kv.z, K[1].z, o.m.z, K[2].z, K[3].z, K[4].z, s.z)};
}
// The restraints' value-row part of it, kV m . (X0 + R). (The corner's part of the
// volume gradient adds its own, sum_j d_j . X_j over GeoCorner::gradient.)
__device__ __forceinline__ Vec3<float> geo_scale_derivative(const Point &o, const GeoPoint &geo, const float X0[3],
                                                            const Vec3<float> &s) {
  return {fma(mul(geo.kV, o.m.x), add(X0[0], geo.R.x), s.x), fma(mul(geo.kV, o.m.y), add(X0[1], geo.R.y), s.y),
          fma(mul(geo.kV, o.m.z), add(X0[2], geo.R.z), s.z)};
}

}  // namespace f32
}  // namespace dev
}  // namespace umcp

// ---------------------------------------------------------------- half-warp form
//
// One face per half-warp, faces in pairs per warp (both halves always run
// together; a half without a face repeats another's). Lanes are control points
// while the local coordinates are formed, quadrature points for the forward
// contractions and the pointwise step, and control points again for the
// gradient: the point lanes leave their adjoints (12 floats) in shared memory,
// and lane j adds B[u][j] Ku + B[v][j] Kv + s[j] m over the points in order, with
// the multiply-adds in the order of the thread-per-face form, so both forms
// give the same gradient bits. Energy terms and box-scale derivatives are
// Kahan-summed per lane over the lane's faces. It is bound by the latency of a
// face's chain on small meshes (a face pass of 1,280 faces takes 6.5 us, 3 us of
// it the launch) and by instruction issue on large ones. (The half-warp form
// before it transposed every point's contribution to every control point
// through shared memory, whose data pipe bounded it: 10.4 us for 1,280 faces.)
namespace umcp {
namespace dev {
namespace f32 {

constexpr int kThreads = 128, kHW = kThreads / 16, kWarps = kThreads / 32;

template <int NCP, int NPT>
struct Smem {
  using L = F32Table<NCP, NPT>;
  float4 B[NPT][L::ROW4];           // rows u, v, uu, uv, vv of point p, control points in fours (forward)
  float4 G4[NPT][NCP];              // u, v, uu, uv of control point j (gradient)
  float G1[NPT][16];                // vv of control point j
  float4 V[NPT][L::NC4];            // value rows
  float4 X[kHW][3][L::NC4];         // coordinate c of the local control points
  float4 D[kHW][3][L::NC4];         // the same points' change from the reference state
  float4 A[kHW][NPT][3];            // {Ku, lb}, {Kv, kb}, {m, nb} of each point
  float2 geo[16];                   // restraints: each point's kA, kV
  float4 M[NCP][L::NC4];            // the corner matrix
  float cV;                         // and dE_r/dV
  float corner[kHW][2][3];          // and each face's corner, hi and lo
  double red[kWarps][6];
};

// Global data of one face, loaded one face ahead.
struct Ahead {
  float hi[3] = {0, 0, 0}, lo[3] = {0, 0, 0}, dsp[3] = {0, 0, 0};
  int code = 13;            // lattice image (13: home)
  float g0 = 1, rr0 = 0, P2 = 0, Hbar = 0, Pres = 0;
  int dest = -1;            // -1: no slot (the lane has no control point, or the half-warp no face)
  bool on = false;          // the half-warp has a face of its own
};

// Face f; a half-warp past the end takes face end - 1 along (on false: nothing
// of it is summed or written).
template <int NCP, int NPT, bool KG_REG>
__device__ __forceinline__ void load(const FaceSrc &S, int f, int end, int lane, Ahead &a) {
  a.on = f < end;
  f = min(f, end - 1);
  if (lane < NCP) {
    const uint32_t packed = __ldg(&S.cp[(size_t)f * NCP + lane]);
    a.code = (int)(packed >> kVertexBits);
    load_vertex(S.rhi, (int)(packed & kVertexMask), a.hi, a.lo, a.dsp);
    a.dest = a.on ? __ldg(&S.dest[(size_t)f * NCP + lane]) : -1;
  }
  if (lane < NPT) {
    a.g0 = __ldg(&S.g0f[(size_t)f * NPT + lane]);
    if constexpr (KG_REG) a.rr0 = __ldg(&S.rr0f[(size_t)f * NPT + lane]);
    a.P2 = __ldg(&S.compf[3 * (size_t)f]);
    a.Hbar = __ldg(&S.compf[3 * (size_t)f + 1]);
    a.Pres = __ldg(&S.compf[3 * (size_t)f + 2]);
  }
}

// Stages a patch type's table; gives this lane's quadrature weight.
template <int NCP, int NPT>
__device__ __forceinline__ double stage(Smem<NCP, NPT> &sm, const float *__restrict__ table) {
  using L = F32Table<NCP, NPT>;
  const float4 *t = reinterpret_cast<const float4 *>(table);
  float4 *b = &sm.B[0][0];
  using S = Smem<NCP, NPT>;
  static_assert(offsetof(S, X) == sizeof(float) * L::kWeights, "the staged part is the table's image");
  for (int i = threadIdx.x; i < L::kWeights / 4; i += kThreads) b[i] = __ldg(t + i);
  if constexpr (NCP % 4 != 0)  // the padding of the last four stays zero
    for (int i = threadIdx.x; i < kHW * 3; i += kThreads) {
      sm.X[i / 3][i % 3][L::NC4 - 1] = make_float4(0.f, 0.f, 0.f, 0.f);
      sm.D[i / 3][i % 3][L::NC4 - 1] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  const int lane = threadIdx.x & 15;
  return lane < NPT ? __ldg(reinterpret_cast<const double *>(table + L::kWeights) + lane) : 0.0;
}

template <int NCP, int NPT, bool KG_REG, bool GEO>
__device__ __forceinline__ void face(Smem<NCP, NPT> &sm, int hw, int lane, const Ahead &cur, const SurfaceParams &P,
                                     const float alpha[3], const float am1[3], const Coef &M, float k_reg, bool reg_alpha, bool want_da, float *__restrict__ partial, KahanSums<6> &sums) {
  constexpr int NC4 = F32Table<NCP, NPT>::NC4;
  // ---- lanes as control points: relative to the patch corner (control point 0)
  // in their lattice images, times alpha, with error-free sums on the hi/lo
  // pairs; and their change from the reference state, alpha L - L0 =
  // (alpha - 1) L + (dsp - dsp of the corner)
  GeoPoint geo{0.f, 0.f, {0.f, 0.f, 0.f}};
  {
    float ahi[3], alo[3], ad[3], l[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      ahi[c] = __shfl_sync(0xFFFFFFFFu, cur.hi[c], 0, 16);
      alo[c] = __shfl_sync(0xFFFFFFFFu, cur.lo[c], 0, 16);
      ad[c] = __shfl_sync(0xFFFFFFFFu, cur.dsp[c], 0, 16);
    }
    local_position(cur.hi, cur.lo, cur.code, ahi, alo, P, l);
    if (lane < NCP) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        reinterpret_cast<float *>(sm.X[hw][c])[lane] = mul(alpha[c], l[c]);
        reinterpret_cast<float *>(sm.D[hw][c])[lane] = fma(am1[c], l[c], sub(cur.dsp[c], ad[c]));
        if (GEO && lane == 0) {
          sm.corner[hw][0][c] = ahi[c];
          sm.corner[hw][1][c] = alo[c];
        }
      }
    }
  }
  __syncwarp();
  // ---- lanes as quadrature points; K[k]_c as two partial sums (even and odd
  // control points) in one paired multiply-add
  if (lane < NPT) {
    float2 A[5][3], Ad[2][3], Av[3];
#pragma unroll
    for (int k = 0; k < 5; ++k) A[k][0] = A[k][1] = A[k][2] = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < 2; ++k) Ad[k][0] = Ad[k][1] = Ad[k][2] = make_float2(0.f, 0.f);
    Av[0] = Av[1] = Av[2] = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int c4 = 0; c4 < NC4; ++c4) {
      float4 x[3], d[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        x[c] = sm.X[hw][c][c4];
        d[c] = sm.D[hw][c][c4];
      }
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const float4 b = sm.B[lane][k * NC4 + c4];
        const float2 b01 = make_float2(b.x, b.y), b23 = make_float2(b.z, b.w);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          A[k][c] = __ffma2_rn(b01, make_float2(x[c].x, x[c].y), A[k][c]);
          A[k][c] = __ffma2_rn(b23, make_float2(x[c].z, x[c].w), A[k][c]);
          if (k < 2) {
            Ad[k][c] = __ffma2_rn(b01, make_float2(d[c].x, d[c].y), Ad[k][c]);
            Ad[k][c] = __ffma2_rn(b23, make_float2(d[c].z, d[c].w), Ad[k][c]);
          }
        }
      }
      if constexpr (GEO) {
        const float4 b = sm.V[lane][c4];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          Av[c] = __ffma2_rn(make_float2(b.x, b.y), make_float2(x[c].x, x[c].y), Av[c]);
          Av[c] = __ffma2_rn(make_float2(b.z, b.w), make_float2(x[c].z, x[c].w), Av[c]);
        }
      }
    }
    Vec3<float> K[5], dR[2];
#pragma unroll
    for (int k = 0; k < 5; ++k) K[k] = {add(A[k][0].x, A[k][0].y), add(A[k][1].x, A[k][1].y), add(A[k][2].x, A[k][2].y)};
#pragma unroll
    for (int k = 0; k < 2; ++k)
      dR[k] = {add(Ad[k][0].x, Ad[k][0].y), add(Ad[k][1].x, Ad[k][1].y), add(Ad[k][2].x, Ad[k][2].y)};
    if constexpr (GEO) {
      geo.R = {add(Av[0].x, Av[0].y), add(Av[1].x, Av[1].y), add(Av[2].x, Av[2].y)};
      geo.kA = sm.geo[lane].x;
      geo.kV = sm.geo[lane].y;
    }
    const Point o = point<KG_REG, GEO>(K, dR, M, k_reg, cur.g0, cur.rr0, cur.P2, cur.Hbar, cur.Pres, geo);
    sm.A[hw][lane][0] = make_float4(o.Ku.x, o.Ku.y, o.Ku.z, o.lb);
    sm.A[hw][lane][1] = make_float4(o.Kv.x, o.Kv.y, o.Kv.z, o.kb);
    sm.A[hw][lane][2] = make_float4(o.m.x, o.m.y, o.m.z, o.nb);
    if (cur.on) {
      sums.add(0, o.ea);
      sums.add(1, o.ec);
      if constexpr (KG_REG) sums.add(2, o.er);
      if (want_da) {
        Vec3<float> d = scale_derivative(o, K, {0.f, 0.f, 0.f});
        if constexpr (GEO) d = geo_scale_derivative(o, geo, GeoCorner(alpha, sm.corner[hw][0], sm.corner[hw][1], 0.f).x, d);
        if (KG_REG && reg_alpha) {
          // the angle term's extra box-scale part (src/grad.C:7414-7421):
          // sum_x (b_u Kreg_u + b_v Kreg_v) X = Kreg_u Ru + Kreg_v Rv, times alpha - 1
          const Vec3<float> &u = K[0], &v = K[1];
          d.x = fma(am1[0], (o.r11 * u.x + o.r12 * v.x) * u.x + (o.r22 * v.x + o.r12 * u.x) * v.x, d.x);
          d.y = fma(am1[1], (o.r11 * u.y + o.r12 * v.y) * u.y + (o.r22 * v.y + o.r12 * u.y) * v.y, d.y);
          d.z = fma(am1[2], (o.r11 * u.z + o.r12 * v.z) * u.z + (o.r22 * v.z + o.r12 * u.z) * v.z, d.z);
        }
        sums.add(3, d.x);
        sums.add(4, d.y);
        sums.add(5, d.z);
      }
    }
  }
  __syncwarp();
  // ---- lanes as control points: the gradient
  if (lane < NCP) {
    float g[3] = {0.f, 0.f, 0.f};
#pragma unroll 3
    for (int p = 0; p < NPT; ++p) {
      const float4 u = sm.A[hw][p][0], v = sm.A[hw][p][1], m = sm.A[hw][p][2], b = sm.G4[p][lane];
      float s = fma(sm.G1[p][lane], m.w, fma(b.w, v.w, mul(b.z, u.w)));
      if constexpr (GEO) s = fma(reinterpret_cast<const float *>(sm.V[p])[lane], sm.geo[p].y, s);
      g[0] = fma(s, m.x, fma(b.y, v.x, fma(b.x, u.x, g[0])));
      g[1] = fma(s, m.y, fma(b.y, v.y, fma(b.x, u.y, g[1])));
      g[2] = fma(s, m.z, fma(b.y, v.z, fma(b.x, u.z, g[2])));
    }
    if (GEO && sm.cV != 0.f) {  // a volume restraint acts
      float t[3] = {0.f, 0.f, 0.f};
#pragma unroll 1
      for (int c4 = 0; c4 < NC4; ++c4) {
        const float4 w = sm.M[lane][c4];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const float4 x = sm.X[hw][c][c4];
          t[c] = fma(w.w, x.w, fma(w.z, x.z, fma(w.y, x.y, fma(w.x, x.x, t[c]))));
        }
      }
      float d[3];
      GeoCorner(alpha, sm.corner[hw][0], sm.corner[hw][1], sm.cV).gradient(t, d);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        g[c] = add(g[c], d[c]);
        if (want_da && cur.on) sums.add(3 + c, mul(d[c], reinterpret_cast<const float *>(sm.X[hw][c])[lane]));
      }
    }
    if (cur.dest >= 0)
      reinterpret_cast<float4 *>(partial)[cur.dest] =
          make_float4(mul(alpha[0], g[0]), mul(alpha[1], g[1]), mul(alpha[2], g[2]), 0.f);
  }
  __syncwarp();  // the next face overwrites X, D and A
}

}  // namespace f32
}  // namespace dev
}  // namespace umcp
