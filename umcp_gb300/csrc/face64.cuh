// The FP64 face pass of one pair of faces by one warp (a half-warp per face):
// the energy model of kernels.cuh with both basis contractions in fixed point
// (fixed64.h) and the pointwise step in FP64.
//
// What bounds it is the FP64 pipe, at 64 to 76 cycles per warp instruction and
// scheduler whatever the number of active lanes. So
//  - both contractions run on the integer multiply-adds (forward 540, backward
//    675 of them per warp, about 4,200 cycles, where the FP64 forms were 180
//    and 225 FP64 instructions, about 28,000 cycles), and the conversions
//    between doubles and integers are integer instructions too;
//  - the pointwise step keeps to one reciprocal square root and one reciprocal
//    (two more square roots' worth with the Gaussian-curvature and angle
//    terms), about 120 FP64 instructions instead of 290;
//  - energies and box-scale derivatives are summed per lane over the lane's
//    faces and reduced once per warp, not once per face;
//  - both half-warps always run together (a half without a face repeats
//    another's): a half-warp alone would cost the pipe as much as a whole one.
// Measured against the all-FP64 form: energy and gradient of a 61 x 46 periodic
// membrane on device arrays 118.9 -> 47.3 us; a BD step of a 642-vertex vesicle
// 73.1 -> 45.6 us; errors against 64-bit sums unchanged (2.7e-15, 1e-15).
#pragma once
#include "fixed64.h"
#include "kernels.cuh"

namespace umcp {
namespace dev {
namespace f64 {

constexpr int kThreads = 128, kHW = kThreads / 16, kWarps = kThreads / 32;

template <int NCP, int NPT>
struct Smem {
  static constexpr int PAIRS = (NCP + 1) / 2, ROW4 = fixed::row_int4(NCP);
  int4 B[NPT][ROW4];          // point p's rows u, v, uu, uv, vv as limb pairs, two control points per int4
  int4 X[kHW][3][PAIRS];      // control points: coordinate c as limb pairs
  int4 K[kHW][NPT][3][3];     // adjoints of the five rows, coordinate c, as limb pairs (the sixth unused)
  double red[kWarps][6];
};

// v 2^(bits - 1 - top) to the nearest integer, as limbs; d = top - exponent of
// v (biased fields) >= 0. Zero and denormal v give 0.
__device__ __forceinline__ int2 to_limbs(double v, int d, int bits) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(v);
  unsigned long long m = ((u & 0xFFFFFFFFFFFFFull) | (1ull << 52)) << (bits - 53);
  m = d < 60 && ((unsigned)(u >> 52) & 0x7FFu) ? (m + ((1ull << (d & 63)) >> 1)) >> (d & 63) : 0ull;
  const long long s = (u >> 63) ? -(long long)m : (long long)m;
  const int l = (int)((unsigned)s << (32 - fixed::kLimb)) >> (32 - fixed::kLimb);
  return make_int2((int)((s - l) >> fixed::kLimb), l);
}
__device__ __forceinline__ int exponent_field(double v) { return (__double2hiint(v) >> 20) & 0x7FF; }
// v 2^e, rounded to nearest; the result's exponent is inside a double's normal range
__device__ __forceinline__ double from_fixed(long long v, int e) {
  const unsigned long long a0 = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
  const int lz = __clzll((long long)a0);
  const unsigned long long a = a0 << (lz & 63);
  const unsigned long long m = (a >> 11) + ((a >> 10) & 1ull);  // 2^52 <= m <= 2^53: its top bit adds 1 to the exponent
  const unsigned long long b = ((unsigned long long)(unsigned)(fixed::kBias + 62 - lz + e) << 52) + m;
  return v == 0 ? 0.0 : __longlong_as_double((long long)(b | ((unsigned long long)v & (1ull << 63))));
}
__device__ __forceinline__ long long mad_wide(int a, int b, long long c) {
  long long d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}
// Largest of q over the half-warp.
__device__ __forceinline__ int half_max(int q) {
#pragma unroll
  for (int off = 8; off >= 1; off >>= 1) q = max(q, __shfl_xor_sync(0xFFFFFFFFu, q, off));
  return q;
}

// Exponents of coordinates and adjoints that the integer forms take: outside,
// the squares and products of the pointwise step leave FP64's range anyway and
// the face's energy and gradient are set to NaN (the run's non-finite status).
constexpr int kPosLow = fixed::kBias - 300, kPosHigh = fixed::kBias + 300;
constexpr int kAdjLow = fixed::kBias - 900, kAdjHigh = fixed::kBias + 900;

// Moduli times a lane's quadrature weight, formed once per launch (or tile).
struct PointCoef {
  double c_curv, c_area, c_gauss, k_reg;  // kc w / 4, dudv w KA, dudv w kg, k_reg
  __device__ __forceinline__ PointCoef(const SurfaceParams &P, double w, double dudv)
      : c_curv(0.25 * P.kc * w), c_area(dudv * w * P.KA), c_gauss(dudv * w * P.kg), k_reg(P.k_reg) {}
};

// Per-lane sums: energy terms of the lane's point, box-scale derivatives of
// its control point (and of its point's angle term).
struct Sums {
  double ea = 0, ec = 0, er = 0, da[3] = {0, 0, 0};
};

// The pointwise energy and adjoint for K = {Ru, Rv, Suu, Suv, Svv}; adds the point's
// energy terms if on, overwrites K with the adjoints. reg_alpha: also adds the
// angle term's extra box-scale part (src/grad.C:7414-7421), times alpha - 1.
template <bool KG_REG>
__device__ __forceinline__ void point(Vec3<double> K[5], const PointCoef &C, double g0, double rr0, double P2,
                                      double Hbar, double Pres, bool on, bool reg_alpha, const double am1[3], Sums &s) {
  // Products and sums are rounded as written (mul, fma; no contraction left to
  // the compiler), so every kernel that inlines this rounds alike.
  auto mul = [](double x, double y) { return __dmul_rn(x, y); };
  auto cross = [&](const Vec3<double> &x, const Vec3<double> &y) {
    return Vec3<double>{fma(x.y, y.z, -mul(x.z, y.y)), fma(x.z, y.x, -mul(x.x, y.z)), fma(x.x, y.y, -mul(x.y, y.x))};
  };
  auto dot = [&](const Vec3<double> &x, const Vec3<double> &y) { return fma(x.x, y.x, fma(x.y, y.y, mul(x.z, y.z))); };
  const Vec3<double> Ru = K[0], Rv = K[1], Suu = K[2], Suv = K[3], Svv = K[4];
  const Vec3<double> m = cross(Ru, Rv);
  const double W = dot(m, m), E11 = dot(Ru, Ru), E12 = dot(Ru, Rv), E22 = dot(Rv, Rv);
  const double l = dot(m, Suu), k = dot(m, Suv), n = dot(m, Svv);
  const double ig = rsqrt(W);
  const double ge = mul(W, ig), g = fma(mul(0.5, ig), fma(-ge, ge, W), ge);  // sqrt(W), one correction
  const double iW = mul(ig, ig), ig3 = mul(iW, ig), ig0 = __drcp_rn(g0);
  const double k2 = mul(-2.0, k);
  const double Tt = fma(l, E22, fma(k2, E12, mul(n, E11)));
  const double dH = fma(-Tt, ig3, -Hbar), a = mul(P2, dH);  // H = -Tt W^-3/2
  const double dg = __dsub_rn(g, g0), t = mul(dg, ig0), ct = mul(C.c_area, t);
  if (on) {
    s.ec = fma(C.c_curv, fma(a, dH, Pres), s.ec);
    s.ea = fma(ct, dg, s.ea);
  }
  const double Tb = mul(mul(mul(-2.0, C.c_curv), a), ig3);
  double W2 = fma(mul(2.0, ct), ig, mul(mul(-3.0, iW), mul(Tb, Tt)));  // 2 dE/dW
  const double kb2 = mul(-2.0, Tb);
  double lb = mul(Tb, E22), kb = mul(kb2, E12), nb = mul(Tb, E11);
  double F11 = -mul(kb2, n), F12 = mul(Tb, k2), F22 = -mul(kb2, l);  // 2 dE/dE11, dE/dE12, 2 dE/dE22
  if constexpr (KG_REG) {
    const double Q = fma(l, n, -mul(k, k)), iW2 = mul(iW, iW), cg = mul(C.c_gauss, g0);
    if (on) s.ec = fma(cg, fma(Q, iW2, -0.25 * kSafety), s.ec);
    const double Qb = mul(cg, iW2);
    W2 = fma(mul(mul(-4.0, Qb), Q), iW, W2);
    lb = fma(Qb, n, lb);
    kb = fma(Qb, k2, kb);
    nb = fma(Qb, l, nb);
    const double is = rsqrt(mul(E11, E22)), val = mul(E12, is), dv = __dsub_rn(val, rr0), kdv = mul(C.k_reg, dv),
                 vb = mul(2.0, kdv);
    if (on) s.er = fma(kdv, dv, s.er);
    const double vv = mul(mul(vb, val), mul(is, is));
    const double r11 = -mul(vv, E22), r12 = mul(vb, is), r22 = -mul(vv, E11);  // E22 / (E11 E22) = 1 / E11
    F11 = __dadd_rn(F11, r11);
    F12 = __dadd_rn(F12, r12);
    F22 = __dadd_rn(F22, r22);
    if (on && reg_alpha) {
      // sum over the control points of (b_u Kreg_u + b_v Kreg_v) X = Kreg_u Ru + Kreg_v Rv
      s.da[0] = fma(am1[0], (r11 * Ru.x + r12 * Rv.x) * Ru.x + (r22 * Rv.x + r12 * Ru.x) * Rv.x, s.da[0]);
      s.da[1] = fma(am1[1], (r11 * Ru.y + r12 * Rv.y) * Ru.y + (r22 * Rv.y + r12 * Ru.y) * Rv.y, s.da[1]);
      s.da[2] = fma(am1[2], (r11 * Ru.z + r12 * Rv.z) * Ru.z + (r22 * Rv.z + r12 * Ru.z) * Rv.z, s.da[2]);
    }
  }
  auto mix = [&](double u, double uv, double v, double w) { return fma(lb, u, fma(kb, uv, fma(nb, v, mul(W2, w)))); };
  const Vec3<double> mb = {mix(Suu.x, Suv.x, Svv.x, m.x), mix(Suu.y, Suv.y, Svv.y, m.y), mix(Suu.z, Suv.z, Svv.z, m.z)};
  // F11 Ru + F12 Rv + Rv x mb and F22 Rv + F12 Ru + mb x Ru
  K[0] = {fma(Rv.y, mb.z, fma(-Rv.z, mb.y, fma(F11, Ru.x, mul(F12, Rv.x)))),
          fma(Rv.z, mb.x, fma(-Rv.x, mb.z, fma(F11, Ru.y, mul(F12, Rv.y)))),
          fma(Rv.x, mb.y, fma(-Rv.y, mb.x, fma(F11, Ru.z, mul(F12, Rv.z))))};
  K[1] = {fma(mb.y, Ru.z, fma(-mb.z, Ru.y, fma(F22, Rv.x, mul(F12, Ru.x)))),
          fma(mb.z, Ru.x, fma(-mb.x, Ru.z, fma(F22, Rv.y, mul(F12, Ru.y)))),
          fma(mb.x, Ru.y, fma(-mb.y, Ru.x, fma(F22, Rv.z, mul(F12, Ru.z))))};
  K[2] = {mul(lb, m.x), mul(lb, m.y), mul(lb, m.z)};
  K[3] = {mul(kb, m.x), mul(kb, m.y), mul(kb, m.z)};
  K[4] = {mul(nb, m.x), mul(nb, m.y), mul(nb, m.z)};
}

// Global data of one face, loaded one face ahead.
struct Ahead {
  double X[3] = {0, 0, 0};  // the lane's control point in its lattice image
  double g0 = 1, rr0 = 0, P2 = 0, Hbar = 0, Pres = 0;
  int dest = -1;            // -1: no slot (the lane has no control point, or the half-warp no face)
  bool on = false;          // the half-warp has a face of its own
};

// Face f of [.., end); a half-warp past the end takes face end - 1 along (on
// false: nothing of it is summed or written).
template <int NCP, int NPT, bool KG_REG>
__device__ __forceinline__ void load(const FaceSrc &S, const SurfaceParams &P, int f, int end, int lane, Ahead &a) {
  a.on = f < end;
  f = min(f, end - 1);
  if (lane < NCP) {
    const uint32_t packed = __ldg(&S.cp[(size_t)f * NCP + lane]);
    const int v = (int)(packed & kVertexMask), code = (int)(packed >> kVertexBits);
#pragma unroll
    for (int c = 0; c < 3; ++c) a.X[c] = S.r[3 * (size_t)v + c];
    if (code != 13) {  // a periodic image
      const int im[3] = {code % 3 - 1, (code / 3) % 3 - 1, code / 9 - 1};
#pragma unroll
      for (int c = 0; c < 3; ++c)
        a.X[c] = fma((double)im[2], P.box[2][c], fma((double)im[1], P.box[1][c], fma((double)im[0], P.box[0][c], a.X[c])));
    }
    a.dest = a.on ? __ldg(&S.dest[(size_t)f * NCP + lane]) : -1;
  }
  if (lane < NPT) {
    a.g0 = __ldg(&S.g0[(size_t)f * NPT + lane]);
    if constexpr (KG_REG) a.rr0 = __ldg(&S.rr0[(size_t)f * NPT + lane]);
    a.P2 = __ldg(&S.comp[3 * (size_t)f]);
    a.Hbar = __ldg(&S.comp[3 * (size_t)f + 1]);
    a.Pres = __ldg(&S.comp[3 * (size_t)f + 2]);
  }
}

// Stages a patch type's table and gives this lane's five row exponents.
template <int NCP, int NPT>
__device__ __forceinline__ void stage(Smem<NCP, NPT> &sm, const int *__restrict__ table, int eb[5]) {
  const int4 *t = reinterpret_cast<const int4 *>(table);
  int4 *b = &sm.B[0][0];
  for (int i = threadIdx.x; i < NPT * Smem<NCP, NPT>::ROW4; i += kThreads) b[i] = __ldg(t + i);
  if constexpr (NCP & 1)  // the padding of the last pair stays zero
    for (int i = threadIdx.x; i < kHW * 3; i += kThreads)
      sm.X[i / 3][i % 3][Smem<NCP, NPT>::PAIRS - 1] = make_int4(0, 0, 0, 0);
  const int lane = threadIdx.x & 15;
#pragma unroll
  for (int k = 0; k < 5; ++k)
    eb[k] = lane < NPT ? __ldg(table + (size_t)NPT * 4 * Smem<NCP, NPT>::ROW4 + 8 * lane + k) : 0;
}

// One face per half-warp.
//  1. lanes = control points: coordinates relative to the patch corner, times
//     alpha, as limbs scaled by the largest of their coordinate;
//  2. lanes = quadrature points: five contractions, pointwise step, adjoints as
//     limbs scaled by the largest of their coordinate over points and rows;
//  3. lanes = control points: the adjoints' contraction with the rows; the
//     alpha-scaled partial to its slot.
template <int NCP, int NPT, bool KG_REG>
__device__ __forceinline__ void face(Smem<NCP, NPT> &sm, int hw, int lane, const int eb[5], const Ahead &cur,
                                     const double alpha[3], const double am1[3], bool unit_alpha, const PointCoef &C,
                                     bool reg_alpha, bool want_da, double *__restrict__ partial, Sums &sums) {
  constexpr int PAIRS = Smem<NCP, NPT>::PAIRS;
  const double nan = __longlong_as_double(0x7FF8000000000000ll);
  // ---- 1. control points
  double xl[3];
  int top[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    xl[c] = __dsub_rn(cur.X[c], __shfl_sync(0xFFFFFFFFu, cur.X[c], 0, 16));
    if (!unit_alpha) xl[c] = __dmul_rn(alpha[c], xl[c]);
    if (lane >= NCP) xl[c] = 0.0;
    top[c] = max(half_max(exponent_field(xl[c])), kPosLow);
  }
  const bool far = max(top[0], max(top[1], top[2])) > kPosHigh;  // non-finite or out of range
  if (lane < NCP) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
      reinterpret_cast<int2 *>(sm.X[hw][c])[lane] = to_limbs(xl[c], top[c] - exponent_field(xl[c]), fixed::kRowBits);
  }
  __syncwarp();
  // ---- 2. quadrature points
  int adj[3] = {0, 0, 0};  // largest biased exponent of the lane's adjoints, row exponents added
  Vec3<double> K[5];
  if (lane < NPT) {
    const int4 *B = sm.B[lane];
    long long hh[5][3], hl[5][3];
#pragma unroll
    for (int k = 0; k < 5; ++k)
#pragma unroll
      for (int c = 0; c < 3; ++c) hh[k][c] = hl[k][c] = 0;
#pragma unroll 1
    for (int j = 0; j < PAIRS; ++j) {
      int4 x[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) x[c] = sm.X[hw][c][j];
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const int4 b = B[k * PAIRS + j];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          hh[k][c] = mad_wide(b.x, x[c].x, hh[k][c]);
          hl[k][c] = mad_wide(b.x, x[c].y, hl[k][c]);
          hl[k][c] = mad_wide(b.y, x[c].x, hl[k][c]);
          hh[k][c] = mad_wide(b.z, x[c].z, hh[k][c]);
          hl[k][c] = mad_wide(b.z, x[c].w, hl[k][c]);
          hl[k][c] = mad_wide(b.w, x[c].z, hl[k][c]);
        }
      }
    }
    // (hh 2^56 + hl 2^28) 2^(eb - 56) 2^(ex - 56), as (2 hh + hl 2^-27) 2^(eb + ex - 57)
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      double v[3];
#pragma unroll
      for (int c = 0; c < 3; ++c)
        v[c] = from_fixed((hh[k][c] << 1) + (hl[k][c] >> 27), eb[k] + top[c] - fixed::kBias - 57);
      K[k] = {v[0], v[1], v[2]};
    }
    if (far) K[0].x = nan;
    point<KG_REG>(K, C, cur.g0, cur.rr0, cur.P2, cur.Hbar, cur.Pres, cur.on, reg_alpha, am1, sums);
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      adj[0] = max(adj[0], exponent_field(K[k].x) + eb[k]);
      adj[1] = max(adj[1], exponent_field(K[k].y) + eb[k]);
      adj[2] = max(adj[2], exponent_field(K[k].z) + eb[k]);
    }
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) adj[c] = max(half_max(adj[c]), kAdjLow);
  if (lane < NPT) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      int2 q[6];
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const double v = c == 0 ? K[k].x : c == 1 ? K[k].y : K[k].z;
        q[k] = to_limbs(v, adj[c] - exponent_field(v) - eb[k], fixed::kAdjointBits);
      }
      q[5] = make_int2(0, 0);
#pragma unroll
      for (int h = 0; h < 3; ++h)
        sm.K[hw][lane][c][h] = make_int4(q[2 * h].x, q[2 * h].y, q[2 * h + 1].x, q[2 * h + 1].y);
    }
  }
  __syncwarp();
  // ---- 3. control points again
  if (lane < NCP) {
    long long hh[3] = {0, 0, 0}, hl[3] = {0, 0, 0};
#pragma unroll 1
    for (int p = 0; p < NPT; ++p) {
      const int2 *B = reinterpret_cast<const int2 *>(sm.B[p]) + lane;
      int2 b[5];
#pragma unroll
      for (int k = 0; k < 5; ++k) b[k] = B[2 * PAIRS * k];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int4 q0 = sm.K[hw][p][c][0], q1 = sm.K[hw][p][c][1];
        const int2 q2 = *reinterpret_cast<const int2 *>(&sm.K[hw][p][c][2]);
        auto add = [&](const int2 w, int qh, int ql) {
          hh[c] = mad_wide(w.x, qh, hh[c]);
          hl[c] = mad_wide(w.x, ql, hl[c]);
          hl[c] = mad_wide(w.y, qh, hl[c]);
        };
        add(b[0], q0.x, q0.y);
        add(b[1], q0.z, q0.w);
        add(b[2], q1.x, q1.y);
        add(b[3], q1.z, q1.w);
        add(b[4], q2.x, q2.y);
      }
    }
    // (hh 2^56 + hl 2^28) 2^-56 2^(adj - 54), as (hh + hl 2^-28) 2^(adj - 54)
    double G[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      G[c] = from_fixed(hh[c] + ((hl[c] + (1ll << 27)) >> 28), adj[c] - fixed::kBias - 54);
      if (adj[c] > kAdjHigh) G[c] = nan;
    }
    if (cur.dest >= 0) {
      // dE/dalpha_c = sum_x G_xc (X - X_0)_xc / alpha_c: the patch gradient sums to
      // zero, so coordinates relative to the corner give the same sum.
      if (want_da)
#pragma unroll
        for (int c = 0; c < 3; ++c) sums.da[c] = fma(G[c], xl[c], sums.da[c]);
#pragma unroll
      for (int c = 0; c < 3; ++c) partial[3 * (size_t)cur.dest + c] = unit_alpha ? G[c] : alpha[c] * G[c];
    }
  }
  __syncwarp();  // the next face overwrites X and K
}

}  // namespace f64
}  // namespace dev
}  // namespace umcp
