// Kernels of the membrane-surface hot path. See kernels.cuh for the model
// and launch.h for the contracts.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <type_traits>

#include "device_common.cuh"
#include "face32.cuh"
#include "geo.cuh"
#include "geo32_table.h"
#include "kernels.cuh"
#include "launch.h"
#include "launch_host.h"
#include "philox.h"

namespace umcp {
namespace dev {


// ---------------------------------------------------------------- tensor-core face pass
//
// Regular faces in the precision form, with the two basis contractions on the
// 5th-generation tensor cores (tcgen05, kind::f16 on fp16 hi/lo splits) and the
// pointwise energy and adjoint on the FP32 pipes. A CTA owns a tile of 128
// faces (the MMA's M; face = TMEM lane) and 256 threads: thread (face, half)
// takes the half-th quadrature point of each 2-point chunk.
//
// Affine centring. The box splines reproduce affine functions, so with the
// patch frame Eu = X2 - X0, Ev = X1 - X0 (control points 2 and 1 sit at
// lattice (1,0) and (0,1)) and X'_x = X_x - X0 - u_x Eu - v_x Ev:
//   Ru = Eu + sum b_u X',  Rv = Ev + sum b_v X',  S.. = sum b_.. X'.
// X' is of the size of the curvature, not of the patch, so the fp16 split
// errors scale with the curvature terms themselves.
//
// Per chunk j (points 2j, 2j+1):
//   GEMM1_j  D1[f, n] = sum_x X'[f, x] B1_j[n, x]      n = 8 h + k (point 2j+h, kind k)
//   pointwise: K -> energy terms, adjoint Kb (tcgen05.ld from D1, tcgen05.st into A2)
//   GEMM2_j  D2[f, x] += sum_n A2[f, n] B2_j[x, n]    (A from tensor memory)
// GEMM2_j and GEMM1_{j+1} are issued together behind one commit.
namespace tc {
// Tensor-core form of the regular-face pass (precision form, 12 control
// points, 15 quadrature points). A CTA owns a tile of 128 faces, one face per
// TMEM lane, and evaluates its points in four chunks of four; thread half h
// (threads 128 h .. 128 h + 127) evaluates points 4 j + 2 h and 4 j + 2 h + 1
// of chunk j and owns control points 8 h .. 8 h + 7 (those below 12).
//
// Per chunk, with fp16 operands split in two (x = hi + lo, about 22 bits) and
// FP32 accumulation in TMEM:
//   GEMM1  D1[face][n] = sum_k X'[face][k] B1[n][k]   per coordinate, K = 32, N = 48
//   GEMM2  D2[face][n] = sum_k Kb[face][k] B2[n][k]   per coordinate, K = 48, N = 32
// X' are the affine-centred control points, Kb the pointwise adjoints. The
// three products of a split (hi hi, lo hi, hi lo) come out of one pass:
// A = [a_hi | a_lo] along K and B's columns [b_hi | b_lo] along N, the lo-lo
// block left zero. Each instruction costs about the same time whatever its N,
// so the contractions are laid out for the fewest instructions: 6 (GEMM1) +
// 9 (GEMM2) per chunk, 60 per tile.
//
// Scaling: every A row is scaled by a power of two that puts its largest
// magnitude in [2^13, 2^14) (per face, coordinate and, for Kb, chunk), the
// basis by 2^8, so neither fp16 half of an operand leaves fp16's normal range
// in a way that costs accuracy. D2 is read back per chunk and summed in
// registers, which lets each chunk's Kb carry its own scale.
constexpr int kThreads = 256, kFaces = 128, kNpt = 15, kNcp = 12, kChunks = 4;
constexpr int kN1 = 48, kK1 = 32, kN2 = 32, kK2 = 48;
constexpr int kSbo1 = kK1 / 8 * 128, kSbo2 = kK2 / 8 * 128;  // bytes between 8-row core-matrix groups
constexpr uint32_t kTmemCols = 256, kD1 = 0, kD2 = 3 * kN1;  // TMEM column bases
constexpr float kBasisScale = 256.f, kInvBasisScale = 1.f / 256.f;
// lattice position of control point x in the regular patch (ceff order)
__constant__ int kLatU[12] = {0, 0, 1, 1, 0, -1, -1, -1, 0, 1, 2, 2};
__constant__ int kLatV[12] = {0, 1, 0, -1, -1, 0, 1, 2, 2, 1, 0, -1};

struct Smem {
  uint4 A1[3][kFaces * kK1 / 8];  // X' (hi at k 0..11, lo at k 16..27), K-major core matrices of 8 rows x 16 B
  uint4 A2[3][kFaces * kK2 / 8];  // Kb: thread half h's slots at k 24 h .. 24 h + 23
  uint4 B1[kChunks][kN1 * kK1 / 8];
  uint4 B2[kChunks][kN2 * kK2 / 8];
  float xmax[2][3][kFaces];       // per-row maxima exchanged between the two thread halves
  float Dd[3][kNcp][kFaces];      // control points' change from the reference state (FP32, per face)
  float Buv[kNpt][2][kNcp];       // basis rows u, v in FP32, for the area strain's tangent changes
  f32::Coef C[16];                // each point's coefficients
  uint64_t mbar;
  uint32_t tmem;
  int abort;
};
constexpr size_t kSmemBytes = sizeof(Smem) + 1024;

// byte offset of element (row, k) of a K-major fp16 operand whose 8-row groups are sbo bytes apart
__host__ __device__ constexpr int core_off(int row, int k, int sbo) {
  return (row >> 3) * sbo + (k >> 3) * 128 + (row & 7) * 16 + (k & 7) * 2;
}
// GEMM1 column of thread half h's slot s (s < 20): slots 0..15 at 16 h + s,
// slots 16..19 at 32 + 8 h + s - 16, so both halves read them with one x16
// and one x8 load at aligned columns.
__host__ __device__ constexpr int d1_col(int h, int s) { return s < 16 ? 16 * h + s : 32 + 8 * h + (s - 16); }

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
// shared-memory matrix descriptor: K-major, no swizzle, 128 B between K-adjacent core matrices
__device__ __forceinline__ uint64_t sdesc(uint32_t addr, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
         ((uint64_t)1 << 46);
}
// instruction descriptor: D F32, A and B F16, both K-major, M = 128
__host__ __device__ constexpr uint32_t idesc(uint32_t n) { return (1u << 4) | ((n >> 3) << 17) | ((128u >> 4) << 24); }

__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t id, uint32_t acc) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
               ::"r"(d), "l"(a), "l"(b), "r"(id), "r"(acc));
}
__device__ __forceinline__ void commit(uint64_t *mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(mbar)));
}
// Bounded wait on the mbarrier's phase; false when it gave up.
__device__ __forceinline__ bool wait_phase(uint64_t *mbar, uint32_t phase) {
  uint32_t done = 0;
  for (int it = 0; it < (1 << 24) && !done; ++it)
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(done) : "r"(smem_u32(mbar)), "r"(phase));
  return done != 0;
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;"); }

// TMEM loads of 8 + 8 consecutive columns of this warp's 32 lanes; the wait is
// inside the same statement, so no use of a result can move above it.
__device__ __forceinline__ void ld8_8(uint32_t ta, uint32_t tb, float v[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%16];\n"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%17];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(ta), "r"(tb));
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// The GEMM1 results of this thread's two points, all three coordinates: per
// coordinate c, 16 + 8 columns at ta[c], tb[c], with one wait.
__device__ __forceinline__ void ld_d1(const uint32_t ta[3], const uint32_t tb[3], float v[3][24]) {
  uint32_t r[72];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%72];\n"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16,%17,%18,%19,%20,%21,%22,%23}, [%73];\n"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%24,%25,%26,%27,%28,%29,%30,%31,%32,%33,%34,%35,%36,%37,%38,%39}, [%74];\n"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%40,%41,%42,%43,%44,%45,%46,%47}, [%75];\n"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%76];\n"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%64,%65,%66,%67,%68,%69,%70,%71}, [%77];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]), "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]), "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]), "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]), "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63]), "=r"(r[64]), "=r"(r[65]), "=r"(r[66]), "=r"(r[67]), "=r"(r[68]), "=r"(r[69]), "=r"(r[70]), "=r"(r[71])
      : "r"(ta[0]), "r"(tb[0]), "r"(ta[1]), "r"(tb[1]), "r"(ta[2]), "r"(tb[2]));
#pragma unroll
  for (int i = 0; i < 72; ++i) v[i / 24][i % 24] = __uint_as_float(r[i]);
}
// 2^e with m * 2^e in [2^13, 2^14) for a finite m > 0 (and its inverse); for
// m = 0 or tiny m the largest scale whose inverse is a normal float; an
// infinite or NaN m gives a small scale, so the values stay non-finite.
__device__ __forceinline__ void pow2_scale(float m, float &s, float &inv) {
  const int e = (int)((__float_as_uint(m) >> 23) & 0xFFu);
  const int f = e == 0 ? 253 : min(253, 267 - e);  // biased exponent of the scale
  s = __uint_as_float((uint32_t)f << 23);
  inv = __uint_as_float((uint32_t)(254 - f) << 23);
}
// (a, b) as an fp16 pair, a in the low half
__device__ __forceinline__ uint32_t cvt2(float a, float b) {
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}
// x0, x1 (already scaled) = hi + lo: hi rounded to 11 significant bits by
// Veltkamp's split (factor 2^13 + 1; explicitly rounded operations, so
// nothing is contracted), exact in fp16; lo = x - hi, exact in FP32 and
// rounded to fp16.
__device__ __forceinline__ void split_pair(float x0, float x1, uint32_t &hi, uint32_t &lo) {
  const float g0 = __fmul_rn(x0, 8193.f), g1 = __fmul_rn(x1, 8193.f);
  const float h0 = __fsub_rn(g0, __fsub_rn(g0, x0)), h1 = __fsub_rn(g1, __fsub_rn(g1, x1));
  hi = cvt2(h0, h1);
  lo = cvt2(__fsub_rn(x0, h0), __fsub_rn(x1, h1));
}

// CTA set-up: mbarrier, TMEM, the basis operands of every chunk, the points' coefficients.
__device__ void setup(Smem &sm, const double *__restrict__ basis, const double *__restrict__ weight,
                      const SurfaceParams &P, double dudv) {
  const int tid = threadIdx.x;
  // fp16 hi or lo part of the scaled basis value of point p, derivative d, control point x
  auto bval = [&](int p, int d, int x, bool lo) -> __half {
    const double b = basis[((size_t)p * 5 + d) * kNcp + x] * (double)kBasisScale;
    const __half hi = __float2half_rn((float)b);
    return lo ? __float2half_rn((float)(b - (double)__half2float(hi))) : hi;
  };
  __half *b1 = reinterpret_cast<__half *>(&sm.B1[0][0]);
  for (int e = tid; e < kChunks * kN1 * kK1; e += kThreads) {
    const int j = e / (kN1 * kK1), n = (e / kK1) % kN1, k = e % kK1;
    const int h = n < 32 ? n >> 4 : (n - 32) >> 3, s = n < 32 ? n & 15 : 16 + ((n - 32) & 7);
    const int x = k & 15;
    __half v = __float2half_rn(0.f);
    if (s < 20 && x < kNcp) {
      const int q = (s % 10) / 5, d = s % 5, p = 4 * j + 2 * h + q;
      if (p < kNpt) {
        if (s < 10) v = bval(p, d, x, false);  // (a_hi + a_lo) b_hi
        else if (k < 16) v = bval(p, d, x, true);  // a_hi b_lo
      }
    }
    b1[(size_t)j * kN1 * kK1 + core_off(n, k, kSbo1) / 2] = v;
  }
  __half *b2 = reinterpret_cast<__half *>(&sm.B2[0][0]);
  for (int e = tid; e < kChunks * kN2 * kK2; e += kThreads) {
    const int j = e / (kN2 * kK2), n = (e / kK2) % kN2, k = e % kK2;
    const int x = n & 15, h = k / 24, s = k % 24;
    __half v = __float2half_rn(0.f);
    if (x < kNcp && s < 20) {
      const int q = (s % 10) / 5, d = s % 5, p = 4 * j + 2 * h + q;
      if (p < kNpt) {
        if (s < 10) v = bval(p, d, x, n >= 16);  // a_hi rows: [b_hi | b_lo]
        else if (n < 16) v = bval(p, d, x, false);  // a_lo rows: [b_hi | 0]
      }
    }
    b2[(size_t)j * kN2 * kK2 + core_off(n, k, kSbo2) / 2] = v;
  }
  if (tid < kNpt) sm.C[tid] = f32::point_coef(P, weight[tid], dudv);
  for (int e = tid; e < kNpt * 2 * kNcp; e += kThreads) {
    const int p = e / (2 * kNcp), k = (e / kNcp) % 2, x = e % kNcp;
    sm.Buv[p][k][x] = (float)basis[((size_t)p * 5 + k) * kNcp + x];
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sm.mbar)));
    asm volatile("fence.mbarrier_init.release.cluster;");
    sm.abort = 0;
  }
  if ((tid >> 5) == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("fence.proxy.async.shared::cta;");
  fence_before();
  __syncthreads();
  fence_after();
}

__device__ void teardown(Smem &sm, uint32_t phase, bool pending) {
  // An aborted tile may leave MMAs in flight: give them a bounded wait before
  // the tensor memory they write is freed.
  if (pending && threadIdx.x == 0) wait_phase(&sm.mbar, phase);
  fence_before();
  __syncthreads();
  fence_after();
  if ((threadIdx.x >> 5) == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(sm.tmem), "r"(kTmemCols));
}

__device__ __forceinline__ void issue_gemm1(Smem &sm, uint32_t tmem, int j) {
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int ks = 0; ks < kK1 / 16; ++ks)
      mma(tmem + kD1 + kN1 * c, sdesc(smem_u32(sm.A1[c]) + 256 * ks, kSbo1), sdesc(smem_u32(sm.B1[j]) + 256 * ks, kSbo1),
          idesc(kN1), ks);
}
__device__ __forceinline__ void issue_gemm2(Smem &sm, uint32_t tmem, int j) {
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int ks = 0; ks < kK2 / 16; ++ks)
      mma(tmem + kD2 + kN2 * c, sdesc(smem_u32(sm.A2[c]) + 256 * ks, kSbo2), sdesc(smem_u32(sm.B2[j]) + 256 * ks, kSbo2),
          idesc(kN2), ks);
}

// Adds chunk D2 (scaled by inv, per coordinate) into G: the hi- and lo-basis columns of this thread's control points.
__device__ __forceinline__ void gather_d2(uint32_t tmem, uint32_t lane_base, int h, const float inv[3], float G[3][8]) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    float v[16];
    ld8_8(tmem + lane_base + kD2 + kN2 * c + 8 * h, tmem + lane_base + kD2 + kN2 * c + 16 + 8 * h, v);
#pragma unroll
    for (int i = 0; i < 8; ++i) G[c][i] += (v[i] + v[8 + i]) * inv[c];
  }
}

// One tile of up to 128 faces [first, first + count) of source S. Returns
// false if a wait gave up (the CTA then stops).
__device__ bool tile(Smem &sm, const FaceSrc &S, const SurfaceParams &P, const float alpha[3], const float ialpha[3],
                     const float am1[3], float k_reg, int first, int count,
                     float *__restrict__ partial,
                     KahanSums<6> &acc, uint32_t &phase) {
  const int tid = threadIdx.x, fs = tid & (kFaces - 1), h = tid >> 7;
  const uint32_t tmem = sm.tmem, lane_base = (uint32_t)(32 * ((tid >> 5) & 3)) << 16;
  const bool active = fs < count;
  const int f = first + fs;
  const int nx = h == 0 ? 8 : kNcp - 8;  // control points of this thread
  float Eu[3] = {0, 0, 0}, Ev[3] = {0, 0, 0}, sA[3], iA[3];
  float P2 = 0, Hbar = 0, Pres = 0;
  {
    float xp[8][3];
#pragma unroll
    for (int i = 0; i < 8; ++i) xp[i][0] = xp[i][1] = xp[i][2] = 0.f;
    if (active) {
      const uint32_t *cp = S.cp + (size_t)f * kNcp;
      // the corner (control point 0) is in the home image: coordinates are relative to its hi/lo pair
      const int v0 = (int)(__ldg(&cp[0]) & kVertexMask);
      float chi[3], clo[3], cd[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const size_t at = kPosStride * (size_t)v0 + c;
        chi[c] = S.rhi[at];
        clo[c] = S.rlo[at];
        cd[c] = S.dsp[at];
      }
      // out = alpha L; with d given, d = (alpha - 1) L + (dsp - dsp of the corner), the change from
      // the reference state (as in the thread-per-face kernel)
      auto local = [&](uint32_t packed, float out[3], float *d = nullptr) {
        const int v = (int)(packed & kVertexMask), code = (int)(packed >> kVertexBits);
        const int im[3] = {code % 3 - 1, (code / 3) % 3 - 1, code / 9 - 1};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          float sh = 0.f, she = 0.f, shl = 0.f;
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            float t, e;
            two_sum(sh, (float)im[d] * P.box_hi[d][c], t, e);
            sh = t;
            she += e;
            shl += (float)im[d] * P.box_lo[d][c];
          }
          float s1, e1, s2, e2;
          const size_t at = kPosStride * (size_t)v + c;
          const float hi = S.rhi[at], lo = S.rlo[at];
          two_sum(hi, sh, s1, e1);
          two_sum(s1, -chi[c], s2, e2);
          const float l = s2 + ((e1 + e2) + ((lo - clo[c]) + (she + shl)));
          out[c] = alpha[c] * l;
          if (d) d[c] = fmaf(am1[c], l, S.dsp[at] - cd[c]);
        }
      };
      local(__ldg(&cp[1]), Ev);  // lattice (0,1)
      local(__ldg(&cp[2]), Eu);  // lattice (1,0)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (i < nx) {
          const int x = 8 * h + i;
          float xl[3], dx[3];
          local(__ldg(&cp[x]), xl, dx);
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            xp[i][c] = xl[c] - (float)kLatU[x] * Eu[c] - (float)kLatV[x] * Ev[c];
            sm.Dd[c][x][fs] = dx[c];
          }
        }
      }
      P2 = S.compf[3 * (size_t)f];
      Hbar = S.compf[3 * (size_t)f + 1];
      Pres = S.compf[3 * (size_t)f + 2];
    }
    // one scale per face and coordinate, from the largest |X'| of both halves
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      float m = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) m = fmaxf(m, fabsf(xp[i][c]));
      sm.xmax[h][c][fs] = m;
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      pow2_scale(fmaxf(sm.xmax[0][c][fs], sm.xmax[1][c][fs]), sA[c], iA[c]);
      uint32_t whi[4], wlo[4];
#pragma unroll
      for (int i = 0; i < 8; i += 2) split_pair(xp[i][c] * sA[c], xp[i + 1][c] * sA[c], whi[i / 2], wlo[i / 2]);
      sm.A1[c][core_off(fs, 8 * h, kSbo1) / 16] = make_uint4(whi[0], whi[1], whi[2], whi[3]);
      sm.A1[c][core_off(fs, 16 + 8 * h, kSbo1) / 16] = make_uint4(wlo[0], wlo[1], wlo[2], wlo[3]);
      iA[c] *= kInvBasisScale;
    }
  }
  asm volatile("fence.proxy.async.shared::cta;");
  fence_before();
  __syncthreads();
  fence_after();
  if (tid == 0) {
    issue_gemm1(sm, tmem, 0);
    commit(&sm.mbar);
  }
  float e3[3] = {0, 0, 0}, G[3][8], iK[3] = {0, 0, 0};
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int i = 0; i < 8; ++i) G[c][i] = 0.f;
  bool ok = true;
#pragma unroll 1
  for (int j = 0; j < kChunks; ++j) {
    float g0[2] = {1.f, 1.f}, rr0[2] = {0.f, 0.f};
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int p = 4 * j + 2 * h + q;
      if (active && p < kNpt) {
        g0[q] = S.g0f[(size_t)f * kNpt + p];
        rr0[q] = S.rr0f[(size_t)f * kNpt + p];
      }
    }
    // warp 0 polls the mbarrier; the other warps sleep at the barrier
    ok = !__syncthreads_or((tid >> 5) == 0 && !wait_phase(&sm.mbar, phase)) && ok;
    phase ^= 1u;
    fence_after();
    if (j > 0) gather_d2(tmem, lane_base, h, iK, G);
    // the five contractions of both points, per coordinate: slot hi + slot lo
    Vec3<float> K[2][5];
    float v3[3][24];
    {
      const uint32_t t0 = tmem + lane_base + kD1;
      const uint32_t ta[3] = {t0 + 16 * h, t0 + kN1 + 16 * h, t0 + 2 * kN1 + 16 * h};
      const uint32_t tb[3] = {t0 + 32 + 8 * h, t0 + kN1 + 32 + 8 * h, t0 + 2 * kN1 + 32 + 8 * h};
      ld_d1(ta, tb, v3);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float *v = v3[c];
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int d = 0; d < 5; ++d) {
          const int shi = 5 * q + d, slo = 10 + 5 * q + d;
          const float val = (v[shi] + v[slo]) * iA[c];
          (c == 0 ? K[q][d].x : c == 1 ? K[q][d].y : K[q][d].z) = val;
        }
    }
    float kbv[3][2][5], km[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int p = 4 * j + 2 * h + q;
      K[q][0].x += Eu[0]; K[q][0].y += Eu[1]; K[q][0].z += Eu[2];
      K[q][1].x += Ev[0]; K[q][1].y += Ev[1]; K[q][1].z += Ev[2];
      Vec3<float> Kb[5];
      if (active && p < kNpt) {
        // the tangents' change from the reference state, for the area strain
        Vec3<float> dR[2] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
#pragma unroll
        for (int x = 0; x < kNcp; ++x) {
          const float bu = sm.Buv[p][0][x], bv = sm.Buv[p][1][x];
          const float d0 = sm.Dd[0][x][fs], d1 = sm.Dd[1][x][fs], d2 = sm.Dd[2][x][fs];
          dR[0].x = fmaf(bu, d0, dR[0].x); dR[0].y = fmaf(bu, d1, dR[0].y); dR[0].z = fmaf(bu, d2, dR[0].z);
          dR[1].x = fmaf(bv, d0, dR[1].x); dR[1].y = fmaf(bv, d1, dR[1].y); dR[1].z = fmaf(bv, d2, dR[1].z);
        }
        const f32::Point o = f32::point<true>(K[q], dR, sm.C[p], k_reg, g0[q], rr0[q], P2, Hbar, Pres);
        e3[0] += o.ea; e3[1] += o.ec; e3[2] += o.er;
        Kb[0] = o.Ku;
        Kb[1] = o.Kv;
        Kb[2] = {o.lb * o.m.x, o.lb * o.m.y, o.lb * o.m.z};
        Kb[3] = {o.kb * o.m.x, o.kb * o.m.y, o.kb * o.m.z};
        Kb[4] = {o.nb * o.m.x, o.nb * o.m.y, o.nb * o.m.z};
      } else {
#pragma unroll
        for (int d = 0; d < 5; ++d) Kb[d] = {0.f, 0.f, 0.f};
      }
#pragma unroll
      for (int d = 0; d < 5; ++d) {
        kbv[0][q][d] = Kb[d].x;
        kbv[1][q][d] = Kb[d].y;
        kbv[2][q][d] = Kb[d].z;
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int d = 0; d < 5; ++d) km[c] = fmaxf(km[c], fabsf(kbv[c][q][d]));
      sm.xmax[h][c][fs] = km[c];
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      float sK;
      pow2_scale(fmaxf(sm.xmax[0][c][fs], sm.xmax[1][c][fs]), sK, iK[c]);
      iK[c] *= kInvBasisScale;
      // slots 0..9 hi, 10..19 lo, 20..23 zero; slot 5 q + d is point q's derivative d
      uint32_t hw[5], lw[5];
#pragma unroll
      for (int t = 0; t < 5; ++t) {
        const int s0 = 2 * t, s1 = 2 * t + 1;
        split_pair(kbv[c][s0 / 5][s0 % 5] * sK, kbv[c][s1 / 5][s1 % 5] * sK, hw[t], lw[t]);
      }
      uint4 *row = sm.A2[c];
      row[core_off(fs, 24 * h, kSbo2) / 16] = make_uint4(hw[0], hw[1], hw[2], hw[3]);
      row[core_off(fs, 24 * h + 8, kSbo2) / 16] = make_uint4(hw[4], lw[0], lw[1], lw[2]);
      row[core_off(fs, 24 * h + 16, kSbo2) / 16] = make_uint4(lw[3], lw[4], 0u, 0u);
    }
    asm volatile("fence.proxy.async.shared::cta;");
    fence_before();
    __syncthreads();
    fence_after();
    if (tid == 0) {
      issue_gemm2(sm, tmem, j);
      if (j + 1 < kChunks) issue_gemm1(sm, tmem, j + 1);
      commit(&sm.mbar);
    }
  }
  ok = !__syncthreads_or((tid >> 5) == 0 && !wait_phase(&sm.mbar, phase)) && ok;
  phase ^= 1u;
  if (!ok) return false;
  fence_after();
  gather_d2(tmem, lane_base, h, iK, G);
  // ---- gradient partials of this thread's control points and dE/dalpha;
  // X' comes back from the GEMM1 operand (hi + lo), the lattice part from Eu, Ev
  float da[3] = {0, 0, 0};
  if (active) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const uint4 wh = sm.A1[c][core_off(fs, 8 * h, kSbo1) / 16], wl = sm.A1[c][core_off(fs, 16 + 8 * h, kSbo1) / 16];
      const uint32_t hw[4] = {wh.x, wh.y, wh.z, wh.w}, lw[4] = {wl.x, wl.y, wl.z, wl.w};
      const float ia = iA[c] * kBasisScale;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (i < nx) {
          const int x = 8 * h + i;
          const __half hh = __ushort_as_half((unsigned short)(hw[i / 2] >> (16 * (i & 1))));
          const __half ll = __ushort_as_half((unsigned short)(lw[i / 2] >> (16 * (i & 1))));
          const float xl = (__half2float(hh) + __half2float(ll)) * ia + (float)kLatU[x] * Eu[c] + (float)kLatV[x] * Ev[c];
          const int dst = __ldg(&S.dest[(size_t)f * kNcp + x]);
          partial[kSlot<float> * (size_t)dst + c] = alpha[c] * G[c][i];
          da[c] += G[c][i] * xl * ialpha[c];
        }
      }
    }
  }
  acc.add(0, e3[0]); acc.add(1, e3[1]); acc.add(2, e3[2]);
  acc.add(3, da[0]); acc.add(4, da[1]); acc.add(5, da[2]);
  // the next tile overwrites A1, A2 and the maxima, and its MMAs D1 and D2: everyone is done with them
  fence_before();
  __syncthreads();
  fence_after();
  return true;
}

// Fixed-order block sum of the six per-thread sums into out[6] (global). The
// reduction buffer lies over the Kb operand, which no MMA reads any more.
__device__ void block_sums(Smem &sm, const KahanSums<6> &acc, const SurfaceParams &P, double *out) {
  double(*red)[6] = reinterpret_cast<double(*)[6]>(&sm.A2[0][0]);
  for (int q = 0; q < 6; ++q) red[threadIdx.x][q] = acc.get(q);
  __syncthreads();
  if (threadIdx.x < 6) {
    double s = 0;
    for (int t = 0; t < kThreads; ++t) s += red[t][threadIdx.x];
    out[threadIdx.x] = threadIdx.x < 3 ? s * P.e_scale[0][threadIdx.x] : s;
  }
  __syncthreads();
}
static_assert(sizeof(double) * 6 * kThreads <= sizeof(uint4) * 3 * kFaces * kK2 / 8, "reduction buffer");
}  // namespace tc

// Single mesh: persistent CTAs over the 128-face tiles of the regular group.
__global__ void __launch_bounds__(tc::kThreads, 2)
    face_tc_kernel(FaceLaunch L, const int *__restrict__ dest, SurfaceParams P, const double *__restrict__ r,
                   const float *__restrict__ rhi, const float *__restrict__ rlo, const float *__restrict__ dsp,
                   float *__restrict__ partial, double *__restrict__ blockpart, int *__restrict__ status,
                   FinishArgs fin) {
  extern __shared__ uint8_t tc_smem_raw[];
  tc::Smem &sm = *reinterpret_cast<tc::Smem *>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~(uintptr_t)1023);
  tc::setup(sm, L.basis, L.weight, P, L.dudv);
  const float alpha[3] = {(float)r[3 * P.nv], (float)r[3 * P.nv + 1], (float)r[3 * P.nv + 2]};
  const float ialpha[3] = {1.f / alpha[0], 1.f / alpha[1], 1.f / alpha[2]};
  const float am1[3] = {(float)(r[3 * P.nv] - 1.0), (float)(r[3 * P.nv + 1] - 1.0), (float)(r[3 * P.nv + 2] - 1.0)};
  const FaceSrc src{L.cp, nullptr, nullptr, nullptr, L.g0f, L.rr0f, L.compf, dest, r, rhi, rlo, dsp, L.nfaces};
  KahanSums<6> acc;
  uint32_t phase = 0;
  bool ok = true;
  const int ntiles = (L.nfaces + tc::kFaces - 1) / tc::kFaces;
  for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
    const int first = t * tc::kFaces;
    ok = tc::tile(sm, src, P, alpha, ialpha, am1, (float)P.k_reg, first, min(tc::kFaces, L.nfaces - first), partial,
                  acc, phase);
  }
  if (!ok && threadIdx.x == 0) atomicOr(status, kStatusTimeout);
  tc::teardown(sm, phase, !ok);
  tc::block_sums(sm, acc, P, blockpart + 6 * (size_t)(L.block_base + blockIdx.x));
  count_and_finish<tc::kThreads>(fin, blockpart);
}

__global__ void split_positions_kernel(int n, const double *__restrict__ r, float *__restrict__ hi,
                                       float *__restrict__ lo, const double *__restrict__ r0,
                                       float *__restrict__ dsp) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    store_f32_position(i, r[i], hi, lo, r0, dsp);
}

// A host call's state, read from page-locked host memory where it lies: one
// kernel in place of a copy, a memset and (precision form) the split, and the
// kernel after it follows without a copy engine in between.
__global__ void stage_in_kernel(int n, const double *__restrict__ host_r, double *__restrict__ r,
                                float *__restrict__ hi, float *__restrict__ lo, const double *__restrict__ r0,
                                float *__restrict__ dsp, int *__restrict__ status) {
  grid_dependency_wait();
  grid_dependents(kFewGatherBlocks);
  if (status && blockIdx.x == 0 && threadIdx.x == 0) *status = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double x = host_r[i];
    r[i] = x;
    if (hi && i < n - 3) store_f32_position(i, x, hi, lo, r0, dsp);
  }
}

__device__ __forceinline__ void prefetch_l1(const void *p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

// dst |= *src (one thread): a status word handed on to another.
__global__ void status_merge_kernel(const int *__restrict__ src, int *__restrict__ dst) {
  const int v = *src;
  if (v) *dst |= v;
}

// Coordinate c of a vertex's gradient partials, in order: its slots are
// base + 32 k for k < n (32 vertices interleaved, so the lanes of a warp read
// consecutive slots). Eight slots' loads are issued before they are handed on.
template <typename T, class F>
__device__ __forceinline__ void each_partial(const T *__restrict__ partial, int base, int n, int c, F add) {
  constexpr int kStep = 32 * kSlot<T>;
  const T *q = partial + kSlot<T> * (size_t)base + c;
  int k = 0;
  for (; k + 8 <= n; k += 8) {
    T x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = q[kStep * (size_t)(k + i)];
#pragma unroll
    for (int i = 0; i < 8; ++i) add(x[i]);
  }
  for (; k < n; ++k) add(q[kStep * (size_t)k]);
}
// The same for a thread with one coordinate to gather: the 24 slots of a vertex of
// valence 6 are loaded together, before what else the thread loads and before its
// normals, and added afterwards (each). In rounds of eight behind the normals and
// the status a BD step took 1.0 to 1.2 us more at every size (320 faces 10.0 ->
// 8.9 us, 32,768 26.2 -> 25.0; FP64, 1,280 faces 29.6 -> 28.6). gather_kernel, which
// has no normals to form meanwhile, gained nothing and lost to its registers.
template <typename T>
struct Partials {
  static constexpr int kAhead = 24, kStep = 32 * kSlot<T>;
  const T *base;
  int2 at;
  int c;
  T x[kAhead];
  __device__ __forceinline__ Partials(const T *__restrict__ partial, int2 loc, int coordinate)
      : base(partial), at(loc), c(coordinate) {
    if (at.y < kAhead) return;
    const T *q = partial + kSlot<T> * (size_t)at.x + c;
#pragma unroll
    for (int i = 0; i < kAhead; ++i) x[i] = q[kStep * (size_t)i];
  }
  template <class F>
  __device__ __forceinline__ void each(F add) const {
    if (at.y < kAhead) {
      each_partial(base, at.x, at.y, c, add);
      return;
    }
#pragma unroll
    for (int i = 0; i < kAhead; ++i) add(x[i]);
    for (int k = kAhead; k < at.y; ++k) add(base[kSlot<T> * ((size_t)at.x + 32 * (size_t)k) + c]);
  }
};
struct GradSum {
  float hi, lo;
};
// Kahan-compensated total hi - lo of FP32 partials.
struct KahanPartial {
  GradSum s{0.f, 0.f};
  __device__ __forceinline__ void operator()(float x) {
    const float y = x - s.lo, t = s.hi + y;
    s.lo = (t - s.hi) - y;
    s.hi = t;
  }
  __device__ __forceinline__ double value() const { return __dsub_rn(convert::to_f64(s.hi), convert::to_f64(s.lo)); }
};
struct PlainPartial {
  double s = 0;
  __device__ __forceinline__ void operator()(double x) { s += x; }
  __device__ __forceinline__ double value() const { return s; }
};
template <typename T>
using PartialSum = std::conditional_t<sizeof(T) == 4, KahanPartial, PlainPartial>;
__device__ __forceinline__ GradSum coordinate_sum(const Partials<float> &partials) {
  KahanPartial s;
  partials.each([&](float x) { s(x); });
  return s.s;
}
template <typename T>
__device__ __forceinline__ double coordinate_gradient(const Partials<T> &partials) {
  PartialSum<T> s;
  partials.each([&](T x) { s(x); });
  return s.value();
}
template <typename T>
__device__ __forceinline__ void vertex_gradient(const T *__restrict__ partial, const int *__restrict__ loc, int v,
                                                double gg[3]) {
  const int base = loc[2 * (size_t)v], n = loc[2 * (size_t)v + 1];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    PartialSum<T> s;
    each_partial(partial, base, n, c, [&](T x) { s(x); });
    gg[c] = s.value();
  }
}

// The same sum in the precision form, its compensated total rounded to FP32.
// Eight slots' loads are issued before they are summed (in the same order), so
// each thread keeps 128 bytes in flight; the partials are read once, so the
// loads are marked evict-first. 839 -> 827 us per 256-vesicle step.
__device__ __forceinline__ void vertex_gradient_f32(const float *__restrict__ partial, const int *__restrict__ loc,
                                                    int v, float g[3]) {
  const int base = loc[2 * (size_t)v], n = loc[2 * (size_t)v + 1];
  float s3[3] = {0, 0, 0}, c3[3] = {0, 0, 0};
  auto add = [&](int c, float x) {
    const float y = x - c3[c], t = s3[c] + y;
    c3[c] = (t - s3[c]) - y;
    s3[c] = t;
  };
  const float4 *q = reinterpret_cast<const float4 *>(partial) + base;
  auto add3 = [&](float4 x) {
    add(0, x.x);
    add(1, x.y);
    add(2, x.z);
  };
  int k = 0;
  for (; k + 8 <= n; k += 8) {
    float4 x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = __ldcs(q + 32 * (size_t)(k + i));
#pragma unroll
    for (int i = 0; i < 8; ++i) add3(x[i]);
  }
  for (; k < n; ++k) add3(__ldcs(q + 32 * (size_t)k));
#pragma unroll
  for (int c = 0; c < 3; ++c) g[c] = s3[c] - c3[c];
}

// g += the gathered gradient, one thread per coordinate: on meshes of a few
// thousand vertices a thread per vertex left most of the GPU idle while its 72
// adds (64 cycles each in FP64) ran one after another.
template <typename T>
__global__ void gather_kernel(int nv, const T *__restrict__ partial, const int *__restrict__ off,
                              double *__restrict__ g, int store) {
  grid_dependency_wait();  // the partials come from the face launches
  grid_dependents(kFewGatherBlocks);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 3 * nv; i += gridDim.x * blockDim.x) {
    const int v = i / 3, c = i - 3 * v;
    const int2 at = __ldg(reinterpret_cast<const int2 *>(off) + v);
    PartialSum<T> s;
    each_partial(partial, at.x, at.y, c, [&](T x) { s(x); });
    const double a = s.value();
    g[i] = store ? a : g[i] + a;
  }
}

// Component c of a vertex's three unit normals (Box-Muller on Philox draws). The
// plain path transforms two draws in FP64 (the oracle's draws up to libm
// rounding), the precision form one draw in FP32 from 24-bit uniforms.
// Components 0 and 1 are the cosine and sine of one pair of uniforms, 2 the
// cosine of another. Every kernel takes its normals from here, whether a thread
// draws one component or three, so that all draw the same bits.
__device__ __forceinline__ float normal_f32(const philox_out &o, int c) {
  const float k = 1.0f / 16777216.0f;
  const float ua = ((float)((c == 2 ? o.v[2] : o.v[0]) >> 8) + 0.5f) * k;
  const float ub = ((float)((c == 2 ? o.v[3] : o.v[1]) >> 8) + 0.5f) * k;
  const float rad = sqrtf(-2.0f * logf(ua));
  float sn, cs;
  sincospif(2.0f * ub, &sn, &cs);
  return rad * (c == 1 ? sn : cs);
}
__device__ __forceinline__ double normal_f64(const philox_out &o, int c) {
  const double u1 = philox_u53(o.v[0], o.v[1]), u2 = philox_u53(o.v[2], o.v[3]);
  const double rad = sqrt(-2.0 * log(u1));
  double sn, cs;
  sincospi(2.0 * u2, &sn, &cs);
  return rad * (c == 1 ? sn : cs);
}
// The Philox draw that component c's normal comes from.
template <typename T>
__device__ __forceinline__ philox_out normal_draw(uint64_t seed, uint32_t stream, uint64_t step, int v, int c) {
  if (sizeof(T) == 8 && c == 2) stream |= 0x80000000u;
  return philox4x32_10((uint32_t)v, (uint32_t)step, (uint32_t)(step >> 32), stream, (uint32_t)seed,
                       (uint32_t)(seed >> 32));
}
__device__ __forceinline__ void normals3_f32(uint64_t seed, uint32_t stream, uint64_t step, int v, float n[3]) {
  const philox_out o = normal_draw<float>(seed, stream, step, v, 0);
#pragma unroll
  for (int c = 0; c < 3; ++c) n[c] = normal_f32(o, c);
}
__device__ __forceinline__ void normals3(uint64_t seed, uint32_t stream, uint64_t step, int v, double n[3]) {
  const philox_out o = normal_draw<double>(seed, stream, step, v, 0);
  n[0] = normal_f64(o, 0);
  n[1] = normal_f64(o, 1);
  n[2] = normal_f64(normal_draw<double>(seed, stream, step, v, 2), 2);
}

// Momentum update of the reference leapfrog (src/hd.C:1546-1693), one coordinate.
// Every product and sum is rounded on its own (no fused multiply-add), in the
// reference's order of operations, so each kernel that uses it rounds alike.
__device__ __forceinline__ double kick(const StepArgs &a, double n, double p, double g) {
  double q = p;
  if (a.kind == 2) q = __dsub_rn(q, __dmul_rn(__dmul_rn(a.gamma, a.AK), q));  // friction
  const double half = __dmul_rn(__dmul_rn(-g, a.AK), 0.5);                     // half kick
  q = __dadd_rn(q, half);
  if (a.kind == 1)
    q = __dadd_rn(q, __ddiv_rn(__dmul_rn(__dmul_rn(__ddiv_rn(1.0, a.gamma), a.sigma), n), a.AK));
  else
    q = __dadd_rn(q, __dmul_rn(a.sigma, n));
  return __dadd_rn(q, half);
}

// The update of one coordinate of one step with identity mass: overdamped BD
// (r += -(D dt/kT) g + sqrt(2 D dt) xi), or the leapfrog kick followed by
// r += p AK (p reset for BD). Rounded as kick() is.
__device__ __forceinline__ double coordinate_update(const StepArgs &a, double g, double n, double r, double *p) {
  if (a.kind == 0) return __dadd_rn(r, __dadd_rn(__dmul_rn(-a.mob_dt, g), __dmul_rn(a.sigma, n)));
  const double q = kick(a, n, *p, g);
  *p = a.kind == 1 ? 0.0 : q;
  return __dadd_rn(r, __dmul_rn(q, a.AK));
}

// Step index of the current step: the run's first step plus the run index,
// which the face pass has already advanced past this step.
__device__ __forceinline__ uint64_t current_step(const uint64_t *cnt) { return cnt[0] + cnt[1] - 1; }

// The precision form's overdamped BD step of one vertex: the gradient total
// and the Box-Muller normals stay in FP32, and so does the increment
// -(D dt / kT) g + sqrt(2 D dt) xi (about 2^-23 relative, 1e-9 A at a 0.02 A
// step); it is added to the FP64 position, from which the FP32 copies are
// then taken. The FP64 work is two additions a coordinate, the position and its
// displacement (eight with casts, 14 with the step in FP64; see convert.h). Explicitly
// rounded, so every kernel that inlines it rounds alike.
__device__ __forceinline__ double bd_coordinate_f32(const StepArgs &a, float g, float n, double r) {
  return __dadd_rn(r, convert::to_f64(__fmaf_rn(-a.mob_dt_f, g, __fmul_rn(a.sigma_f, n))));
}
__device__ __forceinline__ void bd_vertex_f32(const float *__restrict__ partial, const int *__restrict__ off, int v,
                                              const StepArgs &a, uint64_t st, double *__restrict__ r,
                                              float *__restrict__ rhi, const double *__restrict__ r0) {
  float g[3], n[3];
  vertex_gradient_f32(partial, off, v, g);
  normals3_f32(a.seed, a.stream, st, v, n);
  double x[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const size_t i = 3 * (size_t)v + c;
    x[c] = bd_coordinate_f32(a, g[c], n[c], r[i]);
    r[i] = x[c];
  }
  store_f32_vertex(v, x, rhi, r0);
}

// Gather fused with the update of the coordinate (overdamped BD, or the
// leapfrog kinds with identity mass), one thread per coordinate: the chain of a
// coordinate (24 adds, a Box-Muller normal, the update) is a third of a
// vertex's, and a 642-vertex mesh spreads over 31 blocks instead of three. The
// redundant Philox rounds are integer work beside it. 642-vertex FP64 BD step:
// 45.6 -> 32.5 us; 128 x 128 membrane, FP32: 39.6 -> 35.6 us (see also Partials).
template <typename T>
__global__ void gather_step_kernel(int nv, const T *__restrict__ partial, const int *__restrict__ off, StepArgs a,
                                   const uint64_t *__restrict__ cnt, double *__restrict__ r, double *__restrict__ p,
                                   float *__restrict__ rhi, float *__restrict__ rlo, const double *__restrict__ r0,
                                   float *__restrict__ dsp, const int *__restrict__ status) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, v = i / 3, c = i - 3 * v;
  const bool on = i < 3 * nv;
  const int2 at = on ? __ldg(reinterpret_cast<const int2 *>(off) + v) : make_int2(0, 0);  // constant: before the wait
  grid_dependency_wait();  // the partials and the status come from the face launches
  grid_dependents(kFewGatherBlocks);
  if (!on) return;
  // every load of the step at once, then the normals, then the sums
  const Partials<T> partials(partial, at, c);
  const int stopped = *status;
  const uint64_t st = current_step(cnt);
  const double r_old = r[i];
  double q = a.kind != 0 ? p[i] : 0.0;
  if (rhi) prefetch_l1(r0 + i);
  if (stopped) return;
  const philox_out o = normal_draw<T>(a.seed, a.stream, st, v, c);
  double x;
  if constexpr (sizeof(T) == 4) {
    const float n = normal_f32(o, c);
    if (a.kind == 0) {
      const GradSum s = coordinate_sum(partials);
      x = bd_coordinate_f32(a, s.hi - s.lo, n, r_old);
    } else {
      x = coordinate_update(a, coordinate_gradient(partials), convert::to_f64(n), r_old, &q);
    }
  } else {
    const double n = normal_f64(o, c);
    x = coordinate_update(a, coordinate_gradient(partials), n, r_old, &q);
  }
  if (a.kind != 0) p[i] = q;
  r[i] = x;
  if (rhi) store_f32_position(i, x, rhi, rlo, r0, dsp);
}

// The mass path's first half, one thread per coordinate: gather the gradient,
// kick the momentum, and leave its FP32 copy where the precision form's M^-1
// apply reads it (x32: see launch_mass_input32; NULL in the plain path).
template <typename T>
__global__ void gather_kick_kernel(int nv, const T *__restrict__ partial, const int *__restrict__ off, StepArgs a,
                                   const uint64_t *__restrict__ cnt, double *__restrict__ p, float *__restrict__ x32,
                                   int ld, const int *__restrict__ status) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, v = i / 3, c = i - 3 * v;
  const bool on = i < 3 * nv;
  const int2 at = on ? __ldg(reinterpret_cast<const int2 *>(off) + v) : make_int2(0, 0);  // constant: before the wait
  grid_dependency_wait();
  grid_dependents(gridDim.x);  // the apply's first loads do not depend on this
  if (!on) return;
  const Partials<T> partials(partial, at, c);
  const int stopped = *status;
  const uint64_t st = current_step(cnt);
  const double p_old = p[i];
  if (stopped) return;
  const double n = normal_f64(normal_draw<double>(a.seed, a.stream, st, v, c), c);
  const double q = kick(a, n, p_old, coordinate_gradient(partials));
  p[i] = q;
  if (x32) x32[ld > 0 ? (size_t)c * ld + v : 4 * (size_t)v + c] = convert::to_f32(q);
}

__global__ void drift_kernel(int nv, StepArgs a, double *__restrict__ r, double *__restrict__ p,
                             const double *__restrict__ qdot, float *__restrict__ rhi, float *__restrict__ rlo,
                             const double *__restrict__ r0, float *__restrict__ dsp, const int *__restrict__ status) {
  grid_dependency_wait();
  if (*status) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 3 * nv; i += gridDim.x * blockDim.x)
    drift(a, i, qdot[i], r, p, rhi, rlo, r0, dsp);
}

// ---------------------------------------------------------------- batches
//
// Many meshes advance together. A tile is a run of up to tile_faces faces of
// one patch type of one mesh (tiles never straddle meshes); a block takes
// tiles in turn and sums each tile's energy terms in a fixed order, and each
// mesh sums its own tiles in listed order. Every mesh keeps its own state,
// noise stream, step counter and step limit, so a mesh's trajectory does not
// depend on what else is in the batch. Tile and job counts are read from
// device memory, so a captured step stays valid when the membership changes.

// ---------------------------------------------------------------- thread-per-face pass
//
// Regular faces of the precision form (12 control points, 15 quadrature
// points), one face per thread. The thread keeps its face's centred control
// points X[12][3] (and their displacements from the reference state) in its
// own columns of shared memory, its gradient sums G[12][3] in registers, and
// walks the 15 points; every thread of a warp reads the same basis row at the
// same time, so the rows come as a launch parameter through the constant cache
// and both contractions are plain multiply-adds:
//   K[k]_c = sum_j B[p][k][j] X[j]_c          (Ru, Rv, Suu, Suv, Svv)
//   G[j]_c += B[p][u][j] Kb[u]_c + B[p][v][j] Kb[v]_c + s[j] m_c,
//   s[j] = B[p][uu][j] lb + B[p][uv][j] kb + B[p][vv][j] nb
// (the adjoints of Suu, Suv, Svv are lb m, kb m, nb m: one scalar per control
// point times the normal instead of three vector rows). Nothing is shuffled
// or transposed per face. Energy terms and dE/dalpha are Kahan-summed per
// thread over its faces and reduced once at the end, in a fixed order.
//
// Bound by issue and the FP32 pipe (64% busy, 0.6 instructions a cycle and
// scheduler). With the rows in shared memory their broadcasts took the 27 reads a
// point of a data path that X and D also need, and registers to hold them: 256
// vesicles of 5,120 faces 657 us, 320,000 planar faces 122 us; as a parameter 550
// and 111 us. Blocks: the batch kernel gains from a fourth a SM (579 us with
// three); the single-mesh kernel's code for three is the faster one (111 against
// 113 us; both reach four).
namespace tpf {
constexpr int kNcp = 12, kNpt = 15, kNc4 = 3;
constexpr int kThreads = 128, kWarps = kThreads / 32, kMinBlocks = 3, kBatchMinBlocks = 4;
struct Smem {
  // each thread's centred control points, coordinate-major: float4 3 c + q
  // holds coordinate c of control points 4 q .. 4 q + 3; the 144-byte stride
  // is an odd number of 16-byte chunks, so the float4 reads of a warp do not
  // conflict
  float4 X[kThreads][9];
  float4 D[kThreads][9];  // the same control points' change from the reference state, same layout
  float2 C[kNpt];  // each point's coefficients curv, area (f32::Coef)
  float Cg[kNpt];  // and gauss
  float2 geo[kNpt];  // and kA, kV (restraints)
  float cV;          // and dE_r/dV
  double red[kWarps][6];
};
constexpr size_t kSumBytes = sizeof(float) * 12 * kThreads;  // per-thread Kahan totals (dynamic shared memory)
// Thread-private float4 in shared memory, stored and loaded through volatile
// asm so the compiler re-reads it instead of keeping the stored registers
// alive across the point loop (which is the register pressure this layout
// exists to avoid).
__device__ __forceinline__ void st4(float4 *p, float4 v) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"((uint32_t)__cvta_generic_to_shared(p)), "f"(v.x),
               "f"(v.y), "f"(v.z), "f"(v.w));
}
__device__ __forceinline__ float4 ld4(const float4 *p) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"((uint32_t)__cvta_generic_to_shared(p)));
  return v;
}
// Point of the face loop at which the thread prefetches its next face's table
// rows (control points, g0, composition, slot destinations) into L1. Those
// rows are otherwise first touched when the next face starts (control points,
// composition) or point by point (g0), each a round trip to L2.
constexpr int kPrefetchPoint = 10;
}  // namespace tpf

// The restraints' coefficients of the points (which come from the sums kernel).
__device__ __forceinline__ void tpf_stage_geo(tpf::Smem &sm, const float *__restrict__ table,
                                              const double *__restrict__ gterm, double dudv) {
  using L = F32Table<tpf::kNcp, tpf::kNpt>;
  if ((int)threadIdx.x < tpf::kNpt)
    sm.geo[threadIdx.x] = f32::geo_coef(gterm, __ldg(reinterpret_cast<const double *>(table + L::kWeights) + threadIdx.x), dudv);
  if (threadIdx.x == 0) sm.cV = (float)gterm[kGeoCV];
}
// The points' coefficients for a mesh's moduli, by the block's first threads.
__device__ __forceinline__ void tpf_coefs(tpf::Smem &sm, const float *__restrict__ table, const SurfaceParams &P,
                                          double dudv) {
  if ((int)threadIdx.x >= tpf::kNpt) return;
  const double w = __ldg(reinterpret_cast<const double *>(table + F32Table<tpf::kNcp, tpf::kNpt>::kWeights) + threadIdx.x);
  const f32::Coef c = f32::point_coef(P, w, dudv);
  sm.C[threadIdx.x] = make_float2(c.curv, c.area);
  sm.Cg[threadIdx.x] = c.gauss;
}

// Face f's energy terms and dE/dalpha; writes its alpha-scaled gradient
// partials to the face's slots. vec: cp and dest are 16-byte aligned.
// am1 = alpha - 1 (formed in FP64): the box scales' part of the change from
// the reference state. fn: the face this thread takes next (its rows are
// prefetched), or -1.
template <bool KG_REG, bool GEO>
__device__ __forceinline__ void tpf_face(tpf::Smem &sm, const TpfRows &rows, const FaceSrc &S, const SurfaceParams &P, int f,
                                         const float alpha[3], const float ialpha[3], const float am1[3],
                                         float k_reg, bool vec, bool want_da, float *__restrict__ partial,
                                         float e3[3], float da[3], int fn) {
  using namespace tpf;
  uint32_t cp[kNcp];
  if (vec) {
    const uint4 *q = reinterpret_cast<const uint4 *>(S.cp + (size_t)f * kNcp);
#pragma unroll
    for (int i = 0; i < kNc4; ++i) {
      const uint4 v = __ldg(q + i);
      cp[4 * i] = v.x; cp[4 * i + 1] = v.y; cp[4 * i + 2] = v.z; cp[4 * i + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < kNcp; ++j) cp[j] = __ldg(&S.cp[(size_t)f * kNcp + j]);
  }
  const float P2 = __ldg(&S.compf[3 * (size_t)f]), Hbar = __ldg(&S.compf[3 * (size_t)f + 1]),
              Pres = __ldg(&S.compf[3 * (size_t)f + 2]);
  // ---- control points relative to the patch corner (control point 0), in
  // their lattice images, times alpha; error-free sums on the hi/lo pairs as
  // in f32::local_position, so the local coordinates carry full FP32 precision. Their
  // change from the reference state: alpha L - L0 = (alpha - 1) L + (dsp -
  // dsp of the corner). Formed and stored four control points at a time.
  float4 *xs = sm.X[threadIdx.x], *ds = sm.D[threadIdx.x];
  float ahi[3], alo[3], ad[3];
  f32::load_vertex(S.rhi, (int)(cp[0] & kVertexMask), ahi, alo, ad);
#pragma unroll
  for (int c4 = 0; c4 < kNc4; ++c4) {
    float X[4][3], Dx[4][3];
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) {
      const int j = 4 * c4 + jj;
      const int v = (int)(cp[j] & kVertexMask), code = (int)(cp[j] >> kVertexBits);
      float hi[3], lo[3], dv[3], l[3];
      f32::load_vertex(S.rhi, v, hi, lo, dv);
      f32::local_position(hi, lo, code, ahi, alo, P, l);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        X[jj][c] = f32::mul(alpha[c], l[c]);
        Dx[jj][c] = fmaf(am1[c], l[c], f32::sub(dv[c], ad[c]));
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      st4(&xs[kNc4 * c + c4], make_float4(X[0][c], X[1][c], X[2][c], X[3][c]));
      st4(&ds[kNc4 * c + c4], make_float4(Dx[0][c], Dx[1][c], Dx[2][c], Dx[3][c]));
    }
  }
  // ---- the quadrature points
  float G[kNcp][3];  // gradient sums
#pragma unroll
  for (int j = 0; j < kNcp; ++j) G[j][0] = G[j][1] = G[j][2] = 0.f;
  float ea = 0.f, ec = 0.f, er = 0.f;
  Vec3<float> da3 = {0.f, 0.f, 0.f};
#pragma unroll 1
  for (int p = 0; p < kNpt; ++p) {
    if (p == kPrefetchPoint && fn >= 0) {
      prefetch_l1(S.cp + (size_t)fn * kNcp);
      prefetch_l1(S.cp + (size_t)fn * kNcp + kNcp - 1);
      prefetch_l1(S.g0f + (size_t)fn * kNpt);
      prefetch_l1(S.g0f + (size_t)fn * kNpt + kNpt - 1);
      prefetch_l1(S.compf + (size_t)fn * 3);
      prefetch_l1(S.dest + (size_t)fn * kNcp);
      prefetch_l1(S.dest + (size_t)fn * kNcp + kNcp - 1);
    }
    const float g0 = __ldg(&S.g0f[(size_t)f * kNpt + p]);
    float rr0 = 0.f;
    if constexpr (KG_REG) rr0 = __ldg(&S.rr0f[(size_t)f * kNpt + p]);
    // K[k]_c as two partial sums (even, odd control points) in one pair; the
    // u and v rows also over the displacements (dR, the tangents' change
    // from the reference state)
    float2 A[5][3], Ad[2][3], Av[3];
#pragma unroll
    for (int k = 0; k < 5; ++k) A[k][0] = A[k][1] = A[k][2] = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < 2; ++k) Ad[k][0] = Ad[k][1] = Ad[k][2] = make_float2(0.f, 0.f);
    Av[0] = Av[1] = Av[2] = make_float2(0.f, 0.f);
#pragma unroll
    for (int c4 = 0; c4 < kNc4; ++c4) {
      float4 x[3], d[3];  // coordinate c of control points 4 c4 .. 4 c4 + 3
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        x[c] = ld4(&xs[kNc4 * c + c4]);
        d[c] = ld4(&ds[kNc4 * c + c4]);
      }
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const float *b = &rows.B[p][k][4 * c4];
        const float2 b01 = make_float2(b[0], b[1]), b23 = make_float2(b[2], b[3]);
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
        const float *b = &rows.V[p][4 * c4];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          Av[c] = __ffma2_rn(make_float2(b[0], b[1]), make_float2(x[c].x, x[c].y), Av[c]);
          Av[c] = __ffma2_rn(make_float2(b[2], b[3]), make_float2(x[c].z, x[c].w), Av[c]);
        }
      }
    }
    Vec3<float> K[5], dR[2];
#pragma unroll
    for (int k = 0; k < 5; ++k)
      K[k] = {f32::add(A[k][0].x, A[k][0].y), f32::add(A[k][1].x, A[k][1].y), f32::add(A[k][2].x, A[k][2].y)};
#pragma unroll
    for (int k = 0; k < 2; ++k)
      dR[k] = {f32::add(Ad[k][0].x, Ad[k][0].y), f32::add(Ad[k][1].x, Ad[k][1].y), f32::add(Ad[k][2].x, Ad[k][2].y)};
    const float2 cf = sm.C[p];
    const f32::Coef M{cf.x, cf.y, KG_REG ? sm.Cg[p] : 0.f};
    f32::GeoPoint geo{0.f, 0.f, {0.f, 0.f, 0.f}};
    if constexpr (GEO) {
      geo.kA = sm.geo[p].x;
      geo.kV = sm.geo[p].y;
      geo.R = {f32::add(Av[0].x, Av[0].y), f32::add(Av[1].x, Av[1].y), f32::add(Av[2].x, Av[2].y)};
    }
    const f32::Point o = f32::point<KG_REG, GEO>(K, dR, M, k_reg, g0, rr0, P2, Hbar, Pres, geo);
    ea += o.ea;
    ec += o.ec;
    er += o.er;
    if (want_da) {
      da3 = f32::scale_derivative(o, K, da3);
      if constexpr (GEO) da3 = f32::geo_scale_derivative(o, geo, f32::GeoCorner(alpha, ahi, alo, 0.f).x, da3);
    }
    // G[j]_c += B[u][j] Kb[u]_c + B[v][j] Kb[v]_c + s[j] m_c in scalar multiply-adds: with the
    // forward contraction in paired ones, the mix keeps both FP32 multiply-add pipes busy
    // (256-vesicle pass: this mix 550 us, all scalar 591, all paired 727 with spills)
    {
      const float ku[3] = {o.Ku.x, o.Ku.y, o.Ku.z}, kv[3] = {o.Kv.x, o.Kv.y, o.Kv.z}, md[3] = {o.m.x, o.m.y, o.m.z};
#pragma unroll
      for (int c4 = 0; c4 < kNc4; ++c4) {
        const float *u = &rows.B[p][0][4 * c4], *v = &rows.B[p][1][4 * c4], *uu = &rows.B[p][2][4 * c4],
                    *uv = &rows.B[p][3][4 * c4], *vv = &rows.B[p][4][4 * c4];
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          float sj = fmaf(vv[jj], o.nb, fmaf(uv[jj], o.kb, __fmul_rn(uu[jj], o.lb)));
          if constexpr (GEO) sj = fmaf(rows.V[p][4 * c4 + jj], geo.kV, sj);
          float *g = G[4 * c4 + jj];
#pragma unroll
          for (int cc = 0; cc < 3; ++cc) g[cc] = fmaf(sj, md[cc], fmaf(v[jj], kv[cc], fmaf(u[jj], ku[cc], g[cc])));
        }
      }
    }
  }
  // The corner's part of the volume gradient, where that restraint acts; after the
  // points, whose sums would be rounded to its size if they started from it (error of a
  // 40,962-vertex vesicle's gradient 6.0e-7, that way 1.7e-6). Three evaluations in flight
  // 87.4 -> 90.9 us each; in scalar multiply-adds 91.3.
  if (GEO && sm.cV != 0.f) {
    float2 x[3][kNcp / 2];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int c4 = 0; c4 < kNc4; ++c4) {
        const float4 v = ld4(&xs[kNc4 * c + c4]);
        x[c][2 * c4] = make_float2(v.x, v.y);
        x[c][2 * c4 + 1] = make_float2(v.z, v.w);
      }
    const f32::GeoCorner corner(alpha, ahi, alo, sm.cV);
#pragma unroll
    for (int j = 0; j < kNcp; ++j) {
      float2 t2[3];  // even and odd control points
      t2[0] = t2[1] = t2[2] = make_float2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < kNcp / 2; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c)
          t2[c] = __ffma2_rn(make_float2(rows.M[j][2 * i], rows.M[j][2 * i + 1]), x[c][i], t2[c]);
      const float t[3] = {f32::add(t2[0].x, t2[0].y), f32::add(t2[1].x, t2[1].y), f32::add(t2[2].x, t2[2].y)};
      float d[3];
      corner.gradient(t, d);
#pragma unroll
      for (int c = 0; c < 3; ++c) G[j][c] = f32::add(G[j][c], d[c]);
      if (want_da) {
        auto X = [&](int c) { return j & 1 ? x[c][j / 2].y : x[c][j / 2].x; };
        da3 = {fmaf(d[0], X(0), da3.x), fmaf(d[1], X(1), da3.y), fmaf(d[2], X(2), da3.z)};
      }
    }
  }
  // ---- dE/dalpha_c: K is linear in the alpha-scaled coordinates, so
  // alpha_c dE/dalpha_c = sum over points and k of Kb[k]_c K[k]_c
  da[0] = da3.x * ialpha[0]; da[1] = da3.y * ialpha[1]; da[2] = da3.z * ialpha[2];
  int d[kNcp];
  if (vec) {
    const int4 *q = reinterpret_cast<const int4 *>(S.dest + (size_t)f * kNcp);
#pragma unroll
    for (int i = 0; i < kNc4; ++i) {
      const int4 v = __ldg(q + i);
      d[4 * i] = v.x; d[4 * i + 1] = v.y; d[4 * i + 2] = v.z; d[4 * i + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < kNcp; ++j) d[j] = __ldg(&S.dest[(size_t)f * kNcp + j]);
  }
#pragma unroll
  for (int j = 0; j < kNcp; ++j)
    reinterpret_cast<float4 *>(partial)[d[j]] =
        make_float4(f32::mul(alpha[0], G[j][0]), f32::mul(alpha[1], G[j][1]), f32::mul(alpha[2], G[j][2]), 0.f);
  e3[0] = ea; e3[1] = ec; e3[2] = er;
}

__device__ __forceinline__ bool tpf_vec(const FaceSrc &S) {
  return ((reinterpret_cast<uintptr_t>(S.cp) | reinterpret_cast<uintptr_t>(S.dest)) & 15) == 0;
}

// Kahan-compensated FP32 totals of one thread, kept in shared memory (its
// column of s[12][kThreads]) rather than in registers, which the face loop
// needs for itself.
struct SharedSums {
  float *s;
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int q = 0; q < 12; ++q) s[q * tpf::kThreads] = 0.f;
  }
  __device__ __forceinline__ void add(int q, float v) {
    float sum = s[2 * q * tpf::kThreads], c = s[(2 * q + 1) * tpf::kThreads];
    const float y = v - c, t = sum + y;
    s[(2 * q + 1) * tpf::kThreads] = (t - sum) - y;
    s[2 * q * tpf::kThreads] = t;
  }
  __device__ __forceinline__ double total(int q) const {  // over the warp
    return warp_sum(s[2 * q * tpf::kThreads], s[(2 * q + 1) * tpf::kThreads]);
  }
};

// Single mesh, regular faces, precision form: persistent grid, warp w of the
// grid takes faces 32 w .. 32 w + 31, then 32 (w + warps in the grid) ...
// Writes one block partial of the energy terms and dE/dalpha; the last block
// of the pass to finish sums them.
template <bool GEO>  // the restraints' gradient goes along
__global__ void __launch_bounds__(tpf::kThreads, tpf::kMinBlocks)
    face_tpf_kernel(const __grid_constant__ TpfRows rows, FaceLaunch L, const int *__restrict__ dest, SurfaceParams P, const double *__restrict__ r,
                    const float *__restrict__ rhi, const float *__restrict__ rlo, const float *__restrict__ dsp,
                    float *__restrict__ partial, double *__restrict__ blockpart, int *__restrict__ status,
                    FinishArgs fin) {
  using namespace tpf;
  __shared__ Smem sm;
  extern __shared__ __align__(16) unsigned char tpf_dyn[];
  tpf_coefs(sm, L.table, P, L.dudv);
  __syncthreads();
  grid_dependency_wait();  // the state comes from the kernels before
  if constexpr (GEO) {
    tpf_stage_geo(sm, L.table, fin.gterm, L.dudv);
    __syncthreads();
  }
  const bool want_da = fin.galpha != nullptr;  // a run's steps leave the box scales alone
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float alpha[3] = {(float)r[3 * P.nv], (float)r[3 * P.nv + 1], (float)r[3 * P.nv + 2]};
  const float ialpha[3] = {1.f / alpha[0], 1.f / alpha[1], 1.f / alpha[2]};
  const float am1[3] = {(float)(r[3 * P.nv] - 1.0), (float)(r[3 * P.nv + 1] - 1.0), (float)(r[3 * P.nv + 2] - 1.0)};
  const FaceSrc src{L.cp, nullptr, nullptr, nullptr, L.g0f, L.rr0f, L.compf, dest, r, rhi, rlo, dsp, L.nfaces};
  const bool vec = tpf_vec(src);
  const bool kg_reg = P.kg != 0.0 || P.k_reg != 0.0;  // else the pointwise step leaves those terms out
  const float k_reg = (float)P.k_reg;
  const int n = L.nfaces, stride = gridDim.x * kThreads;
  SharedSums acc{reinterpret_cast<float *>(tpf_dyn) + threadIdx.x};
  acc.zero();
  for (int fb = (blockIdx.x * kWarps + warp) * 32; fb < n; fb += stride) {
    const int f = fb + lane;
    if (f < n) {
      float e3[3], da[3];
      // no prefetch: a thread's next face is a grid stride away, and on the
      // 512 x 512 planar pass the prefetch cost 1% instead of gaining
      if (kg_reg) tpf_face<true, GEO>(sm, rows, src, P, f, alpha, ialpha, am1, k_reg, vec, want_da, partial, e3, da, -1);
      else tpf_face<false, GEO>(sm, rows, src, P, f, alpha, ialpha, am1, k_reg, vec, want_da, partial, e3, da, -1);
      acc.add(0, e3[0]); acc.add(1, e3[1]); acc.add(2, e3[2]);
      acc.add(3, da[0]); acc.add(4, da[1]); acc.add(5, da[2]);
      if (!isfinite(e3[0] + e3[1] + e3[2])) atomicOr(status, kStatusNonFinite);
    }
  }
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    const double s = acc.total(q);
    if (lane == 0) sm.red[warp][q] = s;
  }
  __syncthreads();  // every thread has read its sums: the finish may reuse their space
  if (threadIdx.x < 6) {
    double s = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) s += sm.red[w][threadIdx.x];
    blockpart[6 * (size_t)(L.block_base + blockIdx.x) + threadIdx.x] = threadIdx.x < 3 ? s * P.e_scale[0][threadIdx.x] : s;
  }
  count_and_finish<kThreads>(fin, blockpart);
}

// Batched regular faces, precision form: a block takes a tile (faces of one
// job), its warps 32 faces at a time; writes the tile's three energy sums.
// counter[0] hands out the tiles; counter[1] counts the blocks that are done,
// and the last of them zeroes both for the next launch. A block draws its next
// tile while it works on the current one (the draw's round trip hides behind
// the faces), and copies a job's header only when the tile's job changes.
__global__ void __launch_bounds__(tpf::kThreads, tpf::kBatchMinBlocks)
    batch_face_tpf_kernel(const __grid_constant__ TpfRows rows, const BatchJob *__restrict__ jobs, int group, const BatchTile *__restrict__ tiles,
                          const int *__restrict__ counts, const float *__restrict__ table, double dudv,
                          double *__restrict__ tile_sums, int *__restrict__ counter) {
  using namespace tpf;
  __shared__ Smem sm;
  __shared__ BatchFaceJob sj;
  __shared__ int s_active, s_tile[2];
  grid_dependency_wait();        // positions, job states and the counter come from the kernels before
  const int ntiles = counts[group], tile_base = counts[3 + group];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Tiles are handed out by a counter (zeroed before the launch), so blocks
  // that draw cheap tiles take more; each tile's sums go to its own row, so
  // the results do not depend on which block took which tile. Draw k is read
  // from s_tile[k & 1] after the barrier that opens iteration k and written
  // during iteration k - 1, after that iteration's own barrier: its readers
  // of the same slot (iteration k - 2) are done by then.
  if (threadIdx.x == 0) s_tile[0] = (int)blockIdx.x < ntiles ? atomicAdd(&counter[0], 1) : ntiles;
  int job = -1;
  for (int k = 0;; ++k) {
    __syncthreads();  // the previous tile's readers of sj, s_active and sm.red are done; draw k is visible
    const int t = s_tile[k & 1];
    if (t >= ntiles) break;
    const BatchTile tile = tiles[tile_base + t];
    if (tile.job != job) {  // the same for every thread of the block
      const int *src = reinterpret_cast<const int *>(&jobs[tile.job].f);
      int *dst = reinterpret_cast<int *>(&sj);
      for (int i = threadIdx.x; i < (int)(sizeof(BatchFaceJob) / sizeof(int)); i += kThreads) dst[i] = src[i];
      if (threadIdx.x == 0) s_active = job_active(jobs[tile.job].f);
      tpf_coefs(sm, table, jobs[tile.job].f.P, dudv);
      job = tile.job;
      __syncthreads();
    }
    if (threadIdx.x == 0) s_tile[(k + 1) & 1] = atomicAdd(&counter[0], 1);
    KahanSums<3> acc;
    if (s_active) {
      const FaceSrc &src = sj.src[group];
      const SurfaceParams &P = sj.P;
      const double *r = src.r;
      const float alpha[3] = {(float)r[3 * P.nv], (float)r[3 * P.nv + 1], (float)r[3 * P.nv + 2]};
      const float ialpha[3] = {1.f / alpha[0], 1.f / alpha[1], 1.f / alpha[2]};
      const float am1[3] = {(float)(r[3 * P.nv] - 1.0), (float)(r[3 * P.nv + 1] - 1.0),
                            (float)(r[3 * P.nv + 2] - 1.0)};
      const int end = tile.first + tile.count;
      float *partial = (float *)sj.partial;
      const bool kg_reg = P.kg != 0.0 || P.k_reg != 0.0;  // else the pointwise step leaves those terms out
      const float k_reg = (float)P.k_reg;
      const bool vec = tpf_vec(src);
      for (int fb = tile.first + warp * 32; fb < end; fb += kThreads) {
        const int f = fb + lane;
        if (f < end) {
          float e3[3], da[3];
          const int fn = f + kThreads < end ? f + kThreads : -1;
          if (kg_reg) tpf_face<true, false>(sm, rows, src, P, f, alpha, ialpha, am1, k_reg, vec, false, partial, e3, da, fn);
          else tpf_face<false, false>(sm, rows, src, P, f, alpha, ialpha, am1, k_reg, vec, false, partial, e3, da, fn);
          acc.add(0, e3[0]); acc.add(1, e3[1]); acc.add(2, e3[2]);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const double s = warp_sum(acc.s[q], acc.c[q]);
      if (lane == 0) sm.red[warp][q] = s;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
      double s = 0;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) s += sm.red[w][threadIdx.x];
      tile_sums[3 * (size_t)(tile_base + t) + threadIdx.x] = s * sj.P.e_scale[0][threadIdx.x];
    }
  }
  __threadfence();  // this block's last draw on counter[0] is ordered before its count on counter[1]
  if (threadIdx.x == 0 && atomicAdd(&counter[1], 1) == (int)gridDim.x - 1) {
    counter[0] = 0;  // every block has drawn its last tile: reset for the next launch
    counter[1] = 0;
  }
}

// Per job (one warp each): sum its tiles in listed order, record the step's
// energy in the job's run, flag non-finite or diverging energies (src/hd.C:
// 1280-1305) for that job only, advance its run index. live[j] tells the
// update whether job j took this step; prog[j] = {steps done, status}.
__global__ void batch_reduce_kernel(const BatchJob *__restrict__ jobs, const int *__restrict__ counts,
                                    const int *__restrict__ tile_off, const int *__restrict__ tile_idx,
                                    const double *__restrict__ tile_sums, int *__restrict__ live,
                                    unsigned long long *__restrict__ prog) {
  grid_dependency_wait();
  grid_dependents(kFewGatherBlocks);
  const int lane = threadIdx.x & 31;
  const int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (j >= counts[6]) return;
  const BatchJob &J = jobs[j];
  const bool active = job_active(J.f);  // uniform over the warp: nothing below changes it before the sync
  __syncwarp();
  double a[3] = {0, 0, 0};
  if (active)
    for (int k = tile_off[j] + lane; k < tile_off[j + 1]; k += 32)
#pragma unroll
      for (int q = 0; q < 3; ++q) a[q] += tile_sums[3 * (size_t)tile_idx[k] + q];
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1)
#pragma unroll
    for (int q = 0; q < 3; ++q) a[q] += __shfl_xor_sync(0xffffffffu, a[q], off);
  if (lane != 0) return;
  int st = *J.f.status;
  uint64_t done = J.f.cnt[1];
  if (active) {
    const double e = a[0] + a[1] + a[2];
    J.E[0] = e;
    J.parts[0] = a[0]; J.parts[1] = a[1]; J.parts[2] = a[2];
    if (!isfinite(e)) st |= kStatusNonFinite;
    if (J.energies) {
      J.energies[done] = e;
      if (J.threshold > 0 && done > 0 && e - J.energies[done - 1] > J.threshold) st |= kStatusDiverged;
    }
    *J.f.status = st;
    // As in a single-mesh run, the step whose energy is flagged does not move.
    J.f.cnt[1] = ++done;
  }
  live[j] = active && !st;
  prog[2 * j] = done;
  prog[2 * j + 1] = (unsigned long long)st;
}

// Gather fused with each live job's vertex-local update (overdamped BD, or the
// leapfrog kinds with identity mass), with the job's own integrator settings.
template <typename T>
__global__ void batch_gather_step_kernel(const BatchJob *__restrict__ jobs, const BatchTile *__restrict__ vtiles,
                                         const int *__restrict__ counts, const int *__restrict__ live) {
  grid_dependency_wait();
  const int nvtiles = counts[7];
  for (int t = blockIdx.x; t < nvtiles; t += gridDim.x) {
    const BatchTile tile = vtiles[t];
    if (!live[tile.job] || (int)threadIdx.x >= tile.count) continue;
    const BatchJob &J = jobs[tile.job];
    const StepArgs &a = J.a;
    const int v = tile.first + threadIdx.x;
    const uint64_t st = J.f.cnt[0] + J.f.cnt[1] - 1;
    if constexpr (sizeof(T) == 4) {
      if (a.kind == 0) {
        bd_vertex_f32((const float *)J.f.partial, J.off, v, a, st, J.r, J.rhi, J.r0);
        continue;
      }
    }
    double gg[3], n[3];
    vertex_gradient((const T *)J.f.partial, J.off, v, gg);
    if constexpr (sizeof(T) == 8) {
      normals3(a.seed, a.stream, st, v, n);
    } else {
      float nf[3];
      normals3_f32(a.seed, a.stream, st, v, nf);
      for (int c = 0; c < 3; ++c) n[c] = convert::to_f64(nf[c]);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const size_t i = 3 * (size_t)v + c;
      double q = a.kind != 0 ? J.p[i] : 0.0;
      const double x = coordinate_update(a, gg[c], n[c], J.r[i], &q);
      if (a.kind != 0) J.p[i] = q;
      J.r[i] = x;
      if (J.rhi) store_f32_position(i, x, J.rhi, J.rlo, J.r0, J.dsp);
    }
  }
}

// Start of the runs of the jobs flagged in start[]: counters {step0, 0},
// status cleared, FP32 hi/lo pairs of the positions (precision form).
__global__ void batch_start_kernel(const BatchJob *__restrict__ jobs, const BatchTile *__restrict__ vtiles,
                                   const int *__restrict__ counts, const int *__restrict__ start,
                                   const unsigned long long *__restrict__ step0) {
  const int nvtiles = counts[7];
  for (int t = blockIdx.x; t < nvtiles; t += gridDim.x) {
    const BatchTile tile = vtiles[t];
    if (!start[tile.job]) continue;
    const BatchJob &J = jobs[tile.job];
    if (tile.first == 0 && threadIdx.x == 0) {
      J.f.cnt[0] = step0[tile.job];
      J.f.cnt[1] = 0;
      *J.f.status = 0;
    }
    if (J.rhi && (int)threadIdx.x < tile.count) {
      const int v = tile.first + threadIdx.x;
      store_f32_vertex(v, J.r + 3 * (size_t)v, J.rhi, J.r0);
    }
  }
}

// Host-driven batch steps: every job's state (3 nv + 3 doubles: positions,
// then the box scales) packed in job order at pack[off[j] ..]. In: into each
// job's resident state and the precision form's FP32 copies. Out: back into
// the pack, and each job's latest energy into E[j].
__global__ void batch_unpack_kernel(const BatchJob *__restrict__ jobs, const BatchTile *__restrict__ vtiles,
                                    const int *__restrict__ counts, const long long *__restrict__ off,
                                    const double *__restrict__ pack) {
  const int nvtiles = counts[7];
  for (int t = blockIdx.x; t < nvtiles; t += gridDim.x) {
    const BatchTile tile = vtiles[t];
    const BatchJob &J = jobs[tile.job];
    const double *src = pack + off[tile.job];
    if ((int)threadIdx.x < tile.count) {
      const size_t v = (size_t)(tile.first + threadIdx.x);
      double x[3];
      bool changed = false;
      for (int c = 0; c < 3; ++c) {
        x[c] = src[3 * v + c];
        changed = changed || __double_as_longlong(x[c]) != __double_as_longlong(J.r[3 * v + c]);
      }
      // a vertex the caller left as it was keeps its FP32 copies (compared bit
      // for bit, on the integer pipe): most of the unpacking's FP64 work
      if (changed) {
        for (int c = 0; c < 3; ++c) J.r[3 * v + c] = x[c];
        if (J.rhi) store_f32_vertex((int)v, x, J.rhi, J.r0);
      }
    }
    if (tile.first == 0 && threadIdx.x < 3) {
      const size_t a = 3 * (size_t)J.f.P.nv + threadIdx.x;
      J.r[a] = src[a];
    }
  }
}

__global__ void batch_pack_kernel(const BatchJob *__restrict__ jobs, const BatchTile *__restrict__ vtiles,
                                  const int *__restrict__ counts, const long long *__restrict__ off,
                                  double *__restrict__ pack, double *__restrict__ E) {
  const int nvtiles = counts[7];
  for (int t = blockIdx.x; t < nvtiles; t += gridDim.x) {
    const BatchTile tile = vtiles[t];
    const BatchJob &J = jobs[tile.job];
    double *dst = pack + off[tile.job];
    if ((int)threadIdx.x < tile.count) {
      const size_t v = (size_t)(tile.first + threadIdx.x);
      for (int c = 0; c < 3; ++c) dst[3 * v + c] = J.r[3 * v + c];
    }
    if (tile.first == 0 && threadIdx.x < 3) {
      const size_t a = 3 * (size_t)J.f.P.nv + threadIdx.x;
      dst[a] = J.r[a];
    }
    if (tile.first == 0 && threadIdx.x == 3) E[tile.job] = *J.E;
  }
}

// ---------------------------------------------------------------- area, volume
//
// One half-warp per face, as in the face pass: lanes are control points while
// the face's local coordinates are formed, then quadrature points. The value
// and first-derivative basis rows of every patch type sit in shared memory.
//
// Precision. The restraint on V is stiff (K_V (V - V0) is a force per unit
// volume), so V must be exact far below an FP32 ulp of V: on a 1000 A vesicle
// a 1e-3 A^3 error already moves every vertex's restraint force by about
// K_V 1e-3 A^3 x 300 A^2. The sums therefore form R, R_u, R_v and R.(R_u x R_v)
// beyond FP32 from local coordinates (relative to the patch corner, which is
// added back exactly): in FP64 here, in integers and pairs of FP32 in the
// precision form (geo32.cu), whose area, with its soft restraint, and box-scale
// derivatives come from the FP32 leading parts. The gradient needs only the
// relative accuracy of any other gradient term and runs in the form's own
// arithmetic (FP32 local coordinates from the hi/lo pairs, as the face pass forms
// them).

constexpr int kGeoHW = kGeoThreads / 16;  // faces in flight per block

template <typename T>
struct GeoBasis {
  T B[3][kGeoPt][3][kMaxCpDev];  // [group][point][w, u, v][control point]
  T cw[3][kGeoPt];               // dudv * weight
};

template <typename T>
__device__ void stage_geo_basis(const GeoArgs &G, GeoBasis<T> &s) {
  for (int gi = 0; gi < G.ngroups; ++gi) {
    const GeoGroup &g = G.g[gi];
    for (int i = threadIdx.x; i < g.npt * g.ncp; i += blockDim.x) {
      const int p = i / g.ncp, x = i % g.ncp;
      s.B[gi][p][0][x] = (T)g.basis_w[(size_t)p * g.ncp + x];
      s.B[gi][p][1][x] = (T)g.basis[(size_t)p * 5 * g.ncpp + x];
      s.B[gi][p][2][x] = (T)g.basis[(size_t)p * 5 * g.ncpp + g.ncpp + x];
    }
    for (int p = threadIdx.x; p < g.npt; p += blockDim.x) s.cw[gi][p] = (T)(g.dudv * g.weight[p]);
  }
}

// Group of global face f (faces are numbered group after group).
__device__ __forceinline__ int geo_group(const GeoArgs &G, int f, int *local) {
  int k = 0;
  while (k + 1 < G.ngroups && f >= G.g[k + 1].face_base) ++k;
  *local = f - G.g[k].face_base;
  return k;
}

// Absolute (alpha-scaled, lattice-image) FP64 position of control point `lane` of face lf.
__device__ __forceinline__ void geo_abs64(const GeoArgs &G, const GeoGroup &g, int lf, int lane,
                                          const double alpha[3], double X[3], int *dest) {
  const uint32_t packed = __ldg(&g.cp[(size_t)lf * g.ncp + lane]);
  const int v = (int)(packed & kVertexMask), code = (int)(packed >> kVertexBits);
  const int im[3] = {code % 3 - 1, (code / 3) % 3 - 1, code / 9 - 1};
#pragma unroll
  for (int c = 0; c < 3; ++c)
    X[c] = alpha[c] * (G.r[3 * (size_t)v + c] + im[0] * G.box[0][c] + im[1] * G.box[1][c] + im[2] * G.box[2][c]);
  if (dest) *dest = __ldg(&g.dest[(size_t)lf * g.ncp + lane]);
}

__device__ __forceinline__ double shfl_d(unsigned mask, double v, int src) { return __shfl_sync(mask, v, src, 16); }

// Sums A, V and their alpha derivatives in FP64 (the plain path).
__global__ void __launch_bounds__(kGeoThreads) geo_sums_kernel(GeoArgs G) {
  __shared__ GeoBasis<double> sb;
  __shared__ double Xs[kGeoHW][kMaxCpDev][3];
  __shared__ double red[kGeoWords][kGeoThreads];
  stage_geo_basis<double>(G, sb);
  __syncthreads();
  grid_dependency_wait();  // the state comes from the kernels before
  const int hw = threadIdx.x >> 4, lane = threadIdx.x & 15;
  const unsigned hmask = (threadIdx.x & 16) ? 0xFFFF0000u : 0x0000FFFFu;
  const double alpha[3] = {G.r[3 * (size_t)G.nv], G.r[3 * (size_t)G.nv + 1], G.r[3 * (size_t)G.nv + 2]};
  const double ialpha[3] = {1.0 / alpha[0], 1.0 / alpha[1], 1.0 / alpha[2]};
  double acc[kGeoWords] = {0, 0, 0, 0, 0, 0, 0, 0};  // A, V, dA/dalpha (3), dV/dalpha (3)
  for (int f = blockIdx.x * kGeoHW + hw; f < G.nfaces; f += gridDim.x * kGeoHW) {
    int lf;
    const int gi = geo_group(G, f, &lf);
    const GeoGroup &g = G.g[gi];
    double X[3] = {0, 0, 0};
    if (lane < g.ncp) geo_abs64(G, g, lf, lane, alpha, X, nullptr);
    double X0[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) X0[c] = shfl_d(hmask, X[c], 0);
    if (lane < g.ncp)
#pragma unroll
      for (int c = 0; c < 3; ++c) Xs[hw][lane][c] = X[c] - X0[c];
    __syncwarp(hmask);
    if (lane < g.npt) {
      double R[3] = {0, 0, 0}, Ru[3] = {0, 0, 0}, Rv[3] = {0, 0, 0};
      const double *bw = sb.B[gi][lane][0], *bu = sb.B[gi][lane][1], *bv = sb.B[gi][lane][2];
#pragma unroll
      for (int x = 0; x < kMaxCpDev; ++x) {
        if (x < g.ncp) {
          const double w = bw[x], u = bu[x], v = bv[x];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const double xx = Xs[hw][x][c];
            R[c] = fma(w, xx, R[c]);
            Ru[c] = fma(u, xx, Ru[c]);
            Rv[c] = fma(v, xx, Rv[c]);
          }
        }
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) R[c] += X0[c];  // back to absolute: the corner is exact in FP64
      double m[3];
      cross3(Ru, Rv, m);
      const double cw = sb.cw[gi][lane], c3 = cw * (1.0 / 3.0);
      acc[1] += c3 * (R[0] * m[0] + R[1] * m[1] + R[2] * m[2]);
      const double gg = sqrt(m[0] * m[0] + m[1] * m[1] + m[2] * m[2]), ig = 1.0 / gg;
      acc[0] += cw * gg;
      double n[3] = {m[0] * ig, m[1] * ig, m[2] * ig}, a1[3], a2[3], v1[3], v2[3];
      cross3(Rv, n, a1);  // dg/dRu
      cross3(n, Ru, a2);  // dg/dRv
      cross3(Rv, R, v1);  // d(R.m)/dRu
      cross3(R, Ru, v2);  // d(R.m)/dRv
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        acc[2 + k] += cw * (a1[k] * Ru[k] + a2[k] * Rv[k]) * ialpha[k];
        acc[5 + k] += c3 * (m[k] * R[k] + v1[k] * Ru[k] + v2[k] * Rv[k]) * ialpha[k];
      }
    }
    __syncwarp(hmask);
  }
  geo_finish(G, acc, red);
}

// (The gradient goes along in the face kernels, which have the tangents and the
// normal at hand: 10% more of their work instead of a pass of its own over every
// face, 40 to 50 us at 81,920 faces, with a read and write of every partial.
// Three restrained evaluations of a 40,962-vertex vesicle in flight: 179 -> 135
// us each. The pass below remains for the plain path and for meshes whose
// regular faces run on the tensor cores.)

// partial[slot] += alpha * dE_r/dX for every (face, control point):
//   dE_r/dR  = c_V c/3 m,   dE_r/dRu = c_A c (Rv x n) + c_V c/3 (Rv x R),
//   dE_r/dRv = c_A c (n x Ru) + c_V c/3 (R x Ru),
// contracted with the w, u, v rows (lanes = points, then lanes = control points).
template <typename T>
__global__ void __launch_bounds__(kGeoThreads) geo_grad_kernel(GeoArgs G, T *__restrict__ partial) {
  grid_dependency_wait();  // the coefficients come from the sums kernel, the partials from the face launches
  const double cA64 = G.gterm[kGeoCA], cV64 = G.gterm[kGeoCV];
  if (cA64 == 0.0 && cV64 == 0.0) return;
  __shared__ GeoBasis<T> sb;
  __shared__ T Xs[kGeoHW][kMaxCpDev][3];
  __shared__ T Es[kGeoHW][kGeoPt][9];
  if constexpr (sizeof(T) == 4) {
    for (int gi = 0; gi < G.ngroups; ++gi) {
      const GeoGroup &g = G.g[gi];
      auto stage = [&](const auto &t) {
        for (int i = threadIdx.x; i < g.npt * 3 * g.ncp; i += blockDim.x) {
          const int p = i / (3 * g.ncp), k = (i / g.ncp) % 3, x = i % g.ncp;
          sb.B[gi][p][k][x] = t.bf[p][k][x];
        }
        for (int p = threadIdx.x; p < g.npt; p += blockDim.x) sb.cw[gi][p] = t.cw[p];
      };
      if (g.ncp <= 12) stage(*static_cast<const GeoRows<12> *>(g.tab));
      else stage(*static_cast<const GeoRows<16> *>(g.tab));
    }
  } else {
    stage_geo_basis<T>(G, sb);
  }
  __syncthreads();
  const int hw = threadIdx.x >> 4, lane = threadIdx.x & 15;
  const unsigned hmask = (threadIdx.x & 16) ? 0xFFFF0000u : 0x0000FFFFu;
  const double a64[3] = {G.r[3 * (size_t)G.nv], G.r[3 * (size_t)G.nv + 1], G.r[3 * (size_t)G.nv + 2]};
  const T alpha[3] = {(T)a64[0], (T)a64[1], (T)a64[2]};
  const T cA = (T)cA64, cV = (T)cV64;
  for (int f = blockIdx.x * kGeoHW + hw; f < G.nfaces; f += gridDim.x * kGeoHW) {
    int lf;
    const int gi = geo_group(G, f, &lf);
    const GeoGroup &g = G.g[gi];
    {  // the next face's control-point and slot rows into L1 while this face runs
      const int fn = f + gridDim.x * kGeoHW;
      if (lane < 2 && fn < G.nfaces) {
        int lfn;
        const GeoGroup &h = G.g[geo_group(G, fn, &lfn)];
        const size_t at = (size_t)lfn * h.ncp + (lane ? h.ncp - 1 : 0);
        prefetch_l1(h.cp + at);
        prefetch_l1(h.dest + at);
      }
    }
    int dest = 0;
    T X0[3];
    if constexpr (sizeof(T) == 8) {
      double X[3] = {0, 0, 0};
      if (lane < g.ncp) geo_abs64(G, g, lf, lane, a64, X, &dest);
#pragma unroll
      for (int c = 0; c < 3; ++c) X0[c] = shfl_d(hmask, X[c], 0);
      if (lane < g.ncp)
#pragma unroll
        for (int c = 0; c < 3; ++c) Xs[hw][lane][c] = X[c] - X0[c];
    } else {
      // FP32 coordinates relative to the corner from the hi/lo pairs with
      // error-free sums, as the face pass forms them.
      float hi[3] = {0, 0, 0}, lo[3] = {0, 0, 0};
      int img[3] = {0, 0, 0};
      if (lane < g.ncp) {
        const uint32_t packed = __ldg(&g.cp[(size_t)lf * g.ncp + lane]);
        const int v = (int)(packed & kVertexMask), code = (int)(packed >> kVertexBits);
        img[0] = code % 3 - 1; img[1] = (code / 3) % 3 - 1; img[2] = code / 9 - 1;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          hi[c] = G.rhi[kPosStride * (size_t)v + c];
          lo[c] = G.rlo[kPosStride * (size_t)v + c];
        }
        dest = __ldg(&g.dest[(size_t)lf * g.ncp + lane]);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float ahi = __shfl_sync(hmask, hi[c], 0, 16), alo = __shfl_sync(hmask, lo[c], 0, 16);
        float sh = 0.f, she = 0.f, shl = 0.f;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          float t, e;
          two_sum(sh, (float)img[d] * G.box_hi[d][c], t, e);
          sh = t;
          she += e;
          shl += (float)img[d] * G.box_lo[d][c];
        }
        float s1, e1, s2, e2;
        two_sum(hi[c], sh, s1, e1);
        two_sum(s1, -ahi, s2, e2);
        if (lane < g.ncp) Xs[hw][lane][c] = alpha[c] * (s2 + ((e1 + e2) + ((lo[c] - alo) + (she + shl))));
        X0[c] = alpha[c] * (ahi + alo);  // the corner carries no image (its shift is zero)
      }
    }
    // this face's partial slots, read now so that the read-modify-write at the
    // end does not wait on them (no other thread touches these slots)
    T old[3] = {0, 0, 0};
    if (lane < g.ncp)
#pragma unroll
      for (int k = 0; k < 3; ++k) old[k] = partial[kSlot<T> * (size_t)dest + k];
    __syncwarp(hmask);
    if (lane < g.npt) {
      T R[3] = {0, 0, 0}, Ru[3] = {0, 0, 0}, Rv[3] = {0, 0, 0};
      const T *bw = sb.B[gi][lane][0], *bu = sb.B[gi][lane][1], *bv = sb.B[gi][lane][2];
#pragma unroll
      for (int x = 0; x < kMaxCpDev; ++x) {
        if (x < g.ncp) {
          const T w = bw[x], u = bu[x], v = bv[x];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const T xx = Xs[hw][x][c];
            R[c] += w * xx;
            Ru[c] += u * xx;
            Rv[c] += v * xx;
          }
        }
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) R[c] += X0[c];
      T m[3], n[3], a1[3], a2[3], v1[3], v2[3];
      cross3(Ru, Rv, m);
      const T ig = T(1) / sqrt(m[0] * m[0] + m[1] * m[1] + m[2] * m[2]);
#pragma unroll
      for (int c = 0; c < 3; ++c) n[c] = m[c] * ig;
      cross3(Rv, n, a1);
      cross3(n, Ru, a2);
      cross3(Rv, R, v1);
      cross3(R, Ru, v2);
      const T cw = sb.cw[gi][lane], kA = cA * cw, kV = cV * cw * (T(1) / T(3));
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        Es[hw][lane][k] = kV * m[k];
        Es[hw][lane][3 + k] = kA * a1[k] + kV * v1[k];
        Es[hw][lane][6 + k] = kA * a2[k] + kV * v2[k];
      }
    }
    __syncwarp(hmask);
    if (lane < g.ncp) {
      T Gx[3] = {0, 0, 0};
      for (int p = 0; p < g.npt; ++p) {
        const T w = sb.B[gi][p][0][lane], u = sb.B[gi][p][1][lane], v = sb.B[gi][p][2][lane];
#pragma unroll
        for (int k = 0; k < 3; ++k) Gx[k] += w * Es[hw][p][k] + u * Es[hw][p][3 + k] + v * Es[hw][p][6 + k];
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) partial[kSlot<T> * (size_t)dest + k] = old[k] + alpha[k] * Gx[k];
    }
    __syncwarp(hmask);
  }
}

// One warp per row; lanes stride the row's nonzeros (coalesced reads of the
// value/column streams), warp-shuffle sum in fixed order.
__global__ void spmv_kernel(int nrow, const int *__restrict__ row_ptr, const int *__restrict__ col,
                            const double *__restrict__ val, const double *__restrict__ scalev, MassScale F,
                            const double *__restrict__ in, double *__restrict__ out, int accumulate) {
  grid_dependency_wait();
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const double f[3] = {F.f[0], F.f[1], F.f[2]};
  for (int i = warp; i < nrow; i += nwarps) {
    double s0 = 0, s1 = 0, s2 = 0;
    for (int k = row_ptr[i] + lane; k < row_ptr[i + 1]; k += 32) {
      const double v = val[k];
      const int j = col[k];
      s0 += v * in[3 * (size_t)j];
      s1 += v * in[3 * (size_t)j + 1];
      s2 += v * in[3 * (size_t)j + 2];
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
      s0 += __shfl_xor_sync(0xffffffffu, s0, off);
      s1 += __shfl_xor_sync(0xffffffffu, s1, off);
      s2 += __shfl_xor_sync(0xffffffffu, s2, off);
    }
    if (lane == 0) {
      double o[3] = {s0 * f[0], s1 * f[1], s2 * f[2]};
      if (scalev)
#pragma unroll
        for (int c = 0; c < 3; ++c) o[c] *= scalev[(size_t)c * nrow + i];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (accumulate) out[3 * (size_t)i + c] += o[c];
        else out[3 * (size_t)i + c] = o[c];
      }
    }
  }
}

// spmv_kernel on FP32 values and an FP32 copy of the input packed as one
// float4 per row {x, y, z, 0} (the precision form's inverse mass), so each
// nonzero gathers its input with one 16-byte load. kSpmvUnroll nonzeros per
// lane per round have their loads in flight together. Kahan-compensated FP32 sums
// per lane, the cross-lane sum and the scaling in FP64. Reads 8 bytes per
// nonzero instead of 12 and keeps the FP64 pipe out of the loop.
constexpr int kSpmvUnroll = 4;
// spmv32_kernel streams each row's values and columns, kSpmvUnroll windows of
// 32 nonzeros per warp iteration; a warp also asks L2 for the lines
// kSpmvAhead windows ahead of the ones it loads, so that its loads find them
// there (40,962-vertex M^-1, 415 M nonzeros: 546 -> 475 us per apply when it came in).
constexpr int kSpmvAhead = 32;
__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
// kSpmvBlocks: the blocks a SM that its 40 registers allow, given to the compiler. Left
// to itself it took 34 (as many blocks) and put loads of a round behind one another:
// 488 us a call with that matrix, 461 with all of them in flight.
constexpr int kSpmvThreads = 256, kSpmvBlocks = 6;
template <typename C>  // column index type: int, or uint16_t for up to 65,536 columns
__global__ void __launch_bounds__(kSpmvThreads, kSpmvBlocks)
    spmv32_kernel(int nrow, const int *__restrict__ row_ptr, const C *__restrict__ col, const float *__restrict__ val,
                  const double *__restrict__ scalev, MassScale F, const float4 *__restrict__ in4,
                  double *__restrict__ out, int accumulate) {
  grid_dependency_wait();
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const double f[3] = {F.f[0], F.f[1], F.f[2]};
  for (int i = warp; i < nrow; i += nwarps) {
    KahanSums<3> acc;
    const int beg = row_ptr[i], end = row_ptr[i + 1];
    for (int w = 32 * lane; w < 32 * kSpmvAhead; w += 32 * 32) {  // the row's first windows
      if (w < end - beg) {
        prefetch_l2(&val[beg + w]);
        prefetch_l2(&col[beg + w]);
      }
    }
    for (int k0 = beg + lane; k0 < end; k0 += 32 * kSpmvUnroll) {
      if (lane < 2 * kSpmvUnroll) {  // lanes 0..3: value lines ahead; lanes 4..7: their columns
        const int w = k0 - lane, ahead = 32 * (kSpmvAhead + (lane % kSpmvUnroll));
        if (ahead < end - w)
          prefetch_l2(lane < kSpmvUnroll ? (const void *)&val[w + ahead] : (const void *)&col[w + ahead]);
      }
      float v[kSpmvUnroll];
      int j[kSpmvUnroll];
#pragma unroll
      for (int u = 0; u < kSpmvUnroll; ++u) {
        const int k = k0 + 32 * u;
        v[u] = k < end ? __ldcs(&val[k]) : 0.f;
        j[u] = k < end ? (int)__ldcs(&col[k]) : 0;
      }
      float4 x[kSpmvUnroll];
#pragma unroll
      for (int u = 0; u < kSpmvUnroll; ++u) x[u] = __ldg(&in4[j[u]]);
      // groups of four products summed by plain multiply-adds, each group
      // added to the compensated total
#pragma unroll
      for (int g = 0; g < kSpmvUnroll; g += 4) {
        float t0 = v[g] * x[g].x, t1 = v[g] * x[g].y, t2 = v[g] * x[g].z;
#pragma unroll
        for (int u = g + 1; u < g + 4; ++u) {
          t0 = fmaf(v[u], x[u].x, t0);
          t1 = fmaf(v[u], x[u].y, t1);
          t2 = fmaf(v[u], x[u].z, t2);
        }
        acc.add(0, t0);
        acc.add(1, t1);
        acc.add(2, t2);
      }
    }
    double s[3] = {acc.get(0), acc.get(1), acc.get(2)};
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1)
#pragma unroll
      for (int c = 0; c < 3; ++c) s[c] += __shfl_xor_sync(0xffffffffu, s[c], off);
    if (lane == 0) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        double o = s[c] * f[c];
        if (scalev) o *= scalev[(size_t)c * nrow + i];
        if (accumulate) out[3 * (size_t)i + c] += o;
        else out[3 * (size_t)i + c] = o;
      }
    }
  }
}

// Rows of three doubles to float4 {x, y, z, 0}, or (ld > 0) to three vectors.
__global__ void mass_input32_kernel(int n, const double *__restrict__ in, float *__restrict__ out, int ld) {
  grid_dependency_wait();
  grid_dependents(kFewGatherBlocks);
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < 3 * n; t += gridDim.x * blockDim.x) {
    const int i = t / 3, c = t - 3 * i;
    out[ld > 0 ? (size_t)c * ld + i : 4 * (size_t)i + c] = convert::to_f32(in[t]);
  }
}

}  // namespace dev

// The dynamic shared memory limit above 48 KB that the tensor-core kernel
// opts into, once per device; returns the cudaError_t of the opt-in.
static cudaError_t tc_opt_in() {
  static PerDevice pd;
  return (cudaError_t)per_device(pd, [] {
    return (int)cudaFuncSetAttribute(dev::face_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)dev::tc::kSmemBytes);
  });
}
// The thread-per-face kernel's persistent grid (precision form, regular faces).
int face_blocks_tpf(int nfaces) {
  static PerDevice pd;
  const int cached = per_device(pd, [] {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, dev::face_tpf_kernel<false>, dev::tpf::kThreads,
                                                  dev::tpf::kSumBytes);
    return sm_count() * (per_sm > 0 ? per_sm : 1);
  });
  int need = grid_for(nfaces, dev::tpf::kThreads);
  return need < cached ? need : cached;
}

cudaError_t launch_faces_tpf(const TpfRows &rows, const dev::FaceLaunch &L, const int *dest,
                             const dev::SurfaceParams &P, const double *r, const F32Pos &f, float *partial,
                             double *blockpart, int *status, int grid, const FinishArgs &fin, int geo,
                             cudaStream_t s) {
  if (L.nfaces <= 0) return cudaSuccess;
  if (!f.hi || !f.lo || !f.dsp) return cudaErrorInvalidValue;
  return launch_after(geo ? dev::face_tpf_kernel<true> : dev::face_tpf_kernel<false>, grid, dev::tpf::kThreads,
                      dev::tpf::kSumBytes, s, rows, L, dest, P, r, f.hi, f.lo, f.dsp, partial, blockpart, status, fin);
}

cudaError_t launch_split_positions(int n, const double *r, const F32Pos &f, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (!f.hi || !f.lo || !f.r0 || !f.dsp) return cudaErrorInvalidValue;
  dev::split_positions_kernel<<<grid_for(n, 256), 256, 0, s>>>(n, r, f.hi, f.lo, f.r0, f.dsp);
  return cudaGetLastError();
}

constexpr int kStageThreads = 128;
cudaError_t launch_stage_in(int n, const double *host_r, double *r, const F32Pos &f, int *status, cudaStream_t s) {
  return launch_after(dev::stage_in_kernel, grid_for(n, kStageThreads), kStageThreads, 0, s, n, host_r, r, f.hi, f.lo, f.r0, f.dsp, status);
}

cudaError_t launch_status_merge(const int *src, int *dst, cudaStream_t s) {
  dev::status_merge_kernel<<<1, 1, 0, s>>>(src, dst);
  return cudaGetLastError();
}

// Small blocks, so that a small mesh's gather spreads over the SMs.
constexpr int kGatherThreads = 64;
template <typename T>
cudaError_t launch_gather(int nv, const T *partial, const int *off, double *g, int store, cudaStream_t s) {
  if (nv <= 0) return cudaSuccess;
  return launch_after(dev::gather_kernel<T>, grid_for(3 * nv, kGatherThreads), kGatherThreads, 0, s, nv, partial, off,
                      g, store);
}
template cudaError_t launch_gather<double>(int, const double *, const int *, double *, int, cudaStream_t);
template cudaError_t launch_gather<float>(int, const float *, const int *, double *, int, cudaStream_t);

template <typename T>
cudaError_t launch_gather_step(int nv, const T *partial, const int *off, const StepArgs &a, const uint64_t *cnt,
                               double *r, double *p, const F32Pos &f, const int *status, cudaStream_t s) {
  return launch_after(dev::gather_step_kernel<T>, grid_for(3 * nv, kGatherThreads), kGatherThreads, 0, s, nv, partial,
                      off, a, cnt, r, p, f.hi, f.lo, f.r0, f.dsp, status);
}
template cudaError_t launch_gather_step<double>(int, const double *, const int *, const StepArgs &, const uint64_t *,
                                                double *, double *, const F32Pos &, const int *, cudaStream_t);
template cudaError_t launch_gather_step<float>(int, const float *, const int *, const StepArgs &, const uint64_t *,
                                               double *, double *, const F32Pos &, const int *, cudaStream_t);

template <typename T>
cudaError_t launch_gather_kick(int nv, const T *partial, const int *off, const StepArgs &a, const uint64_t *cnt,
                               double *p, float *x32, int ld, const int *status, cudaStream_t s) {
  return launch_after(dev::gather_kick_kernel<T>, grid_for(3 * nv, kGatherThreads), kGatherThreads, 0, s, nv, partial,
                      off, a, cnt, p, x32, ld, status);
}
template cudaError_t launch_gather_kick<double>(int, const double *, const int *, const StepArgs &, const uint64_t *,
                                                double *, float *, int, const int *, cudaStream_t);
template cudaError_t launch_gather_kick<float>(int, const float *, const int *, const StepArgs &, const uint64_t *,
                                               double *, float *, int, const int *, cudaStream_t);
cudaError_t launch_drift(int nv, const StepArgs &a, double *r, double *p, const double *qdot, const F32Pos &f,
                         const int *status, cudaStream_t s) {
  return launch_after(dev::drift_kernel, grid_for(3 * nv, 256), 256, 0, s, nv, a, r, p, qdot, f.hi, f.lo, f.r0, f.dsp,
                      status);
}
cudaError_t launch_spmv32(int nrow, const int *row_ptr, const void *col, bool col16, const float *val,
                          const double *scalev, const MassScale &f, const float4 *in, double *out, int accumulate,
                          cudaStream_t s) {
  if (nrow <= 0) return cudaSuccess;
  int grid = grid_for(nrow, dev::kSpmvThreads / 32);
  if (grid > 152 * 16) grid = 152 * 16;
  // consecutive lanes take consecutive nonzeros, so runs of consecutive columns
  // gather the input with coalesced loads (a form with four nonzeros per lane,
  // 16-byte value loads, was slower: 0.80 against 0.55 ms at 40,962 rows)
  if (col16)
    return launch_after(dev::spmv32_kernel<uint16_t>, grid, dev::kSpmvThreads, 0, s, nrow, row_ptr,
                        static_cast<const uint16_t *>(col), val, scalev, f, in, out, accumulate);
  return launch_after(dev::spmv32_kernel<int>, grid, dev::kSpmvThreads, 0, s, nrow, row_ptr,
                      static_cast<const int *>(col), val, scalev, f, in, out, accumulate);
}

cudaError_t launch_mass_input32(int n, const double *in, float *out, int ld, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  return launch_after(dev::mass_input32_kernel, grid_for(3 * n, 256), 256, 0, s, n, in, out, ld);
}

cudaError_t launch_spmv(int nrow, const int *row_ptr, const int *col, const double *val, const double *scalev,
                        const MassScale &f, const double *in, double *out, int accumulate, cudaStream_t s) {
  if (nrow <= 0) return cudaSuccess;
  int warps_per_block = 8;
  int grid = grid_for(nrow, warps_per_block);
  if (grid > 152 * 16) grid = 152 * 16;
  return launch_after(dev::spmv_kernel, grid, 32 * warps_per_block, 0, s, nrow, row_ptr, col, val, scalev, f, in, out,
                      accumulate);
}

}  // namespace umcp

namespace umcp {

int batch_face_blocks_tpf() {
  static PerDevice pd;
  return per_device(pd, [] {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, dev::batch_face_tpf_kernel, dev::tpf::kThreads, 0);
    return sm_count() * (per_sm > 0 ? per_sm : 1);
  });
}

cudaError_t launch_batch_faces_tpf(const TpfRows &rows, const BatchJob *jobs, int group, const BatchTile *tiles,
                                   const int *counts, const float *table, double dudv, double *tile_sums, int grid,
                                   int *next_tile, cudaStream_t s) {
  if (!next_tile) return cudaErrorInvalidValue;
  return launch_after(dev::batch_face_tpf_kernel, grid, dev::tpf::kThreads, 0, s, rows, jobs, group, tiles, counts,
                      table, dudv, tile_sums, next_tile);
}

cudaError_t launch_batch_reduce(const BatchJob *jobs, const int *counts, int max_jobs, const int *tile_off,
                                const int *tile_idx, const double *tile_sums, int *live, unsigned long long *prog,
                                cudaStream_t s) {
  return launch_after(dev::batch_reduce_kernel, grid_for(max_jobs * 32, 256), 256, 0, s, jobs, counts, tile_off,
                      tile_idx, tile_sums, live, prog);
}

template <typename T>
cudaError_t launch_batch_gather_step(const BatchJob *jobs, const BatchTile *vtiles, const int *counts,
                                     const int *live, int grid, cudaStream_t s) {
  return launch_after(dev::batch_gather_step_kernel<T>, grid, kVertexTile, 0, s, jobs, vtiles, counts, live);
}
template cudaError_t launch_batch_gather_step<double>(const BatchJob *, const BatchTile *, const int *, const int *,
                                                      int, cudaStream_t);
template cudaError_t launch_batch_gather_step<float>(const BatchJob *, const BatchTile *, const int *, const int *,
                                                     int, cudaStream_t);

cudaError_t launch_batch_start(const BatchJob *jobs, const BatchTile *vtiles, const int *counts, const int *start,
                               const unsigned long long *step0, int grid, cudaStream_t s) {
  dev::batch_start_kernel<<<grid, kVertexTile, 0, s>>>(jobs, vtiles, counts, start, step0);
  return cudaGetLastError();
}

cudaError_t launch_batch_unpack(const BatchJob *jobs, const BatchTile *vtiles, const int *counts,
                                const long long *off, const double *pack, int grid, cudaStream_t s) {
  dev::batch_unpack_kernel<<<grid, kVertexTile, 0, s>>>(jobs, vtiles, counts, off, pack);
  return cudaGetLastError();
}

cudaError_t launch_batch_pack(const BatchJob *jobs, const BatchTile *vtiles, const int *counts, const long long *off,
                              double *pack, double *E, int grid, cudaStream_t s) {
  dev::batch_pack_kernel<<<grid, kVertexTile, 0, s>>>(jobs, vtiles, counts, off, pack, E);
  return cudaGetLastError();
}

}  // namespace umcp

namespace umcp {

// The FP64 pipe bounds the plain path's sums, so their blocks have to lie evenly over
// the SMs. Launched early beside a gather or a host call's stage-in that triggers
// (they do up to kFewGatherBlocks blocks), the blocks gather on the few SMs which
// that kernel leaves first. So above kChainedSums blocks they are a plain launch on
// meshes for which it triggers: a restrained evaluation of a 42 x 42 membrane (111
// blocks) 174 -> 150 us. Below, the early launch gains 3% (36 x 36, 81 blocks: 147 /
// 152 us; 38 x 38, 91 blocks: 172 / 150 us).
constexpr int kChainedSums = 84;
cudaError_t launch_geo_sums(const GeoArgs &G, bool staged, cudaStream_t s) {
  const int grid = geo_blocks(G.nfaces);
  const int triggering = (int)dev::kFewGatherBlocks * (staged ? kStageThreads : kGatherThreads) / 3;  // vertices
  if (grid <= kChainedSums || G.nv > triggering)
    return launch_after(dev::geo_sums_kernel, grid, kGeoThreads, 0, s, G);
  dev::geo_sums_kernel<<<grid, kGeoThreads, 0, s>>>(G);
  return cudaGetLastError();
}

// (The FP64 face pass does not trigger where this launch follows it, see face64.cu.)
template <typename T>
cudaError_t launch_geo_grad(const GeoArgs &G, T *partial, cudaStream_t s) {
  if (G.nfaces <= 0) return cudaSuccess;
  return launch_after(dev::geo_grad_kernel<T>, geo_blocks(G.nfaces), kGeoThreads, 0, s, G, partial);
}
template cudaError_t launch_geo_grad<double>(const GeoArgs &, double *, cudaStream_t);
template cudaError_t launch_geo_grad<float>(const GeoArgs &, float *, cudaStream_t);

}  // namespace umcp

namespace umcp {

int face_blocks_tc(int nfaces) {
  const int tiles = (nfaces + dev::tc::kFaces - 1) / dev::tc::kFaces;
  const int cap = 2 * sm_count();  // two CTAs per SM (shared memory and tensor memory)
  return tiles < 1 ? 1 : (tiles < cap ? tiles : cap);
}

cudaError_t launch_faces_tc(const dev::FaceLaunch &L, const int *dest, const dev::SurfaceParams &P, const double *r,
                            const float *rhi, const float *rlo, const float *dsp, float *partial, double *blockpart,
                            int *status, int grid, const FinishArgs &fin, cudaStream_t s) {
  if (!dsp) return cudaErrorInvalidValue;
  const cudaError_t e = tc_opt_in();
  if (e != cudaSuccess) return e;
  dev::face_tc_kernel<<<grid, dev::tc::kThreads, dev::tc::kSmemBytes, s>>>(L, dest, P, r, rhi, rlo, dsp, partial,
                                                                           blockpart, status, fin);
  return cudaGetLastError();
}

}  // namespace umcp
