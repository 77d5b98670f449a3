// The precision form's area and volume sums: A = sum dudv w |Ru x Rv| and
// V = 1/3 sum dudv w R.(Ru x Rv) over every quadrature point, V to float-float
// accuracy (why, stands at geo_sums_kernel), the area and the box-scale
// derivatives from the FP32 leading parts with Kahan sums. FP64 enters only in the
// per-block and final sums.
//
// Bound by issue: 108 multiply-adds of better than FP32 accuracy a point (three
// rows, three coordinates, 12 control points), and about 250 instructions of the
// triple product. A float-float multiply-add takes 12 FP32 instructions. Here a
// coordinate is an integer of 28 bits h, scaled by a power of two that its patch
// shares, and an FP32 remainder l; a row entry likewise (bh, bl). The leading
// products bh h are exact in 64-bit integers (one instruction of 3.4 cycles, and
// none of their sums rounds), and bl x + bf l, 2^-28 of them, is two FP32
// multiply-adds: 5.4 cycles for 12, and a sum good to 2^-50 of the patch's size
// where the float-float chain kept about 2^-48.
//
// A block takes 32 faces of one patch type at a time. Its four warps share them:
// lane = face, and each warp prepares a quarter of the control points and then
// walks a quarter of the quadrature points. So a warp's row reads are broadcasts
// from shared memory, what a face needs there is spread over four threads, and a
// mesh of 1,280 faces still has 40 blocks.
//
// Measured on 81,920 faces: a restrained evaluation alone 206 -> 121 us (27 us of it by
// summing the block rows in parallel), three in flight 129 -> 88 us each (91 with the
// volume gradient's corner part, GeoCorner).
// The error of V against extended precision is the smaller one, 0.4e-15 to 1.1e-15
// relative where it was 0.4e-15 to 1.4e-15 (162 to 40,962 vertices). Rows through
// the constant cache: 3 us slower in the best form, the rows take registers before
// their use; five blocks a SM: 4 us slower (96 registers); the point's control-point
// loop unrolled: 10 us slower (spills).
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_common.cuh"
#include "face32.cuh"
#include "geo.cuh"
#include "geo32_table.h"
#include "launch.h"
#include "launch_host.h"

namespace umcp {
namespace dev {

// ---- float-float (double-FP32) arithmetic.
// A value is hi + lo with |lo| <= ulp(hi)/2; the error-free transformations
// are Knuth's two-sum and the FMA two-product (Dekker's product with a fused
// multiply-add), so the arithmetic stays on the FP32 pipes and carries about
// 44 bits. Every product and sum inside them is rounded on its own (no
// contraction into an FMA), as the transformations require.
struct FF {
  float hi, lo;
};
__device__ __forceinline__ FF ff_fast_two_sum(float a, float b) {  // |a| >= |b| or a == 0
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ FF ff_add(FF x, FF y) {
  float s, e;
  two_sum(x.hi, y.hi, s, e);
  e = __fadd_rn(e, __fadd_rn(x.lo, y.lo));
  return ff_fast_two_sum(s, e);
}
__device__ __forceinline__ FF ff_mul(FF x, FF y) {
  const float p = __fmul_rn(x.hi, y.hi);
  float e = __fmaf_rn(x.hi, y.hi, -p);
  e = __fmaf_rn(x.hi, y.lo, e);
  e = __fmaf_rn(x.lo, y.hi, e);
  return ff_fast_two_sum(p, e);
}
__device__ __forceinline__ FF ff_of(double x) {
  const float h = (float)x;
  return {h, (float)(x - (double)h)};
}


namespace geo32 {
constexpr int kThreads = kGeoThreads, kWarps = kThreads / 32, kMinBlocks = 4;
static_assert(kWarps == 4, "a warp takes a quarter of the points");
// floats of a face's column: h, x, l of each coordinate, padded so that its length
// is an odd number of 16-byte chunks and a warp's 16-byte reads do not conflict
template <int NCPP>
constexpr int kStride = NCPP == 12 ? 108 : 148;
constexpr int kColumns = 32 * kStride<16>;
static_assert(sizeof(float) * kColumns >= sizeof(double) * kGeoWords * kThreads, "block sums use the columns' space");
constexpr int kTop = 34;  // low bits of a 64-bit sum that go to the low part

__device__ __forceinline__ float exp2i(int e) { return __int_as_float((e + 127) << 23); }  // -126 <= e <= 127
__device__ __forceinline__ long long mad_wide(int a, int b, long long c) {
  long long d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}
// S 2^(e - 56) + c: the bits from 2^kTop up are the high part, exact in FP32 (|S| < 2^58: a
// row's entries add up to less than 4 in magnitude).
__device__ __forceinline__ FF from_sum(long long S, float c, int e) {
  const int top = ((int)(S >> (kTop - 1)) + 1) >> 1;  // S / 2^kTop, rounded
  const int low = (int)(S >> 2);                      // the rest: the kTop bits below, as a signed number
  static_assert(kTop == 34, "low: bits 2 to 33 are a word");
  return ff_fast_two_sum(__fmul_rn((float)top, exp2i(e - 2 * kGeoRowBits + kTop)),
                         __fmaf_rn((float)low, exp2i(e - 2 * kGeoRowBits + 2), c));
}

// x y as hi + lo without normalising lo (terms of a sum that is normalised at its end).
__device__ __forceinline__ FF product(FF x, FF y) {
  const float p = __fmul_rn(x.hi, y.hi);
  return {p, __fmaf_rn(x.lo, y.hi, __fmaf_rn(x.hi, y.lo, __fmaf_rn(x.hi, y.hi, -p)))};
}

// One thread's running sums.
struct Sums {
  FF V = {0, 0};
  float s[kGeoWords] = {}, c[kGeoWords] = {};  // Kahan: A, -, dA/dalpha (3), dV/dalpha (3)
  __device__ __forceinline__ void add(int q, float v) {
    const float y = v - c[q], t = s[q] + y;
    c[q] = (t - s[q]) - y;
    s[q] = t;
  }
};

// 32 faces of one patch type, from face `first` of it.
template <int NCP, int NPT, int NCPP, bool DA>
__device__ __forceinline__ void faces(const GeoRows<NCPP> &rows, const GeoArgs &G, const GeoGroup &g, int first,
                                      const FF alpha[3], const float ialpha[3], float *cols, unsigned (*most)[32],
                                      Sums &acc) {
  constexpr int PER = NCPP / kWarps;  // control points a warp prepares
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool on = first + lane < g.nfaces;
  const uint32_t *cp = g.cp + (size_t)min(first + lane, g.nfaces - 1) * NCP;
  float *col = cols + kStride<NCPP> * lane;
  // ---- coordinates relative to the corner, in their images, times alpha: float-float
  float ahi[3], alo[3], dsp[3];  // dsp: not used here
  f32::load_vertex(G.rhi, (int)(__ldg(&cp[0]) & kVertexMask), ahi, alo, dsp);
  FF X0[3], X[PER][3];
#pragma unroll
  for (int c = 0; c < 3; ++c) X0[c] = ff_mul(alpha[c], FF{ahi[c], alo[c]});  // the corner carries no image
  unsigned top = 0;  // largest magnitude, as bits (a NaN is above all)
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int j = warp * PER + k;
    X[k][0] = X[k][1] = X[k][2] = FF{0.f, 0.f};
    if (j < NCP) {
      const uint32_t packed = __ldg(&cp[j]);
      const int v = (int)(packed & kVertexMask), code = (int)(packed >> kVertexBits);
      float vh[3], vl[3], e1[3] = {0.f, 0.f, 0.f};  // vh + e1: the lattice image, e1 also the low part of the shift
      f32::load_vertex(G.rhi, v, vh, vl, dsp);
      if (code != 13) {  // a periodic image
        const int img[3] = {code % 3 - 1, (code / 3) % 3 - 1, code / 9 - 1};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          float sh = 0.f, she = 0.f, shl = 0.f;
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            float t, e;
            two_sum(sh, __fmul_rn((float)img[d], G.box_hi[d][c]), t, e);
            sh = t;
            she = __fadd_rn(she, e);
            shl = __fadd_rn(shl, __fmul_rn((float)img[d], G.box_lo[d][c]));
          }
          float s1;
          two_sum(vh[c], sh, s1, e1[c]);
          vh[c] = s1;
          e1[c] = __fadd_rn(e1[c], __fadd_rn(she, shl));
        }
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        float s2, e2;
        two_sum(vh[c], -ahi[c], s2, e2);
        const float res = __fadd_rn(__fadd_rn(e1[c], e2), __fsub_rn(vl[c], alo[c]));
        X[k][c] = ff_mul(alpha[c], ff_fast_two_sum(s2, res));
        top = max(top, __float_as_uint(X[k][c].hi) & 0x7FFFFFFFu);
      }
    }
  }
  most[warp][lane] = top;
  __syncthreads();  // and every warp is done with the columns of the faces before
  top = max(max(most[0][lane], most[1][lane]), max(most[2][lane], most[3][lane]));
  const bool far = top >= (unsigned)(127 + 90) << 23;  // R.(Ru x Rv) leaves FP32's range far below this
  const int e = far ? 0 : max((int)(top >> 23) - 126, -60);  // |x| < 2^e
  const float up = exp2i(kGeoRowBits - e), down = exp2i(e - kGeoRowBits);
#pragma unroll
  for (int k = 0; k < PER; ++k)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int h = far ? 0 : __float2int_rn(__fmul_rn(X[k][c].hi, up));
      float *q = col + c * NCPP + warp * PER + k;
      q[0] = __int_as_float(h);
      q[3 * NCPP] = X[k][c].hi;
      // (float)h is exact: above 2^24 it is the FP32 coordinate itself
      q[6 * NCPP] = __fadd_rn(__fmaf_rn((float)h, -down, X[k][c].hi), X[k][c].lo);
    }
  __syncthreads();
  // ---- the warp's points
  constexpr int kPer = (NPT + kWarps - 1) / kWarps;
  const int end = min((warp + 1) * kPer, NPT);
#pragma unroll 1
  for (int p = warp * kPer; p < end; ++p) {
    long long S[3][3];
    float C[3][3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int c = 0; c < 3; ++c) S[k][c] = 0, C[k][c] = 0.f;
#pragma unroll 1
    for (int q = 0; q < NCPP / 4; ++q) {
      int4 bh4[3];
      float4 bl4[3], bf4[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        bh4[k] = *reinterpret_cast<const int4 *>(&rows.bh[p][k][4 * q]);
        bl4[k] = *reinterpret_cast<const float4 *>(&rows.bl[p][k][4 * q]);
        bf4[k] = *reinterpret_cast<const float4 *>(&rows.bf[p][k][4 * q]);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int4 h4 = *reinterpret_cast<const int4 *>(&col[c * NCPP + 4 * q]);
        const float4 x4 = *reinterpret_cast<const float4 *>(&col[(3 + c) * NCPP + 4 * q]);
        const float4 l4 = *reinterpret_cast<const float4 *>(&col[(6 + c) * NCPP + 4 * q]);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const int4 bh = bh4[k];
          const float4 bl = bl4[k], bf = bf4[k];
          S[k][c] = mad_wide(bh.x, h4.x, S[k][c]);
          S[k][c] = mad_wide(bh.y, h4.y, S[k][c]);
          S[k][c] = mad_wide(bh.z, h4.z, S[k][c]);
          S[k][c] = mad_wide(bh.w, h4.w, S[k][c]);
          float a = C[k][c];
          a = __fmaf_rn(bl.x, x4.x, a);
          a = __fmaf_rn(bl.y, x4.y, a);
          a = __fmaf_rn(bl.z, x4.z, a);
          a = __fmaf_rn(bl.w, x4.w, a);
          a = __fmaf_rn(bf.x, l4.x, a);
          a = __fmaf_rn(bf.y, l4.y, a);
          a = __fmaf_rn(bf.z, l4.z, a);
          C[k][c] = __fmaf_rn(bf.w, l4.w, a);
        }
      }
    }
    FF Ra[3], Ru[3], Rv[3], m[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      Ra[c] = ff_add(X0[c], from_sum(S[0][c], C[0][c], e));
      Ru[c] = from_sum(S[1][c], C[1][c], e);
      Rv[c] = from_sum(S[2][c], C[2][c], e);
    }
    if (far) Ru[0].hi = __int_as_float(0x7FC00000);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int a = (c + 1) % 3, b = (c + 2) % 3;
      const FF p = product(Ru[a], Rv[b]), q = product(Ru[b], Rv[a]);
      float s, t;
      two_sum(p.hi, -q.hi, s, t);
      m[c] = ff_fast_two_sum(s, __fadd_rn(t, __fsub_rn(p.lo, q.lo)));
    }
    FF dot;
    {
      const FF x = product(Ra[0], m[0]), y = product(Ra[1], m[1]), z = product(Ra[2], m[2]);
      float s, t, s2, t2;
      two_sum(x.hi, y.hi, s, t);
      two_sum(s, z.hi, s2, t2);
      dot = ff_fast_two_sum(s2, __fadd_rn(__fadd_rn(t, t2), __fadd_rn(__fadd_rn(x.lo, y.lo), z.lo)));
    }
    const FF c3 = {rows.c3[0][p], rows.c3[1][p]};
    // area and box-scale derivatives from the leading parts
    const float Rf[3] = {Ra[0].hi, Ra[1].hi, Ra[2].hi}, Uf[3] = {Ru[0].hi, Ru[1].hi, Ru[2].hi},
                Vf[3] = {Rv[0].hi, Rv[1].hi, Rv[2].hi}, mf[3] = {m[0].hi, m[1].hi, m[2].hi};
    const float gg2 = mf[0] * mf[0] + mf[1] * mf[1] + mf[2] * mf[2];
    const float ig = rsqrtf(gg2), gg = gg2 * ig;
    const float cwf = rows.cw[p], c3f = c3.hi;
    if (!on) continue;
    // the weight's third part, 2^-50 of it: the same in every face, it would not average out
    FF v = ff_mul(c3, dot);
    v.lo = __fmaf_rn(rows.c3[2][p], dot.hi, v.lo);
    acc.V = ff_add(acc.V, v);
    acc.add(0, cwf * gg);
    if constexpr (!DA) continue;
    float n[3] = {mf[0] * ig, mf[1] * ig, mf[2] * ig}, a1[3], a2[3], v1[3], v2[3];
    cross3(Vf, n, a1);
    cross3(n, Uf, a2);
    cross3(Vf, Rf, v1);
    cross3(Rf, Uf, v2);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      acc.add(2 + k, cwf * (a1[k] * Uf[k] + a2[k] * Vf[k]) * ialpha[k]);
      acc.add(5 + k, c3f * (mf[k] * Rf[k] + v1[k] * Uf[k] + v2[k] * Vf[k]) * ialpha[k]);
    }
  }
}
}  // namespace geo32

// DA: the box-scale derivatives too (else the face launches form them).
template <bool DA>
__global__ void __launch_bounds__(geo32::kThreads, geo32::kMinBlocks)
    geo_sums32_kernel(const GeoArgs G) {
  using namespace geo32;
  __shared__ __align__(16) float cols[kColumns];
  __shared__ __align__(16) GeoRows<16> rows;  // of the patch type at hand (GeoRows<12> for the smaller ones)
  __shared__ unsigned most[kWarps][32];
  __shared__ FF alpha_s[3];
  __shared__ float ialpha_s[3];
  grid_dependency_wait();  // the state comes from the kernels before
  if (threadIdx.x < 3) {
    const double a = G.r[3 * (size_t)G.nv + threadIdx.x];
    alpha_s[threadIdx.x] = ff_of(a);
    ialpha_s[threadIdx.x] = 1.f / (float)a;
  }
  __syncthreads();
  const FF alpha[3] = {alpha_s[0], alpha_s[1], alpha_s[2]};
  const float ialpha[3] = {ialpha_s[0], ialpha_s[1], ialpha_s[2]};
  Sums acc;
  int batch = blockIdx.x, base = 0;  // batches count on from group to group
  for (int gi = 0; gi < G.ngroups; ++gi) {
    const GeoGroup &g = G.g[gi];
    const int n = (g.nfaces + 31) / 32;
    if (batch < base + n) {
      if (base > 0) __syncthreads();  // the rows of the type before are done with
      const int words = (int)((g.ncp <= 12 ? sizeof(GeoRows<12>) : sizeof(GeoRows<16>)) / 16);
      for (int i = threadIdx.x; i < words; i += kThreads)
        reinterpret_cast<float4 *>(&rows)[i] = __ldg(static_cast<const float4 *>(g.tab) + i);
      __syncthreads();
    }
    for (; batch < base + n; batch += gridDim.x) {
      const int first = 32 * (batch - base);
      if (g.ncp == 12)
        faces<12, 15, 12, DA>(*reinterpret_cast<const GeoRows<12> *>(&rows), G, g, first, alpha, ialpha, cols, most, acc);
      else if (g.ncp == 11)
        faces<11, 16, 12, DA>(*reinterpret_cast<const GeoRows<12> *>(&rows), G, g, first, alpha, ialpha, cols, most, acc);
      else
        faces<13, 16, 16, DA>(rows, G, g, first, alpha, ialpha, cols, most, acc);
    }
    base += n;
  }
  // block sums: warps in FP32 pairs, then the four of them
  __syncthreads();  // every column is done with: the block sums reuse their space
  double(*red)[kThreads] = reinterpret_cast<double(*)[kThreads]>(cols);
#pragma unroll
  for (int q = 0; q < kGeoWords; ++q) {
    const double s = q == kGeoV ? warp_sum(acc.V.hi, -acc.V.lo) : DA || q == kGeoA ? warp_sum(acc.s[q], acc.c[q]) : 0.0;
    if ((threadIdx.x & 31) == 0) red[q][threadIdx.x >> 5] = s;
  }
  __syncthreads();
  if (threadIdx.x < kGeoWords) {
    double s = red[threadIdx.x][0];
    for (int w = 1; w < kWarps; ++w) s += red[threadIdx.x][w];
    red[threadIdx.x][0] = s;
  }
  __syncthreads();
  geo_finish_rows(G, red);
}

}  // namespace dev

cudaError_t launch_geo_sums32(const GeoArgs &G, bool fused, cudaStream_t s) {
  int batches = 0;
  for (int k = 0; k < G.ngroups; ++k) batches += (G.g[k].nfaces + 31) / 32;
  // one round of blocks where there is work for one (four a SM; a constant, and the
  // sums' order with it a function of the face counts only), within the rows of geo_blocks
  constexpr int kRound = 152 * dev::geo32::kMinBlocks;
  const int most = geo_blocks(G.nfaces) < kRound ? geo_blocks(G.nfaces) : kRound;
  const int grid = batches < 1 ? 1 : (batches < most ? batches : most);
  return launch_after(fused ? dev::geo_sums32_kernel<false> : dev::geo_sums32_kernel<true>, grid, dev::geo32::kThreads,
                      0, s, G);
}

}  // namespace umcp
