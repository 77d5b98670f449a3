// The precision form's dense M^-1 apply: a row-major FP32 matrix (rows padded to
// 32 columns with zeros) times three FP32 vectors, with Kahan-compensated sums.
//
// What bounds it: the matrix streams from HBM once (10,242 rows: 420 MB, 62 us
// at the measured copy rate), and the compensated sums take 12 FP32 operations
// per element (about 35 us of the FP32 pipes). So every warp keeps two rounds of
// 16-byte loads in flight, the sums run as paired FP32 operations (two columns
// per instruction), and the work is cut evenly: the (row group, 128-column
// chunk) units, group by group, are dealt to the warps in equal runs, so that
// neither a last wave of row groups nor a mesh with few rows leaves SMs idle. A
// warp's run may start and end inside a row group; each piece's sums go to their
// own slot and the finish adds a row's slots in order. Results depend on the
// device's SM count only.
// Measured (one call on device arrays, about 19 us of it launch and wait):
// 10,242 rows 152 -> 98 us, 2,562 rows 46 -> 25 us, against four whole rows per
// warp with 4-byte loads. (Two units of loads ahead in registers instead of one:
// no gain at 10,242 rows, a Langevin step of 2,562 vertices 9% slower; through a
// shared-memory ring of two or three units: 3% faster than in registers before the
// vectors kept their L1 lines, not kept.)
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_common.cuh"
#include "face32.cuh"
#include "launch.h"
#include "launch_host.h"

namespace umcp {
namespace dev {
namespace dense32 {

constexpr int kRows = 4;      // rows of a group: one load of the vectors serves them all
constexpr int kChunk = 128;   // columns of a unit: a float4 per lane and row
constexpr int kThreads = 256, kWarps = kThreads / 32, kMinBlocks = 2;
constexpr int kSums = 3 * kRows;

// Two FP32 values in one register pair, and the paired operations on them.
typedef unsigned long long f2;
__device__ __forceinline__ f2 pair(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void split(f2 v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// A load of the matrix, which is read once: it leaves the L1 cache to the vectors
// (a warp reads their next chunk only when it sums it, so a miss is a stall: 10,242
// rows 106 us a call with evict-first loads, 98 with these).
__device__ __forceinline__ float4 load_once(const float *p) {
  float4 v;
  asm("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
// Units of warp w of W: [w U / W, (w + 1) U / W); the warp of unit u.
__host__ __device__ __forceinline__ long long first_unit(long long w, long long U, long long W) { return w * U / W; }
__host__ __device__ __forceinline__ long long warp_of(long long u, long long U, long long W) {
  return ((u + 1) * W - 1) / U;
}

// hi + lo of 12 sums over the warp by halving exchanges, error-free in pairs:
// lane l < 24 with l even (l / 2 < 12) ends with sum l / 2.
__device__ __forceinline__ double warp_sums(float (&hi)[16], float (&lo)[16]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int n = 16; n >= 2; n >>= 1) {  // n values left; partners differ in bit n of the lane
    const bool up = lane & n;
#pragma unroll
    for (int i = 0; i < n / 2; ++i) {
      // keep the half of the values that the lane's bit selects, send the other
      const float kh = up ? hi[i + n / 2] : hi[i], kl = up ? lo[i + n / 2] : lo[i];
      const float sh = up ? hi[i] : hi[i + n / 2], sl = up ? lo[i] : lo[i + n / 2];
      const float oh = __shfl_xor_sync(0xFFFFFFFFu, sh, n), ol = __shfl_xor_sync(0xFFFFFFFFu, sl, n);
      float t, e;
      two_sum(kh, oh, t, e);
      hi[i] = t;
      lo[i] = e + (kl + ol);
    }
  }
  const float oh = __shfl_xor_sync(0xFFFFFFFFu, hi[0], 1), ol = __shfl_xor_sync(0xFFFFFFFFu, lo[0], 1);
  float t, e;
  two_sum(hi[0], oh, t, e);
  return (double)t + (double)(e + (lo[0] + ol));
}

__global__ void __launch_bounds__(kThreads, kMinBlocks)
    dense_apply32_kernel(int n, int ld, int chunks, long long units, const float *__restrict__ A,
                         const float *__restrict__ x, double *__restrict__ part, int slots) {
  const int lane = threadIdx.x & 31;
  const long long W = (long long)gridDim.x * kWarps, w = (long long)blockIdx.x * kWarps + (threadIdx.x >> 5);
  const long long u0 = first_unit(w, units, W), u1 = first_unit(w + 1, units, W);
  if (u0 >= u1) return;
  int g = (int)(u0 / chunks), c = (int)(u0 % chunks);
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  auto load = [&](int gg, int cc, float4 m[kRows]) {
    const int j = cc * kChunk + 4 * lane;
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const int i = gg * kRows + r;
      m[r] = (i < n && j < ld) ? load_once(A + (size_t)i * ld + j) : zero4;
    }
  };
  f2 s[kSums], nc[kSums];  // Kahan sums of even and odd columns, and minus their compensations
#pragma unroll
  for (int q = 0; q < kSums; ++q) s[q] = nc[q] = 0;
  float4 m[kRows], nx[kRows];
  load(g, c, m);
  grid_dependency_wait();  // the vectors come from the kernel before; the matrix does not
  grid_dependents(gridDim.x);  // the finish is short and its blocks few
  for (long long u = u0; u < u1; ++u) {
    int gn = g, cn = c + 1;
    if (cn == chunks) { cn = 0; ++gn; }
    if (u + 1 < u1) load(gn, cn, nx);
    const int j = c * kChunk + 4 * lane;
    if (j < ld) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float4 v = *reinterpret_cast<const float4 *>(x + (size_t)k * ld + j);
        const f2 x01 = pair(v.x, v.y), x23 = pair(v.z, v.w);
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
          const int q = 3 * r + k;
          f2 y = fma2(pair(m[r].x, m[r].y), x01, nc[q]), t = add2(s[q], y);
          nc[q] = sub2(y, sub2(t, s[q]));
          s[q] = t;
          y = fma2(pair(m[r].z, m[r].w), x23, nc[q]);
          t = add2(s[q], y);
          nc[q] = sub2(y, sub2(t, s[q]));
          s[q] = t;
        }
      }
    }
    if (gn != g || u + 1 == u1) {  // the row group's last unit here: its sums to their slot
      float hi[16], lo[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        hi[q] = lo[q] = 0.f;
        if (q < kSums) {
          float a, b, ca, cb, e;
          split(s[q], a, b);
          split(nc[q], ca, cb);
          two_sum(a, b, hi[q], e);
          lo[q] = e + (ca + cb);
          s[q] = nc[q] = 0;
        }
      }
      const double sum = warp_sums(hi, lo);
      // after the exchanges lane l holds value (bit 4 of l) 8 + (bit 3) 4 + (bit 2) 2 + (bit 1)
      const int q = (lane >> 1) & 15;
      const int slot = (int)(w - warp_of((long long)g * chunks, units, W));
      if (!(lane & 1) && q < kSums) part[((size_t)g * slots + slot) * kSums + q] = sum;
    }
#pragma unroll
    for (int r = 0; r < kRows; ++r) m[r] = nx[r];
    g = gn;
    c = cn;
  }
}

// The slots of coordinate t = 3 i + k of the product and their sum, in order. Where
// they lie does not depend on the kernel before: found (by 64-bit divisions) before
// the wait for it.
struct Slots {
  const double *first;
  int n;
  __device__ __forceinline__ Slots(int t, int chunks, long long units, long long W, const double *__restrict__ part,
                                   int slots) {
    const int i = t / 3, k = t - 3 * i, g = i / kRows;
    n = (int)(warp_of((long long)(g + 1) * chunks - 1, units, W) - warp_of((long long)g * chunks, units, W)) + 1;
    first = part + (size_t)g * slots * kSums + 3 * (i - g * kRows) + k;
  }
  __device__ __forceinline__ double sum() const {
    double s = 0;
    int a = 0;
    for (; a + 4 <= n; a += 4) {
      double x[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) x[j] = first[(size_t)(a + j) * kSums];
#pragma unroll
      for (int j = 0; j < 4; ++j) s += x[j];
    }
    for (; a < n; ++a) s += first[(size_t)a * kSums];
    return s;
  }
};

// out (+)= f_c (scalev ? scalev[c n + i] : 1) (A x), one thread per coordinate.
__global__ void dense_finish32_kernel(int n, int chunks, long long units, long long W, const double *__restrict__ part,
                                      int slots, MassScale f, const double *__restrict__ scalev,
                                      double *__restrict__ out, int accumulate) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, i = t / 3, k = t - 3 * i;
  const bool on = t < 3 * n;
  const Slots mine(on ? t : 0, chunks, units, W, part, slots);
  grid_dependency_wait();
  if (!on) return;
  double v = f.f[k];
  if (scalev) v *= scalev[(size_t)k * n + i];
  const double before = accumulate ? out[t] : 0.0;
  v *= mine.sum();
  out[t] = accumulate ? before + v : v;
}

__global__ void dense_drift32_kernel(int n, int chunks, long long units, long long W, const double *__restrict__ part,
                                     int slots, StepArgs a, double *__restrict__ r, double *__restrict__ p,
                                     float *__restrict__ rhi, float *__restrict__ rlo, const double *__restrict__ r0,
                                     float *__restrict__ dsp, const int *__restrict__ status) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const bool on = t < 3 * n;
  const Slots mine(on ? t : 0, chunks, units, W, part, slots);
  grid_dependency_wait();
  if (!on) return;
  const int stopped = *status;
  const double q = mine.sum();  // its loads go out beside the status word's
  if (stopped) return;
  drift(a, t, q, r, p, rhi, rlo, r0, dsp);
}

}  // namespace dense32
}  // namespace dev

namespace {
struct Plan32 {
  int groups, chunks, grid, slots;
  long long units;
};
Plan32 plan32(int n, int ld) {
  using namespace dev::dense32;
  Plan32 p;
  p.groups = (n + kRows - 1) / kRows;
  p.chunks = (ld + kChunk - 1) / kChunk;
  p.units = (long long)p.groups * p.chunks;
  // at least two units a warp, so that the loads ahead have something to load
  const long long most = (p.units + 2 * kWarps - 1) / (2 * kWarps), fit = (long long)sm_count() * kMinBlocks;
  p.grid = (int)(most < fit ? most : fit);
  const long long W = (long long)p.grid * kWarps, least = p.units / W > 0 ? p.units / W : 1;
  p.slots = (int)((p.chunks + least - 1) / least) + 1;
  return p;
}
}  // namespace

size_t dense32_scratch_doubles(int n) {
  const Plan32 p = plan32(n, dense32_ld(n));
  return (size_t)p.groups * p.slots * dev::dense32::kSums;
}

static cudaError_t launch_units(int n, const float *A, const float *x, double *scratch, const Plan32 &p,
                                cudaStream_t s) {
  using namespace dev::dense32;
  return launch_after(dense_apply32_kernel, p.grid, kThreads, 0, s, n, dense32_ld(n), p.chunks, p.units, A, x, scratch,
                      p.slots);
}

cudaError_t launch_dense_apply32(int n, const float *A, const float *x, double *scratch, const MassScale &f,
                                 const double *scalev, double *out, int accumulate, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const Plan32 p = plan32(n, dense32_ld(n));
  const cudaError_t e = launch_units(n, A, x, scratch, p, s);
  if (e != cudaSuccess) return e;
  return launch_after(dev::dense32::dense_finish32_kernel, grid_for(3 * n, 128), 128, 0, s, n, p.chunks, p.units,
                      (long long)p.grid * dev::dense32::kWarps, scratch, p.slots, f, scalev, out, accumulate);
}

cudaError_t launch_dense_drift32(int n, const float *A, const float *x, double *scratch, const StepArgs &a, double *r,
                                 double *p, const F32Pos &f, const int *status, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const Plan32 q = plan32(n, dense32_ld(n));
  const cudaError_t e = launch_units(n, A, x, scratch, q, s);
  if (e != cudaSuccess) return e;
  return launch_after(dev::dense32::dense_drift32_kernel, grid_for(3 * n, 128), 128, 0, s, n, q.chunks, q.units,
                      (long long)q.grid * dev::dense32::kWarps, scratch, q.slots, a, r, p, f.hi, f.lo, f.r0, f.dsp,
                      status);
}

}  // namespace umcp
