// The precision form's staged table of a patch type: the image of the leading
// part of the half-warp face kernel's shared memory (face32.cuh), then the
// quadrature weights, then the restraints' corner matrix. Formed once per mesh on
// the host, so that no block converts rows from FP64.
#pragma once
#include <string.h>

#include <algorithm>
#include <cmath>
#include <vector>

namespace umcp {

template <int NCP, int NPT>
struct F32Table {
  static constexpr int NC4 = (NCP + 3) / 4;       // control points in fours
  static constexpr int ROW4 = (5 * NC4) | 1;      // float4 stride of a point's rows: odd, free of bank conflicts
  static constexpr int kRows = 0;                 // [NPT][ROW4][4]: rows u, v, uu, uv, vv
  static constexpr int kPoint4 = NPT * ROW4 * 4;  // [NPT][NCP][4]: u, v, uu, uv of each control point
  static constexpr int kPoint1 = kPoint4 + NPT * NCP * 4;  // [NPT][16]: vv
  static constexpr int kValue = kPoint1 + NPT * 16;        // [NPT][4 NC4]: the value row (restraints)
  static constexpr int kWeights = kValue + NPT * 4 * NC4;  // [16] doubles
  static constexpr int kCorner = kWeights + 32;            // [NCP][4 NC4]: corner_matrix
  static constexpr int kFloats = kCorner + NCP * 4 * NC4;
};

// The regular patch's rows for the thread-per-face kernel, which takes them as a
// launch parameter: all threads of a warp are at the same quadrature point, so its
// multiply-adds read them through the constant cache.
struct TpfRows {
  float B[15][5][12];  // rows u, v, uu, uv, vv of each point
  float V[15][12];     // value rows (restraints)
  float M[12][12];     // corner matrix (restraints)
};

// What the patch corner's position X0 has to do with the volume's gradient. Of the
// limit point R in the volume's sum c R.(Ru x Rv) the gradient's terms b_u (Rv x R) +
// b_v (R x Ru) take the corner's part as (sum_i M[j][i] X_i) x X0 for control point j,
//   M[j][i] = sum over the points of c (b_u[j] b_v[i] - b_v[j] b_u[i]),  c = dudv w / 3.
// The corner is a vesicle's radius away and the patch some tenths of an edge wide: left
// in the points' sums, X0 makes of every product a number that the others cancel to a
// fiftieth.
inline double corner_entry(const double *basis, const std::vector<double> &weight, double dudv, int npt, int ncpp, int j,
                           int i) {
  double s = 0;
  for (int p = 0; p < npt; ++p) {
    const double *u = basis + (size_t)p * 5 * ncpp, *v = u + ncpp;
    s += dudv * weight[p] / 3.0 * (u[j] * v[i] - v[j] * u[i]);
  }
  return s;
}

// A regular patch's first-derivative row in FP32, its entries chosen so that the row
// still gives the derivative of a linear field: over the control points' lattice
// coordinates (relative to control point 0, the patch corner) the rounding errors sum
// to nothing, to about 4e-9. A field that is linear over the patch is most of the
// tangents Ru and Rv, and every face has the same rows, so what plain rounding leaves
// of the two sums is one relative error of every tangent (2e-8 of the curvature
// energy). Largest entry first, each rounded after the least change of the entries
// still to be rounded that takes up the errors so far.
inline void round_tangent_row(const double *b, float *f) {
  static const int at[12][2] = {{0, 0},  {0, 1},  {1, 0}, {1, -1}, {0, -1}, {-1, 0},
                                {-1, 1}, {-1, 2}, {0, 2}, {1, 1},  {2, 0},  {2, -1}};
  int order[12];
  for (int x = 0; x < 12; ++x) order[x] = x;
  std::stable_sort(order, order + 12, [&](int x, int y) { return std::fabs(b[x]) > std::fabs(b[y]); });
  double sum[2] = {0, 0};  // errors so far times the lattice coordinates
  for (int k = 0; k < 12; ++k) {
    double uu = 0, uv = 0, vv = 0;
    for (int i = k; i < 12; ++i) {
      const int *q = at[order[i]];
      uu += q[0] * q[0];
      uv += q[0] * q[1];
      vv += q[1] * q[1];
    }
    const int x = order[k], *q = at[x];
    const double det = uu * vv - uv * uv;
    double change = 0;
    if (det > 0.5)
      change = -(q[0] * (vv * sum[0] - uv * sum[1]) + q[1] * (uu * sum[1] - uv * sum[0])) / det;
    else if (uu + vv > 0)  // the entries left lie on one line
      change = -(q[0] * sum[0] + q[1] * sum[1]) / (uu + vv);
    f[x] = (float)(b[x] + change);
    for (int d = 0; d < 2; ++d) sum[d] += ((double)f[x] - b[x]) * q[d];
  }
}

// Floats of a patch type's table.
inline int f32_table_floats(int ncp) {
  return ncp == 12 ? F32Table<12, 15>::kFloats : ncp == 11 ? F32Table<11, 16>::kFloats : F32Table<13, 16>::kFloats;
}

template <int NCP, int NPT>
void fill_f32_table(const std::vector<double> &basis, const std::vector<double> &value,
                    const std::vector<double> &weight, std::vector<float> *t) {
  using L = F32Table<NCP, NPT>;
  t->assign(L::kFloats, 0.f);
  for (int p = 0; p < NPT; ++p) {
    for (int k = 0; k < 5; ++k) {
      const double *row = &basis[((size_t)p * 5 + k) * (4 * L::NC4)];
      float *f = &(*t)[(size_t)(p * L::ROW4 + k * L::NC4) * 4];
      if (NCP == 12 && k < 2) round_tangent_row(row, f);
      else std::copy(row, row + NCP, f);
      for (int x = 0; x < NCP; ++x) (k < 4 ? (*t)[L::kPoint4 + (p * NCP + x) * 4 + k] : (*t)[L::kPoint1 + p * 16 + x]) = f[x];
    }
    for (int x = 0; x < NCP; ++x) (*t)[L::kValue + p * 4 * L::NC4 + x] = (float)value[(size_t)p * NCP + x];
  }
  memcpy(t->data() + L::kWeights, weight.data(), NPT * sizeof(double));
  for (int j = 0; j < NCP; ++j)
    for (int i = 0; i < NCP; ++i)
      (*t)[L::kCorner + j * 4 * L::NC4 + i] =
          (float)corner_entry(basis.data(), weight, NCP == 12 ? 0.5 : 1.0, NPT, 4 * L::NC4, j, i);
}

// The table from rows basis[npt][5][ncp rounded up to 4], value rows [npt][ncp] and the weights.
inline std::vector<float> f32_table(const std::vector<double> &basis, const std::vector<double> &value,
                                    const std::vector<double> &weight, int ncp) {
  std::vector<float> t;
  if (ncp == 12) fill_f32_table<12, 15>(basis, value, weight, &t);
  else if (ncp == 11) fill_f32_table<11, 16>(basis, value, weight, &t);
  else if (ncp == 13) fill_f32_table<13, 16>(basis, value, weight, &t);
  return t;
}

// The thread-per-face kernel's rows: the same values as the table's (12 control points).
inline TpfRows tpf_rows(const std::vector<float> &table) {
  using L = F32Table<12, 15>;
  TpfRows r;
  for (int p = 0; p < 15; ++p) {
    memcpy(r.B[p], &table[(size_t)p * L::ROW4 * 4], sizeof r.B[p]);
    memcpy(r.V[p], &table[L::kValue + (size_t)p * 12], sizeof r.V[p]);
  }
  memcpy(r.M, &table[L::kCorner], sizeof r.M);
  return r;
}

}  // namespace umcp
