// The precision form's restraint table of a patch type: the value and first-
// derivative rows and the point weights for the sums kernel (geo32.cu) and the
// gradient pass (geo_grad_kernel). Formed once, when restraints are first set.
#pragma once
#include <cmath>
#include <vector>

namespace umcp {

constexpr int kGeoRowBits = 28;  // a row entry is bh 2^-28 + bl
constexpr int kGeoPt = 16;       // quadrature points of the largest rule

// Rows w, u, v of every point, control points padded with zeros to NCPP.
template <int NCPP>
struct alignas(16) GeoRows {
  int bh[kGeoPt][3][NCPP];
  float bl[kGeoPt][3][NCPP], bf[kGeoPt][3][NCPP];  // the remainder; the entry in FP32
  float cw[kGeoPt], c3[3][kGeoPt];                 // dudv w; dudv w / 3 as a sum of three, largest first
};
inline int geo_padded(int ncp) { return ncp <= 12 ? 12 : 16; }

// From rows basis[npt][5][ncpp] (u, v first), value rows bw[npt][ncp] and the weights.
template <int NCPP>
void fill_geo_rows(const std::vector<double> &basis, const std::vector<double> &bw, const std::vector<double> &weight,
                   double dudv, int ncp, int npt, int ncpp, GeoRows<NCPP> *t) {
  *t = GeoRows<NCPP>{};
  for (int p = 0; p < npt; ++p) {
    for (int k = 0; k < 3; ++k)
      for (int x = 0; x < ncp; ++x) {
        const double b = k == 0 ? bw[(size_t)p * ncp + x] : basis[((size_t)p * 5 + (k - 1)) * ncpp + x];
        const int h = (int)std::lrint(std::ldexp(b, kGeoRowBits));
        t->bh[p][k][x] = h;
        t->bl[p][k][x] = (float)(b - std::ldexp((double)h, -kGeoRowBits));
        t->bf[p][k][x] = (float)b;
      }
    const double cw = dudv * weight[p], c3 = cw / 3.0;
    t->cw[p] = (float)cw;
    double rest = c3;
    for (int k = 0; k < 3; ++k) {
      t->c3[k][p] = (float)rest;
      rest -= (double)t->c3[k][p];
    }
  }
}

}  // namespace umcp
