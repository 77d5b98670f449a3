// Fixed-point numbers of the FP64 face pass (face64.cuh), host and device.
//
// GB300's FP64 pipe takes 64 cycles per warp instruction and scheduler (half a
// lane per cycle); a 32 x 32 + 64 bit integer multiply-add takes about 3.5. So
// the face pass forms its two basis contractions, two thirds of its FP64
// multiply-adds, in integers: a value is an integer of up to 57 bits times a
// power of two that its whole row (or control-point column) shares, held as two
// signed limbs, v = h 2^28 + l with -2^27 <= l < 2^27. A product takes three
// multiply-adds (h h, and h l + l h into one sum; l l is below the last bit
// kept). Magnitudes: basis rows and coordinates below 2^57 (|h| <= 2^29),
// adjoints below 2^55 (|h| <= 2^27 + 1), so the 64-bit sums hold 13 (forward)
// and 80 (backward) products. Operands keep 2^-57 (2^-55 the adjoints) of the
// largest of their row, the sums at least 2^-54 of the largest product, where a
// chain of FP64 multiply-adds rounds each partial sum to 2^-53: the integer
// sums are the more accurate ones.
#pragma once
#include <stdint.h>

#include <cmath>
#include <vector>

namespace umcp {
namespace fixed {

constexpr int kLimb = 28;        // bits of the low limb
constexpr int kRowBits = 57;     // |integer| < 2^57: basis rows, coordinates
constexpr int kAdjointBits = 55; // |integer| < 2^55: pointwise adjoints
constexpr int kBias = 1023;      // exponent bias of a double

// int4 stride of one point's five rows of limb pairs: two control points per
// int4, an odd count, so that the lanes of a quarter warp that read their own
// point's rows do not share banks.
constexpr int row_int4(int ncp) { return (5 * ((ncp + 1) / 2)) | 1; }
// ints of a patch type's table: the rows of every point, then five row exponents per point (padded to 8)
constexpr int table_ints(int ncp, int npt) { return npt * (4 * row_int4(ncp) + 8); }

// The table of a patch type from its rows basis[npt][5][ncpp]: each row as
// integers b 2^(56 - e), e the exponent of the row's largest entry.
inline std::vector<int> basis_table(const std::vector<double> &basis, int ncp, int npt, int ncpp) {
  std::vector<int> t((size_t)table_ints(ncp, npt), 0);
  const int row4 = row_int4(ncp), pairs = (ncp + 1) / 2;
  for (int p = 0; p < npt; ++p)
    for (int k = 0; k < 5; ++k) {
      const double *b = &basis[((size_t)p * 5 + k) * ncpp];
      double most = 0;
      for (int x = 0; x < ncp; ++x) most = std::fmax(most, std::fabs(b[x]));
      const int e = most > 0 ? std::ilogb(most) : 0;
      t[(size_t)npt * 4 * row4 + 8 * p + k] = e;
      for (int x = 0; x < ncp; ++x) {
        const int64_t v = std::llrint(std::ldexp(b[x], kRowBits - 1 - e));
        int64_t l = v & ((1ll << kLimb) - 1);
        if (l >= (1ll << (kLimb - 1))) l -= 1ll << kLimb;
        int *o = &t[((size_t)p * row4 + (size_t)k * pairs + x / 2) * 4 + 2 * (x & 1)];
        o[0] = (int)((v - l) / (1ll << kLimb));
        o[1] = (int)l;
      }
    }
  return t;
}

}  // namespace fixed
}  // namespace umcp
