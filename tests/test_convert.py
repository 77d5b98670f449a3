"""The integer conversions between doubles and floats (csrc/convert.h) give the
casts' bits: every exponent, halfway cases and their neighbours, signed zeros,
subnormals, infinities and NaN. The header is compiled for the host."""
from __future__ import annotations

import ctypes as C
import pathlib
import subprocess

import numpy as np
import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "umcp_gb300" / "csrc"


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("convert")
    (d / "c.cpp").write_text("""#include "convert.h"
extern "C" void down(long n, const double *x, float *y) { for (long i = 0; i < n; ++i) y[i] = umcp::convert::to_f32(x[i]); }
extern "C" void up(long n, const float *x, double *y) { for (long i = 0; i < n; ++i) y[i] = umcp::convert::to_f64(x[i]); }
extern "C" void two(long n, const double *x, float *h, float *l) {
  for (long i = 0; i < n; ++i) umcp::convert::to_f32_pair(x[i], h[i], l[i]);
}
""")
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", f"-I{CSRC}", "-o",
                    str(d / "c.so"), str(d / "c.cpp")], check=True)
    return C.CDLL(str(d / "c.so"))


def _doubles():
    rng = np.random.default_rng(7)
    frac = rng.integers(0, 1 << 52, 2047 * 40, dtype=np.uint64)
    frac[::5] &= ~np.uint64((1 << 29) - 1)               # exact floats
    frac[1::5] = (frac[1::5] & ~np.uint64((1 << 29) - 1)) | np.uint64(1 << 28)  # halfway
    frac[2::5] |= np.uint64(((1 << 23) - 1) << 29)        # rounding up carries into the exponent
    frac[3::10] = (frac[3::10] & ~np.uint64((1 << 29) - 1)) | np.uint64((1 << 28) + 1)
    exp = np.repeat(np.arange(2047, dtype=np.uint64), 40)
    sign = rng.integers(0, 2, exp.size, dtype=np.uint64)
    x = (sign << np.uint64(63) | exp << np.uint64(52) | frac).view(np.float64)
    return np.concatenate([x, [0.0, -0.0, np.inf, -np.inf, np.nan, 1.0, -1.0, 5e-324, -5e-324]])


def _same(got, want):
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    assert np.array_equal(got[ok], want[ok]) and np.array_equal(np.signbit(got[ok]), np.signbit(want[ok]))


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


@pytest.mark.filterwarnings("ignore:.*encountered in cast:RuntimeWarning")
def test_to_float(lib):
    x = _doubles()
    y = np.empty(x.size, np.float32)
    lib.down(C.c_long(x.size), _p(x), _p(y))
    _same(y, x.astype(np.float32))


def test_to_double(lib):
    rng = np.random.default_rng(8)
    exp = np.repeat(np.arange(256, dtype=np.uint32), 64)
    x = (rng.integers(0, 2, exp.size, dtype=np.uint32) << np.uint32(31) | exp << np.uint32(23)
         | rng.integers(0, 1 << 23, exp.size, dtype=np.uint32)).view(np.float32)
    x = np.concatenate([x, np.array([0.0, -0.0, np.inf, -np.inf], np.float32)])
    y = np.empty(x.size, np.float64)
    lib.up(C.c_long(x.size), _p(x), _p(y))
    _same(y, x.astype(np.float64))


@pytest.mark.filterwarnings("ignore:.*encountered in:RuntimeWarning")
def test_to_pair(lib):
    x = _doubles()
    h, l = np.empty(x.size, np.float32), np.empty(x.size, np.float32)
    lib.two(C.c_long(x.size), _p(x), _p(h), _p(l))
    want = x.astype(np.float32)
    _same(h, want)
    _same(l, (x - want.astype(np.float64)).astype(np.float32))
