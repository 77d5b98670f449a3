"""The first-derivative rows of a regular patch in FP32 (face32_table.h): each
entry the row's, to a rounding of its largest entries, and the row still exact on
fields that are linear over the patch."""
from __future__ import annotations

import subprocess

import numpy as np

import umcp_gb300 as U
from conftest import GOLDEN, ROOT

PROGRAM = """
#include <stdio.h>
#include "face32_table.h"
int main() {
  double b[12];
  for (;;) {
    for (int x = 0; x < 12; ++x)
      if (scanf("%lf", b + x) != 1) return 0;
    float f[12];
    umcp::round_tangent_row(b, f);
    for (int x = 0; x < 12; ++x) printf("%.9g ", f[x]);
    printf("\\n");
  }
}
"""


def test_rounded_rows_reproduce_linear_fields(tmp_path):
    basis = U.Plan(GOLDEN / "ico2_plain.mesh").basis(6)
    w, rows = basis["rows"][0], basis["rows"][1:3].reshape(30, 12)
    # the control points' lattice coordinates: the value rows reproduce (u, v)
    at = np.rint(np.linalg.lstsq(w, np.stack([basis["u"], basis["v"]], 1), rcond=None)[0])
    assert np.allclose(w @ at, np.stack([basis["u"], basis["v"]], 1), atol=1e-12)
    (tmp_path / "p.cpp").write_text(PROGRAM)
    exe = tmp_path / "p"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "umcp_gb300" / "csrc"), "-o", str(exe),
                    str(tmp_path / "p.cpp")], check=True)
    # the patch's rows, and rows that are no derivative of anything: zeros, one entry, ties
    extra = np.random.default_rng(3).normal(size=(20, 12))
    extra[0], extra[1], extra[2] = 0.0, np.eye(12)[10], 0.1
    cases = np.concatenate([rows, extra])
    text = "\n".join(" ".join("%.17g" % v for v in r) for r in cases)
    res = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout
    got = np.array([[float(v) for v in line.split()] for line in res.strip().split("\n")])
    assert got.shape == cases.shape
    most = np.abs(cases).max(axis=1, keepdims=True)
    # an entry takes its own rounding (2^-24 of the row's largest entry at most) and its share of the others'
    assert np.all(np.abs(got - cases) <= 2.0 ** -22 * most)
    assert np.array_equal(got[30], np.zeros(12)) and np.array_equal(got[31], np.eye(12)[10])
    error = np.abs((got[:30] - rows) @ at)
    plain = np.abs((rows.astype(np.float32).astype(np.float64) - rows) @ at)
    assert error.max() <= 4e-9 < plain.max()
