"""The M^-1 apply at sizes that leave row groups, column chunks and warps with
remainders, against the installed matrix (umcp_mass_get) in numpy.

Bounds: each output against sum_j |A_ij| |x_j| times the rounding of the form's
products and input, 2^-52 per term in FP64 (n terms) and 4 x 2^-24 in the FP32
form (input and product rounded once each, sums compensated, with a factor 2).
"""
from __future__ import annotations

import numpy as np
import pytest

import umcp_gb300 as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [U.FP64, U.FP32_CENTRED])
@pytest.mark.parametrize("rel_tol", [1e-20, 0.02])
@pytest.mark.parametrize("mesh", ["planar 5x4", "planar 7x6", "planar 16x8", "planar 33x26", "level 2", "level 4"])
def test_apply_matches_the_installed_matrix(tmp_path, mesh, rel_tol, precision):
    path = tmp_path / "m.mesh"
    kind, size = mesh.split()
    if kind == "level":
        U.generate_icosphere(path, int(size), 100.0, 0.5, 3)
    else:
        nx, ny = map(int, size.split("x"))
        U.generate_planar(path, nx, ny, 10.0, 20.0, 3)
    prm = U.params(precision=precision)
    plan = U.Plan(path, prm)
    m = U.Mesh(U.Context(0), plan, prm)
    m.mass_build(plan, rel_tol=rel_tol)
    A, n = m.mass_get(), plan.nv
    rng = np.random.default_rng(7)
    x, out0, sv = rng.normal(size=3 * n), rng.normal(size=3 * n), rng.uniform(0.5, 2.0, 3 * n)
    alphas = (1.1, 0.9, 1.0)
    want = 0.7 * (A @ x.reshape(n, 3)) / np.square(alphas) * sv.reshape(3, n).T
    size_of = 0.7 * (np.abs(A) @ np.abs(x.reshape(n, 3))) / np.square(alphas) * sv.reshape(3, n).T
    tol = (n * 2.0 ** -52 if precision == U.FP64 else 4 * 2.0 ** -24) * size_of
    out = out0.copy()
    m.mass_apply(x, out, scalev=sv, scale=0.7, alphas=alphas)
    assert np.all(np.abs(out.reshape(n, 3) - out0.reshape(n, 3) - want) <= tol + 2.0 ** -50 * np.abs(out0.reshape(n, 3)))
    torch = pytest.importorskip("torch")
    dx, dv = torch.tensor(x, device="cuda"), torch.tensor(sv, device="cuda")
    do = torch.tensor(out0, device="cuda")
    torch.cuda.synchronize()
    m.mass_apply_device(dx.data_ptr(), do.data_ptr(), dv.data_ptr(), scale=0.7, alphas=alphas)
    assert np.array_equal(do.cpu().numpy(), out)
