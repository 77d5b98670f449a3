"""The face pass at the edges of its kernels' ranges, against the oracle: face
counts that leave half-warps and blocks without work, patches of valence 5 and
7, flat membranes (a coordinate that is zero on every patch), coordinates many
powers of two away from 1 (each coordinate's integers carry their own
exponent), and non-finite ones.

Tolerances as in test_gpu_parity.py: 1e-10 of |E| and of max|g| in FP64, 1e-6
in the FP32 form.
"""
from __future__ import annotations

import numpy as np
import pytest

import umcp_gb300 as U
from conftest import rel_inf
from oracle import bridge as B

TOL = {U.FP64: 1e-10, U.FP32_CENTRED: 1e-6}


def flipped_vesicle(path, radius=100.0, seed=3):
    """A closed mesh with isolated vertices of valence 5 and 7: an icosphere
    with one edge flipped between regular vertices, each triangle then cut in
    four, the new vertices at edge midpoints pushed to the sphere."""
    U.generate_icosphere(path, 2, radius, 0.0, seed)
    plan = U.Plan(path)
    x = plan.positions()[:-3].reshape(-1, 3)
    val, ring = plan.rings()
    off = np.concatenate([[0], np.cumsum(val)])
    nb = [list(ring[off[i]:off[i + 1]]) for i in range(len(val))]
    tri = sorted({tuple(sorted((i, a, b))) for i in range(len(val)) for a in nb[i] for b in nb[a] if b in nb[i]})
    far = [i for i in range(len(val)) if val[i] == 6 and all(val[j] == 6 for j in nb[i])]
    a, b = next((i, j) for i in far for j in nb[i] if j in far)
    c, d = (k for k in nb[a] if k in nb[b])
    tri = [t for t in tri if not {a, b} <= set(t)] + [tuple(sorted((a, c, d))), tuple(sorted((b, c, d)))]
    pts, mid = [p for p in x], {}

    def half(i, j):
        key = (min(i, j), max(i, j))
        if key not in mid:
            m = x[i] + x[j]
            mid[key] = len(pts)
            pts.append(radius * m / np.linalg.norm(m))
        return mid[key]

    fine = []
    for i, j, k in tri:
        ij, jk, ki = half(i, j), half(j, k), half(k, i)
        fine += [(i, ij, ki), (j, jk, ij), (k, ki, jk), (ij, jk, ki)]
    nbr = [set() for _ in pts]
    for t in fine:
        for i in t:
            nbr[i] |= set(t) - {i}
    with open(path, "w") as f:
        f.write("3D flipped vesicle\n400 0 0\n0 400 0\n0 0 400\n")
        for i, p in enumerate(pts):
            f.write("%d %.17g %.17g %.17g %d %s\n" % (i, *p, len(nbr[i]), " ".join(map(str, sorted(nbr[i])))))
    return path


def _check(precision, path, scale=1.0, kg=-1.0, k_reg=0.1, flat=False, alpha=(1.0, 1.0, 1.0), sigma=0.05):
    prm = U.params(kc=U.kc_from_kT(20.0), KA=0.215, kg=kg, k_reg=k_reg, precision=precision)
    plan = U.Plan(path, prm)
    r = plan.positions()
    r[:-3] += np.random.default_rng(5).normal(0.0, sigma, r.size - 3)
    r[:-3] *= scale
    r[-3:] = alpha
    if flat:
        r[2:-3:3] = 0.0
    O = B.Oracle(plan, prm)
    E, g = U.Mesh(U.Context(0), plan, prm).energy_grad(r)
    Eo, go = O.energy(r), O.grad(r)
    assert abs(E - Eo) <= TOL[precision] * abs(Eo)
    assert rel_inf(g[:-3], go[:-3]) <= TOL[precision]
    if precision == U.FP64:
        assert np.allclose(g[-3:], go[-3:], rtol=TOL[precision], atol=TOL[precision] * np.abs(go).max())


def test_flipped_vesicle_has_patches_of_both_valences(tmp_path):
    plan = U.Plan(flipped_vesicle(tmp_path / "m.mesh"))
    v = plan.faces(1)["valence"]
    assert (v == 7).sum() == 14 and (v == 5).sum() == 70 and plan.n_regular > 0


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [U.FP64, U.FP32_CENTRED])
@pytest.mark.parametrize("terms", [False, True])
@pytest.mark.parametrize("nx,ny", [(4, 4), (5, 4), (7, 6), (9, 18), (33, 30)])
def test_remainders_of_periodic_membranes(tmp_path, nx, ny, terms, precision):
    if precision == U.FP32_CENTRED and nx < 7:
        pytest.skip("a patch wraps round a box this narrow: a folded surface, outside the FP32 form's stated bound")
    path = tmp_path / "m.mesh"
    U.generate_planar(path, nx, ny, 10.0, 20.0, 7)
    _check(precision, path, kg=-1.0 if terms else 0.0, k_reg=0.1 if terms else 0.0, alpha=(1.002, 0.999, 1.001))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [U.FP64, U.FP32_CENTRED])
@pytest.mark.parametrize("terms", [False, True])
def test_patches_of_valence_5_and_7(tmp_path, terms, precision):
    _check(precision, flipped_vesicle(tmp_path / "m.mesh"), kg=-1.0 if terms else 0.0, k_reg=0.1 if terms else 0.0,
           alpha=(1.003, 1.0, 0.998))


@pytest.mark.gpu
def test_flat_membrane(tmp_path):
    path = tmp_path / "m.mesh"
    U.generate_planar(path, 12, 10, 10.0, 20.0, 7)
    _check(U.FP64, path, flat=True)


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1e-6, 1e5])
def test_coordinates_of_other_magnitudes(tmp_path, scale):
    path = tmp_path / "m.mesh"
    U.generate_icosphere(path, 2, 100.0, 1.0, 11)
    _check(U.FP64, path, scale=scale)  # the state only: the reference metric stays


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [U.FP64, U.FP32_CENTRED])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_non_finite_coordinates_are_reported(tmp_path, value, precision):
    path = tmp_path / "m.mesh"
    U.generate_icosphere(path, 2, 100.0, 1.0, 11)
    prm = U.params(precision=precision)
    plan = U.Plan(path, prm)
    mesh = U.Mesh(U.Context(0), plan, prm)
    r = plan.positions()
    r[31] = value
    with pytest.raises(U.UmcpError, match="non-finite"):
        mesh.energy_grad(r)
    mesh.energy_grad(plan.positions())  # and the mesh is usable after it


@pytest.mark.gpu
@pytest.mark.parametrize("level", [5, 6])
def test_restrained_gradient_of_large_meshes(tmp_path, level):
    """Below and above the size where a thread per face takes over: the FP32
    form's restrained energy and gradient against the FP64 path's."""
    path = tmp_path / "m.mesh"
    U.generate_icosphere(path, level, 160.0 * 2 ** (level - 4), 1.0, 11)
    ctx, got = U.Context(0), {}
    for precision in (U.FP64, U.FP32_CENTRED):
        prm = U.params(kc=U.kc_from_kT(20.0), precision=precision)
        plan = U.Plan(path, prm)
        mesh = U.Mesh(ctx, plan, prm)
        mesh.restraints_set(K_area=0.2, K_volume=1e-4)
        r = plan.positions()
        r[:-3] += np.random.default_rng(5).normal(0.0, 0.05, r.size - 3)
        got[precision] = mesh.energy_grad(r)
    (E64, g64), (E32, g32) = got[U.FP64], got[U.FP32_CENTRED]
    assert abs(E32 - E64) <= TOL[U.FP32_CENTRED] * abs(E64)
    assert rel_inf(g32, g64) <= TOL[U.FP32_CENTRED]
