"""The area and volume sums at the edges of their kernel's ranges, against the
oracle: patches of valence 5 and 7, face counts that are no multiple of a
block's 32, more faces than one round of blocks, periodic images (area only),
box scales, coordinates far from 1, and non-finite ones.

Tolerances of the FP32 form. A: 1e-6, as in test_restraints.py. V: the positions
and box scales enter as pairs of FP32 (2^-48 each, four of them to a product:
1.4e-14) and the oracle sums up to 2e4 terms in FP64 (1e-14 at random): 1e-13.
"""
from __future__ import annotations

import numpy as np
import pytest

import umcp_gb300 as U
from oracle import restraints as OR
from test_face_edges import flipped_vesicle


def _mesh(path, precision, alpha=(1.01, 0.99, 1.02), sigma=0.2, scale=1.0):
    prm = U.params(precision=precision)
    plan = U.Plan(path, prm)
    r = plan.positions()
    r[:-3] += np.random.default_rng(5).normal(0.0, sigma, r.size - 3)
    r[:-3] *= scale
    r[-3:] = alpha
    return plan, U.Mesh(U.Context(0), plan, prm), r


def _check(plan, mesh, r, precision, volume=True):
    A, V = OR.area_volume(plan, r)
    mesh.restraints_set(K_area=0.2, area0=1.01 * A, K_volume=1e-4 if volume else 0.0,
                        volume0=1.001 * V if volume else 0.0)
    mesh.energy_grad(r)
    a, v, _ = mesh.restraints_get()
    assert abs(a - A) <= (1e-12 if precision == U.FP64 else 1e-6) * A
    if volume:
        assert abs(v - V) <= (1e-12 if precision == U.FP64 else 1e-13) * abs(V)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [U.FP64, U.FP32_CENTRED])
@pytest.mark.parametrize("scale", [1.0, 1e-3, 1e4])
def test_sums_with_patches_of_valence_5_and_7(tmp_path, scale, precision):
    plan, mesh, r = _mesh(flipped_vesicle(tmp_path / "m.mesh"), precision, scale=scale)
    assert plan.n_regular % 32 != 0
    _check(plan, mesh, r, precision)


@pytest.mark.gpu
@pytest.mark.parametrize("level", [1, 2, 4])
def test_sums_of_vesicles(tmp_path, level):
    path = tmp_path / "m.mesh"
    U.generate_icosphere(path, level, 30.0 * 2 ** level, 1.0, 11)
    _check(*_mesh(path, U.FP32_CENTRED), U.FP32_CENTRED)


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(7, 6), (33, 30), (110, 120)])
def test_area_of_periodic_membranes(tmp_path, nx, ny):
    path = tmp_path / "m.mesh"
    U.generate_planar(path, nx, ny, 10.0, 20.0, 7)
    _check(*_mesh(path, U.FP32_CENTRED), U.FP32_CENTRED, volume=False)


@pytest.mark.gpu
@pytest.mark.parametrize("value", [np.nan, np.inf, 1e35])
def test_coordinates_out_of_range_are_reported(tmp_path, value):
    path = tmp_path / "m.mesh"
    U.generate_icosphere(path, 2, 100.0, 1.0, 11)
    plan, mesh, r = _mesh(path, U.FP32_CENTRED)
    mesh.restraints_set(K_area=0.2, K_volume=1e-4)
    bad = r.copy()
    bad[31] = value
    with pytest.raises(U.UmcpError, match="non-finite"):
        mesh.energy_grad(bad)
    mesh.energy_grad(r)
