"""Roundings that every face of the FP32 form has in common: no sum over faces
averages them out, so they are looked at apart from the random ones.

Bound: a face's own roundings (some 2^-22 of its energy, its points' partly in
common) average over n faces to about 2^-22 / sqrt(n), at 1,280 faces 7e-9.
Common are the basis rows' roundings (up to 2e-8 of the curvature energy when
each entry is rounded to nearest, worked out in FP64 from those rows). The two
add up to less than 3e-8, whatever the moduli. (The tensor-core option's rows
are 22-bit numbers, so it is not held to this.)
"""
from __future__ import annotations

import numpy as np
import pytest

import umcp_gb300 as U
from oracle import bridge as B

pytestmark = pytest.mark.gpu
BOUND = 3e-8

TWO_LIPIDS = "lipid library Lo 68.3 0.004\nlipid library Li 68.3 -0.004\nlipid outer Lo 1\nlipid inner Li 1\n"
OTHER_AREA = "lipid library La 61.7 0\nlipid outer La 1\nlipid inner La 1\n"


def _meshes(tmp_path):
    path = tmp_path / "m.mesh"
    U.generate_icosphere(path, 3, 100.0, 1.0, 11)
    return path


@pytest.mark.parametrize("lipids", [None, TWO_LIPIDS, OTHER_AREA])
@pytest.mark.parametrize("kc", [10.0, 12.5, 15.0, 17.3, 20.0, 37.0])
def test_energy_of_one_surface(tmp_path, kc, lipids):
    path = _meshes(tmp_path)
    prm = U.params(kc=U.kc_from_kT(kc), KA=0.215, precision=U.FP32_CENTRED, lipids=lipids)
    plan = U.Plan(path, prm)
    mesh = U.Mesh(U.Context(0), plan, prm)
    off = []
    for seed in range(4):
        r = plan.positions()
        r[:-3] += np.random.default_rng(seed).normal(0.0, 0.05, r.size - 3)
        want = B.Oracle(plan, prm).energy(r)
        off.append(mesh.energy(r) / want - 1.0)
    assert abs(np.mean(off)) <= BOUND, off


def test_parameters_set_later_and_batches(tmp_path):
    """The same for moduli set after the mesh was made, and for the jobs of a batch."""
    path = _meshes(tmp_path)
    kcs = [10.0, 15.0, 20.0, 37.0]
    made = U.params(kc=U.kc_from_kT(5.0), KA=0.1, precision=U.FP32_CENTRED)
    plan = U.Plan(path, made)
    ctx, meshes, want = U.Context(0), [], []
    r = plan.positions()
    r[:-3] += np.random.default_rng(0).normal(0.0, 0.05, r.size - 3)
    batch = U.Batch(ctx, U.FP32_CENTRED)
    for kc in kcs:
        prm = U.params(kc=U.kc_from_kT(kc), KA=0.215, precision=U.FP32_CENTRED)
        mesh = U.Mesh(ctx, plan, made)
        mesh.set_params(prm)
        fresh = U.Mesh(ctx, plan, prm)
        want.append(B.Oracle(plan, prm).energy(r))
        assert mesh.energy(r) == fresh.energy(r)
        assert abs(mesh.energy(r) / want[-1] - 1.0) <= BOUND
        meshes.append(mesh)
        batch.add(mesh, U.integrator(U.OVERDAMPED_BD, time_step=1.0, D=1e-6, seed=3), 0, 4)
    E, out = np.zeros(len(kcs)), np.zeros(len(kcs) * r.size)
    batch.step_host(np.tile(r, len(kcs)), out, E, 1)
    assert np.all(np.abs(E / np.array(want) - 1.0) <= BOUND)
