"""The FP32 form's gradients where one comparison of the whole vector would hide
them: the vertices' and the box scales' apart (dE/dalpha is orders of magnitude
the larger), the vertices' under a volume restraint that acts, and dE/dalpha with
the angle term and box scales other than 1 on patches of every valence."""
from __future__ import annotations

import numpy as np
import pytest

import umcp_gb300 as U
from conftest import rel_l2
from oracle import bridge as B
from test_face_edges import flipped_vesicle

pytestmark = pytest.mark.gpu


def _partials_rounding(plan, r):
    """The volume gradient's partials of the regular faces, one per face and
    control point, as exact numbers rounded to FP32: (the norm of what that does to
    the vertices' sums) / (the norm of the sums)."""
    rows, weight = plan.basis(6)["rows"], plan.basis(6)["weight"]
    x, all_cp = r[:-3].reshape(-1, 3), plan.faces(0)["cp"][:, :12]
    w, u, v = rows[0], rows[1], rows[2]
    total, off = np.zeros_like(x), np.zeros_like(x)
    for k in range(0, len(all_cp), 8192):
        cp = all_cp[k:k + 8192]
        X = x[cp]
        R, Ru, Rv = (np.einsum("px,fxc->fpc", b, X) for b in (w, u, v))
        c = (0.5 * weight / 3.0)[None, :, None]
        part = (np.einsum("px,fpc->fxc", w, c * np.cross(Ru, Rv)) + np.einsum("px,fpc->fxc", u, c * np.cross(Rv, R))
                + np.einsum("px,fpc->fxc", v, c * np.cross(R, Ru)))
        np.add.at(total, cp.ravel(), part.reshape(-1, 3))
        np.add.at(off, cp.ravel(), (part.astype(np.float32).astype(np.float64) - part).reshape(-1, 3))
    return np.linalg.norm(off) / np.linalg.norm(total)


@pytest.mark.parametrize("level", [5, 6])  # half-warps, a thread per face
def test_vertex_gradient_under_a_volume_restraint(tmp_path, level):
    """Bound: a partial is a number some fifty times its share of the vertex's
    gradient, so its rounding to the FP32 slot is the floor. Forming it takes about
    nine roundings of its size besides (twelve multiply-adds on sums that grow, the
    corner's position, two products and their sum): sqrt(10) of the floor."""
    path = tmp_path / "m.mesh"
    U.generate_icosphere(path, level, 1000.0 * 2.0 ** (level - 6), 1.0, 11)
    ctx, got = U.Context(0), {}
    for precision in (U.FP64, U.FP32_CENTRED):
        prm = U.params(kc=U.kc_from_kT(20.0), precision=precision)
        plan = U.Plan(path, prm)
        mesh = U.Mesh(ctx, plan, prm)
        mesh.restraints_set(K_volume=0.01)  # target: the file's volume
        r = plan.positions()
        r[:-3] *= 1.0001                    # 0.03% off it: the restraint is nearly all of the gradient
        got[precision] = mesh.energy_grad(r)
    (E64, g64), (E32, g32) = got[U.FP64], got[U.FP32_CENTRED]
    assert abs(E32 - E64) <= 1e-6 * abs(E64)
    floor = _partials_rounding(plan, r)
    assert rel_l2(g32[:-3], g64[:-3]) <= np.sqrt(10.0) * floor, (rel_l2(g32[:-3], g64[:-3]), floor)
    assert rel_l2(g32[-3:], g64[-3:]) <= 1e-6


@pytest.mark.parametrize("level", [5, 6])
def test_vertex_gradient_under_both_restraints(tmp_path, level):
    """The FP32 form's bound for the vertices' part by itself, area and volume restrained, box scales off 1."""
    path = tmp_path / "m.mesh"
    U.generate_icosphere(path, level, 160.0 * 2 ** (level - 4), 1.0, 11)
    ctx, got = U.Context(0), {}
    for precision in (U.FP64, U.FP32_CENTRED):
        prm = U.params(kc=U.kc_from_kT(20.0), precision=precision)
        plan = U.Plan(path, prm)
        mesh = U.Mesh(ctx, plan, prm)
        r = plan.positions()
        mesh.restraints_set(K_area=0.2, K_volume=1e-4)
        mesh.energy(r)
        area, volume, _ = mesh.restraints_get()
        mesh.restraints_set(K_area=0.2, area0=0.999 * area, K_volume=1e-4, volume0=0.999 * volume)
        r[:-3] += np.random.default_rng(5).normal(0.0, 0.05, r.size - 3)
        r[-3:] = (1.002, 0.999, 1.001)
        got[precision] = mesh.energy_grad(r)
    (_, g64), (_, g32) = got[U.FP64], got[U.FP32_CENTRED]
    assert rel_l2(g32[:-3], g64[:-3]) <= 1e-6
    assert rel_l2(g32[-3:], g64[-3:]) <= 1e-6


@pytest.mark.parametrize("terms", [False, True])
@pytest.mark.parametrize("alpha", [(1.0, 1.0, 1.0), (1.003, 1.0, 0.998)])
def test_box_scale_derivatives_on_every_valence(tmp_path, alpha, terms):
    """dE/dalpha against the oracle, 1e-6 of its norm (the angle term adds a part of its own on valence 5 and 7)."""
    prm = U.params(kc=U.kc_from_kT(20.0), KA=0.215, kg=-1.0 if terms else 0.0, k_reg=0.5 if terms else 0.0,
                   precision=U.FP32_CENTRED)
    plan = U.Plan(flipped_vesicle(tmp_path / "m.mesh"), prm)
    r = plan.positions()
    r[:-3] += np.random.default_rng(5).normal(0.0, 0.05, r.size - 3)
    r[-3:] = alpha
    _, g = U.Mesh(U.Context(0), plan, prm).energy_grad(r)
    assert rel_l2(g[-3:], B.Oracle(plan, prm).grad(r)[-3:]) <= 1e-6
