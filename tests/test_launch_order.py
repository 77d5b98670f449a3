"""A kernel that is launched early beside the one before it must not end up on a
few SMs only: the work of a larger mesh is more, and so is its time."""
from __future__ import annotations

import numpy as np
import pytest

import umcp_gb300 as U

pytestmark = pytest.mark.gpu


def _time_us(ctx, mesh, r, torch):
    """Median time of a restrained evaluation on device arrays."""
    stream = torch.cuda.ExternalStream(ctx.stream())
    d_r = torch.from_numpy(r).cuda()
    d_g, d_E = torch.zeros_like(d_r), torch.zeros(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    times = []
    for k in range(40):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record(stream)
        for _ in range(4):
            mesh.energy_grad_device(d_r.data_ptr(), d_E.data_ptr(), d_g.data_ptr())
        b.record(stream)
        b.synchronize()
        if k >= 8:
            times.append(a.elapsed_time(b) / 4 * 1e3)
    return float(np.median(times))


def test_restrained_fp64_evaluation_grows_with_the_mesh(tmp_path):
    """642 against 2,562 vertices, with restraints that act: a quarter of the
    work (139 and 251 us; 437 us for the smaller one while its gradient
    pass shared a few SMs)."""
    torch = pytest.importorskip("torch")
    ctx, times = U.Context(0), []
    for level in (3, 4):
        path = tmp_path / "m.mesh"
        U.generate_icosphere(path, level, 60.0 * 2 ** (level - 2), 1.0, 11)
        prm = U.params(kc=U.kc_from_kT(20.0))
        plan = U.Plan(path, prm)
        mesh = U.Mesh(ctx, plan, prm)
        r = plan.positions()
        mesh.restraints_set(K_area=0.2, K_volume=1e-5)
        mesh.energy(r)
        area, volume, _ = mesh.restraints_get()
        mesh.restraints_set(K_area=0.2, area0=0.999 * area, K_volume=1e-5, volume0=0.999 * volume)
        times.append(_time_us(ctx, mesh, r, torch))
    assert times[0] < times[1]
