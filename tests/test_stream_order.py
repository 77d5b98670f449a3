"""What a call puts into device memory is there before the context's stream uses
it. Copies and memsets without a stream go to the legacy stream, which a
context's non-blocking stream does not wait for, so the engine makes them in one
helper that waits (or makes them on the context's stream)."""
from __future__ import annotations

import re

import numpy as np
import pytest

import umcp_gb300 as U
from conftest import ROOT, rel_inf
from oracle import bridge as B

HELPER = "fill_device"


def _calls_without_a_stream(text):
    """Plain cudaMemset / cudaMemcpy to the device in a source text, outside the helper that waits for them."""
    helper = re.search(r"inline cudaError_t %s\(.*?\n}\n" % HELPER, text, re.S)
    if helper:
        assert "cudaStreamSynchronize(0)" in helper.group(0)
        text = text.replace(helper.group(0), "")
    calls = re.findall(r"\bcuda(?:Memset|Memset2D)\([^;]*;", text)
    calls += [c for c in re.findall(r"\bcuda(?:Memcpy|Memcpy2D)\([^;]*;", text) if "DeviceToHost" not in c]
    return calls


def test_device_memory_is_filled_with_a_wait_or_on_a_stream():
    sources = [p for p in sorted((ROOT / "umcp_gb300" / "csrc").iterdir()) if p.suffix in (".cu", ".cuh", ".h", ".cpp")]
    found = {p.name: _calls_without_a_stream(p.read_text()) for p in sources}
    assert len(found) > 10 and not {k: v for k, v in found.items() if v}


def _hold_the_legacy_stream(torch):
    """Some 30 ms of work on the legacy stream, queued."""
    x = torch.ones(1 << 28, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.default_stream()):
        for _ in range(100):
            x.mul_(1.0)
    return x


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [U.FP64, U.FP32_CENTRED])
@pytest.mark.parametrize("dense", [False, True])
def test_inverse_mass_installed_beside_a_busy_legacy_stream(tmp_path, dense, precision):
    """The first product, and the first steps with it, see the whole matrix and an input of their own."""
    torch = pytest.importorskip("torch")
    path = tmp_path / "m.mesh"
    U.generate_icosphere(path, 2, 75.0, 0.5, 3)
    prm = U.params(precision=precision)
    plan = U.Plan(path, prm)
    n = plan.nv
    rng = np.random.default_rng(7)
    x = rng.normal(size=3 * n)
    it = U.integrator(U.LANGEVIN, time_step=1e-15, gamma=10.0, seed=5, stream=2, use_mass=1)
    outs = []
    for hold in (True, False):
        m = U.Mesh(U.Context(0), plan, prm)
        held = _hold_the_legacy_stream(torch) if hold else None
        if dense:
            m.mass_build(plan)
        else:
            cols = np.stack([np.arange(n), (np.arange(n) + 1) % n], 1).astype(np.int32)
            m.mass_set(np.arange(0, 2 * n + 1, 2, dtype=np.int32), np.sort(cols, 1).ravel(), np.tile([0.5, 0.25], n))
        out = m.mass_apply(x, np.zeros_like(x))
        e = m.run(it, 0, 40)
        outs.append((m.mass_get(), out, e, *m.state_get()))
        del held
    if not dense:  # (an inverse built twice is the solver's, not bit for bit the same by contract)
        for a, b in zip(*outs):
            assert np.array_equal(a, b)
    A, out = outs[0][:2]
    want, size = A @ x.reshape(n, 3), np.abs(A) @ np.abs(x.reshape(n, 3))
    tol = n * 2.0 ** -52 if precision == U.FP64 else 4 * 2.0 ** -24  # as in test_mass_apply_edges.py
    assert np.all(np.abs(out.reshape(n, 3) - want) <= tol * size)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [U.FP64, U.FP32_CENTRED])
def test_mesh_and_restraints_made_beside_a_busy_legacy_stream(tmp_path, precision):
    torch = pytest.importorskip("torch")
    path = tmp_path / "m.mesh"
    U.generate_icosphere(path, 2, 75.0, 0.5, 3)
    prm = U.params(kc=U.kc_from_kT(20.0), precision=precision)
    plan = U.Plan(path, prm)
    r = plan.positions()
    r[:-3] += np.random.default_rng(5).normal(0.0, 0.05, r.size - 3)
    outs = []
    for hold in (True, False):
        held = _hold_the_legacy_stream(torch) if hold else None
        m = U.Mesh(U.Context(0), plan, prm)
        plain = m.energy_grad(r)
        held = _hold_the_legacy_stream(torch) if hold else None
        m.restraints_set(K_area=0.2, K_volume=1e-4)
        restrained = m.energy_grad(r)
        outs.append((*plain, *restrained))
        del held
    for a, b in zip(*outs):
        assert np.array_equal(a, b)
    O = B.Oracle(plan, prm)
    assert rel_inf(outs[0][1][:-3], O.grad(r)[:-3]) <= (1e-10 if precision == U.FP64 else 1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [U.FP64, U.FP32_CENTRED])
def test_runs_queued_behind_one_another_keep_their_steps(tmp_path, precision):
    """Two runs queued while the context's stream is still busy draw the noise of
    their own steps, as the same runs do one by one."""
    torch = pytest.importorskip("torch")
    path = tmp_path / "m.mesh"
    U.generate_icosphere(path, 2, 75.0, 0.5, 3)
    prm = U.params(precision=precision)
    plan = U.Plan(path, prm)
    it = U.integrator(U.OVERDAMPED_BD, time_step=1.0, D=1e-4, seed=5, stream=2)
    states = []
    for queued in (False, True):
        ctx = U.Context(0)
        m = U.Mesh(ctx, plan, prm)
        m.run(it, 0, 16)  # the steps are captured
        m.state_set(plan.positions())
        x = torch.ones(1 << 28, device="cuda")
        torch.cuda.synchronize()
        if queued:
            with torch.cuda.stream(torch.cuda.ExternalStream(ctx.stream())):
                for _ in range(100):  # some 30 ms
                    x.mul_(1.0)
        for step0 in (40, 1000, 56):
            m.run_async(it, step0, 16)
            if not queued:
                ctx.synchronize()
        ctx.synchronize()
        states.append(m.state_get()[0])
        del x
    assert np.array_equal(*states)
