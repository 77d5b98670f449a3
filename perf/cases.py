"""Workloads of the membrane engine, each one call (or one short run) through
the package's public entry points, with its inputs, its minimal work and its
value in 64 bits.

  listed()            the workloads by name
  draw(rng)           one more of the same ranges
  prepare(case, seed) what the caller has in hand: mesh, plan, state, handles
  run(state)          one pass; its outputs
  work(case)          bytes and operations a pass cannot do without
  exact(case, seed)   the same outputs from plain torch in 64 bits

Results that the FP32 form computes in FP32 (energies, gradients, momenta,
M^-1 products) are handed back as float32, as a caller that chose that form
holds them; positions stay FP64 in both forms.

The 64-bit values are formed from the discretisation the plan holds (control
points, lattice images, basis rows, quadrature weights, reference metric,
leaflet areas) and, for the M^-1 workloads, from the installed matrix: these
are the inputs of the measured calls. The energy, its derivative (by reverse
differentiation), the noise, the integrators and the products are plain torch.
"""
from __future__ import annotations

import concurrent.futures as cf
import math
import os
import random
import tempfile

import numpy as np
import torch

import umcp_gb300 as U

KT = U.KCAL_MOL_PER_KT_298
AKMA_S = 0.04888e-12  # one AKMA time unit in seconds
KA = 0.215


def listed():
    return [
        # The smallest call: energy and gradient of a 162-vertex vesicle (320
        # faces) from host arrays, as the reference's energy()/grad() are called.
        dict(name="eg_host_fp32_v162", op="eg", host=True, fp64=False, mesh="vesicle", level=2, radius=75.0, kc=20.0,
             c0=0.005, kg=0.0, k_reg=0.0, restrained=False),
        # One energy+gradient evaluation of the plain FP64 path, the 642-vertex
        # vesicle the reference is run on directly.
        dict(name="eg_host_fp64_v642", op="eg", host=True, fp64=True, mesh="vesicle", level=3, radius=100.0, kc=20.0,
             c0=0.0, kg=0.0, k_reg=0.0, restrained=False),
        # The same vesicle's overdamped BD, a stretch of its run with every energy kept.
        dict(name="bd_fp64_v642", op="run", kind="bd", fp64=True, mesh="vesicle", level=3, radius=100.0, kc=20.0,
             c0=0.0, kg=0.0, k_reg=0.0, steps=64),
        # FP64 on a periodic membrane of odd size, with the Gaussian-curvature
        # and angle terms and a box scale away from 1, on device arrays.
        dict(name="eg_dev_fp64_planar_61x46", op="eg", host=False, fp64=True, mesh="planar", nx=61, ny=46, kc=20.0,
             c0=0.0, kg=-5.0, k_reg=0.5, restrained=False),
        # The 128 x 128 periodic membrane's BD in the FP32 form.
        dict(name="bd_fp32_planar128", op="run", kind="bd", fp64=False, mesh="planar", nx=128, ny=128, kc=20.0, c0=0.0,
             kg=0.0, k_reg=0.0, steps=32),
        # A 10,242-vertex vesicle in the FP32 form on device arrays, with
        # spontaneous curvature, Gaussian-curvature and angle terms.
        dict(name="eg_dev_fp32_v10242", op="eg", host=False, fp64=False, mesh="vesicle", level=5, radius=300.0, kc=15.0,
             c0=-0.004, kg=-4.0, k_reg=0.3, restrained=False),
        # The large vesicle with global area and volume restraints.
        dict(name="eg_restrained_fp32_v40962", op="eg", host=False, fp64=False, mesh="vesicle", level=6, radius=1000.0,
             kc=20.0, c0=0.0, kg=0.0, k_reg=0.0, restrained=True),
        # Langevin dynamics with a truncated (sparse) M^-1 in the FP32 form.
        dict(name="ld_mass_fp32_v2562", op="run", kind="ld_mass", fp64=False, mesh="vesicle", level=4, radius=250.0,
             kc=20.0, c0=0.0, kg=0.0, k_reg=0.0, steps=32, rel_tol=1e-8),
        # M^-1 times a vector from host arrays, FP64, as the reference's
        # sparse multiply is called by a caller with its own integrator.
        dict(name="mass_host_fp64_v642", op="mass", host=True, fp64=True, mesh="vesicle", level=3, radius=100.0,
             rel_tol=1e-20),
        # The same product of a 10,242-vertex vesicle on device arrays in the
        # FP32 form (M^-1 stays dense at the reference's tolerance).
        dict(name="mass_dev_fp32_v10242", op="mass", host=False, fp64=False, mesh="vesicle", level=5, radius=300.0,
             rel_tol=1e-20),
        # 256 vesicles of mixed size driven from the host, one step per call:
        # states in, one batched step, states and energies out.
        dict(name="batch256_host_step", op="batch", fp64=False, jobs=256, mix=1003, steps=1),
        # A smaller mixed batch (as a server's slots hold), 32 steps on the device per call.
        dict(name="batch37_chunk32", op="batch", fp64=False, jobs=37, mix=11, steps=32),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    op = rng.choice(["eg", "eg", "eg", "run", "run", "mass", "batch"])
    fp64 = rng.random() < 0.4
    if op == "batch":
        return dict(op="batch", fp64=False, jobs=round(_log_uniform(rng, 3, 200)), mix=rng.randrange(10 ** 6),
                    steps=rng.choice([1, 1, 5, 16, 20]))
    if op == "mass":
        return dict(op="mass", host=rng.random() < 0.5, fp64=fp64, mesh="vesicle", level=rng.choice([2, 3, 4]),
                    radius=round(_log_uniform(rng, 60, 300), 2), rel_tol=rng.choice([1e-20, 1e-8, 1e-4]))
    c = dict(op=op, fp64=fp64)
    if rng.random() < 0.5:
        c |= dict(mesh="vesicle", level=rng.choice([2, 3, 4, 5] if fp64 else [2, 3, 4, 5, 6]),
                  radius=0.0, kc=round(rng.uniform(10, 40), 2))
        c["radius"] = round({2: 60.0, 3: 100.0, 4: 220.0, 5: 400.0, 6: 900.0}[c["level"]] * rng.uniform(0.8, 1.3), 2)
        c["c0"] = round(rng.uniform(-0.01, 0.01), 5) if rng.random() < 0.6 else 0.0
    else:
        top = 90 if fp64 else 220
        c |= dict(mesh="planar", nx=round(_log_uniform(rng, 8, top)), ny=2 * round(_log_uniform(rng, 4, top / 2)),
                  kc=round(rng.uniform(10, 40), 2), c0=0.0)
    terms = rng.random() < 0.4
    c |= dict(kg=round(rng.uniform(-8, 0), 2) if terms else 0.0, k_reg=round(rng.uniform(0, 1), 2) if terms else 0.0)
    if op == "eg":
        c |= dict(host=rng.random() < 0.5, restrained=c["mesh"] == "vesicle" and rng.random() < 0.3)
    else:
        c |= dict(kind=rng.choice(["bd", "bd", "ld"]), steps=rng.choice([1, 7, 20, 32]))
    return c


# ------------------------------------------------------------------ inputs


def _lipids(c0):
    """c0 on the outer leaflet's lipid, -c0 on the inner one's (the input file's only channel for c0)."""
    return (f"lipid library Lo 68.3 {c0!r}\nlipid library Li 68.3 {-c0!r}\nlipid outer Lo 1\nlipid inner Li 1\n"
            if c0 else None)


def _plan(case, seed, folder, name="m"):
    path = os.path.join(folder, name + ".mesh")
    if case["mesh"] == "vesicle":
        noise = 0.01 * case["radius"] if case["level"] < 6 else 2.0
        U.generate_icosphere(path, case["level"], case["radius"], noise, seed)
    else:
        U.generate_planar(path, case["nx"], case["ny"], 10.0, case["kc"], seed)
    prm = U.params(kc=U.kc_from_kT(case.get("kc", 20.0)), KA=KA, kg=case.get("kg", 0.0), k_reg=case.get("k_reg", 0.0),
                   precision=U.FP64 if case["fp64"] else U.FP32_CENTRED, lipids=_lipids(case.get("c0", 0.0)))
    plan = U.Plan(path, prm)
    os.remove(path)
    return plan, prm


def _jobs(case, seed):
    """The vesicles of a batch: levels from the case, everything else from the seed."""
    lev, rng = random.Random(case["mix"]), random.Random(seed)
    out = []
    for _ in range(case["jobs"]):
        level, u = lev.choice([2, 3, 4, 5]), rng.random()
        out.append(dict(mesh="vesicle", fp64=case["fp64"], level=level, radius=50.0 * 6.0 ** u,
                        kc=rng.uniform(10.0, 40.0), c0=rng.uniform(-0.01, 0.01)))
    return out


def _plans(case, seed):
    with tempfile.TemporaryDirectory() as folder:
        if case["op"] != "batch":
            return [_plan(case, seed, folder)]
        jobs = _jobs(case, seed)
        with cf.ThreadPoolExecutor(max_workers=min(16, os.cpu_count() or 1)) as ex:
            return list(ex.map(lambda k: _plan(jobs[k], seed * 1009 + k, folder, "m%d" % k), range(len(jobs))))


def _state(case, plan, seed):
    """A state of a run: the file's positions moved by 0.05 A per coordinate; a periodic box also scaled a little."""
    rng = np.random.default_rng(seed)
    r = plan.positions()
    r[:-3] += rng.normal(0.0, 0.05, r.size - 3)
    if case["op"] == "eg" and case["mesh"] == "planar":
        r[-3:] = 1.0 + rng.uniform(-0.01, 0.01, 3)
    return r


def _rms_step(case):
    """sqrt(2 D dt) of a BD step: 0.05 A on the single surfaces, 0.02 A where small stiff vesicles are in the mix."""
    return 0.02 if case["op"] == "batch" else 0.05


def _integrator(case, info=None, nv=0, stream=1):
    if case["op"] == "batch" or case["kind"] == "bd":
        s = _rms_step(case)
        return U.integrator(U.OVERDAMPED_BD, time_step=1.0, D=0.5 * s * s, seed=17, stream=stream)
    # a time step whose thermal displacement sqrt(kT <M^-1_ii>) dt is about 0.01 A; friction 1 / ps
    minv = 1.0 if info is None else float("%.3g" % (10.0 * nv / (info.mass_per_point * info.points)))
    return U.integrator(U.LANGEVIN, time_step=0.01 / math.sqrt(KT * minv) * AKMA_S, gamma=AKMA_S * 1e12, seed=17,
                        stream=stream, use_mass=1 if info is not None else 0)


def prepare(case, seed):
    ctx = U.Context(0)
    plans = _plans(case, seed)
    st = {"case": case, "ctx": ctx, "plans": plans}
    if case["op"] == "batch":
        with cf.ThreadPoolExecutor(max_workers=min(16, os.cpu_count() or 1)) as ex:
            st["meshes"] = list(ex.map(lambda q: U.Mesh(ctx, q[0], q[1]), plans))
        st["batch"] = U.Batch(ctx, U.FP64 if case["fp64"] else U.FP32_CENTRED)
        for k, m in enumerate(st["meshes"]):
            st["batch"].add(m, _integrator(case, stream=k), 0, 200_000)
        pack = np.concatenate([_state(case, plan, seed * 1013 + k) for k, (plan, _) in enumerate(plans)])
        st["r_in"] = torch.from_numpy(pack).pin_memory()
        st["r_out"] = torch.empty_like(st["r_in"]).pin_memory()
        st["E"] = torch.empty(len(plans), dtype=torch.float64).pin_memory()
        st["batch"].step_host(None, None, None, case["steps"])  # chooses the layout and captures the steps
        return st
    plan, prm = plans[0]
    mesh = st["mesh"] = U.Mesh(ctx, plan, prm)
    info = None
    if case["op"] == "mass" or case.get("kind") == "ld_mass":
        info = mesh.mass_build(plan, rel_tol=case["rel_tol"])
    if case.get("restrained"):
        mesh.restraints_set(K_area=0.2, K_volume=0.01)  # targets: the file's area and volume
    if case["op"] == "mass":
        x = np.random.default_rng(seed).normal(size=3 * plan.nv)
        if case["host"]:
            st |= {"x": x, "out": np.zeros_like(x)}
        else:
            st |= {"x": torch.from_numpy(x).cuda(), "out": torch.zeros(x.size, dtype=torch.float64, device="cuda")}
    elif case["op"] == "run":
        st |= {"r": _state(case, plan, seed), "it": _integrator(case, info, plan.nv)}
    elif case["host"]:
        st["r"] = _state(case, plan, seed)
    else:
        r = torch.from_numpy(_state(case, plan, seed)).cuda()
        st |= {"r": r, "g": torch.zeros_like(r), "E": torch.zeros(1, dtype=torch.float64, device="cuda")}
    if not case.get("host", True):
        st["stream"] = torch.cuda.ExternalStream(ctx.stream())
        torch.cuda.synchronize()
    return st


# ------------------------------------------------------------------ one pass


def _out(case, v):
    """v as a caller of the case's precision form holds it."""
    if case["fp64"]:
        return v if isinstance(v, torch.Tensor) else np.asarray(v)
    return v.float() if isinstance(v, torch.Tensor) else np.asarray(v, dtype=np.float32)


def run(st):
    case = st["case"]
    if case["op"] == "batch":
        st["batch"].step_host(st["r_in"].data_ptr(), st["r_out"].data_ptr(), st["E"].data_ptr(), case["steps"])
        return {"r": st["r_out"], "E": _out(case, st["E"])}
    mesh = st["mesh"]
    if case["op"] == "run":
        mesh.state_set(st["r"])
        e = mesh.run(st["it"], 0, case["steps"])
        r, p = mesh.state_get()
        return {"E": _out(case, e), "r": r} if case["kind"] == "bd" else {"E": _out(case, e), "r": r, "p": _out(case, p)}
    if case["op"] == "mass":
        if case["host"]:
            st["out"][:] = 0.0
            return _out(case, mesh.mass_apply(st["x"], st["out"], scale=0.5))
        with torch.cuda.stream(st["stream"]):
            st["out"].zero_()
            mesh.mass_apply_device(st["x"].data_ptr(), st["out"].data_ptr(), scale=0.5)
            return _out(case, st["out"])
    if case["host"]:
        e, g = mesh.energy_grad(st["r"])
        return {"E": _out(case, e), "g": _out(case, g)}
    with torch.cuda.stream(st["stream"]):
        st["g"].zero_()
        mesh.energy_grad_device(st["r"].data_ptr(), st["E"].data_ptr(), st["g"].data_ptr())
        return {"E": _out(case, st["E"]), "g": _out(case, st["g"])}


# ------------------------------------------------------------------ minimal work


def _sizes(case):
    """(vertices, regular faces, valence-5 faces) of each surface."""
    if case["op"] == "batch":
        out = []
        for j in _jobs(case, 0):
            out += _sizes(dict(j, op="eg"))
        return out
    if case["mesh"] == "planar":
        n = case["nx"] * (case["ny"] + case["ny"] % 2)
        return [(n, 2 * n, 0)]
    f = 20 * 4 ** case["level"]
    return [(f // 2 + 2, f - 60, 60)]


def work(case):
    b = 8 if case["fp64"] else 4
    terms = 2 if case.get("k_reg") else 1
    nbytes = flops = 0.0
    for nv, reg, irr in _sizes(case):
        state = 8.0 * (3 * nv + 3)
        if case["op"] == "mass":
            nbytes += b * float(nv) ** 2 + 2 * state
            flops += 6.0 * nv * nv
            continue
        # a face: its control points, the reference metric (and angle) of its points, its composition
        tables = reg * (12 * 4 + 15 * terms * b + 3 * b) + irr * (11 * 4 + 16 * terms * b + 3 * b)
        # a point: five rows over the control points, the pointwise energy and its derivative, the rows back
        ops = reg * 15 * (12 * 3 * (5 + 4) * 2 + 300) + irr * 16 * (11 * 3 * (5 + 4) * 2 + 300)
        n = case.get("steps", 1)
        if case["op"] == "eg":
            nbytes += tables + 2 * state + 8
            flops += ops * (1.5 if case.get("restrained") else 1.0)
        else:  # a run keeps its tables and state on the device: in and out once, and each step's energy
            nbytes += n * (tables + 2 * state) + 2 * state + 8 * n
            flops += n * (ops + 60.0 * nv)
            if case.get("kind") == "ld_mass":
                kept = 0.15 * nv * nv  # about what this truncation leaves of M^-1
                nbytes += n * kept * (b + 2)
                flops += n * 6.0 * kept
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------ in 64 bits


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Surfaces:
    """The limit-surface energy of one or many surfaces (vertices numbered through) in float64."""

    def __init__(self, plans, chunk=40_000):
        dev = _device()
        self.n, self.groups = len(plans), []
        self.off = np.cumsum([0] + [p.nv for p, _ in plans])
        self.nv = int(self.off[-1])
        self.vjob = torch.from_numpy(np.repeat(np.arange(self.n), np.diff(self.off))).to(dev)
        parts = {}
        for j, (plan, prm) in enumerate(plans):
            c0, _ = plan.lipids()
            for kind in (0, 1):
                if not (plan.n_irregular if kind else plan.n_regular):
                    continue
                t = plan.faces(kind)
                for val in ([6] if kind == 0 else sorted(set(t["valence"].tolist()))):
                    s = np.arange(len(t["cp"])) if kind == 0 else np.flatnonzero(t["valence"] == val)
                    ncp = val + 6
                    lip = np.stack([t["outer"][s].sum(1), t["outer"][s] @ c0, t["outer"][s] @ c0 ** 2,
                                    t["inner"][s].sum(1), t["inner"][s] @ c0, t["inner"][s] @ c0 ** 2], 1)
                    parts.setdefault(val, []).append((
                        t["cp"][s, :ncp].astype(np.int64) + self.off[j], t["img"][s, :ncp].astype(float) @ plan.box,
                        t["g0"][s], t["rr0"][s], lip, np.full(len(s), j), np.full(len(s), prm.kc)))
        self.KA, self.kg, self.k_reg = (getattr(plans[0][1], k) for k in ("KA", "kg", "k_reg"))
        for val, g in parts.items():
            basis = plans[0][0].basis(val)
            rows, w = (torch.from_numpy(np.ascontiguousarray(basis[k])).to(dev) for k in ("rows", "weight"))
            cols = [torch.from_numpy(np.ascontiguousarray(np.concatenate(c))).to(dev) for c in zip(*g)]
            for a in range(0, len(cols[0]), chunk):
                self.groups.append((rows, w, 0.5 if val == 6 else 1.0, [c[a:a + chunk] for c in cols]))

    def _points(self, g, r, alpha):
        rows, _, _, (cp, shift, *_rest) = g
        X = (r[cp] + shift) * alpha[_rest[3]][:, None, :]
        Y = X - X[:, :1]  # every row but the first sums to zero over the control points
        return X[:, 0], Y, [torch.einsum("pj,fjc->fpc", rows[k], Y) for k in range(1, 6)]

    def _energy(self, g, r, alpha):
        """Energy per surface of one group of faces."""
        _, w, dudv, (_, _, g0, rr0, lip, job, kc) = g
        _, _, (Ru, Rv, uu, uv, vv) = self._points(g, r, alpha)
        m = torch.linalg.cross(Ru, Rv)
        W = (m * m).sum(-1)
        E11, E12, E22 = (Ru * Ru).sum(-1), (Ru * Rv).sum(-1), (Rv * Rv).sum(-1)
        l, k, n = (m * uu).sum(-1), (m * uv).sum(-1), (m * vv).sum(-1)
        A = W.sqrt()
        H = -(l * E22 - 2 * k * E12 + n * E11) / (W * A)
        o, oc, occ, i, ic, icc = (lip[:, q, None] for q in range(6))
        bend = 0.25 * kc[:, None] * w * ((o * H - 2 * oc) * H + occ + (i * H + 2 * ic) * H + icc)
        e = bend + dudv * w * self.KA * (A - g0) ** 2 / g0
        if self.kg:
            e = e + dudv * g0 * w * self.kg * ((l * n - k * k) / W ** 2 - 0.25e-12)
        if self.k_reg:
            e = e + self.k_reg * (E12 / (E11 * E22).sqrt() - rr0) ** 2
        return torch.zeros(self.n, dtype=torch.float64, device=r.device).index_add(0, job, e.sum(1))

    def area_volume(self, r, alpha):
        A = V = 0.0
        for g in self.groups:
            X0, Y, (Ru, Rv, *_q) = self._points(g, r, alpha)
            R = X0[:, None] + torch.einsum("pj,fjc->fpc", g[0][0], Y)
            m, c = torch.linalg.cross(Ru, Rv), g[2] * g[1]
            A = A + (c * m.norm(dim=-1)).sum()
            V = V + (c * (R * m).sum(-1)).sum() / 3
        return A, V

    def energy_grad(self, r, alpha, restraint=None):
        """(E per surface, dE/dr, dE/dalpha) at r [nv, 3], alpha [surfaces, 3]."""
        r, alpha = r.detach().requires_grad_(), alpha.detach().requires_grad_()
        E = torch.zeros(self.n, dtype=torch.float64, device=r.device)
        for g in self.groups:
            e = self._energy(g, r, alpha)
            e.sum().backward()
            E += e.detach()
        if restraint is not None:
            KAr, A0, KV, V0 = restraint
            A, V = self.area_volume(r, alpha)
            e = 0.5 * KAr * (A - A0) ** 2 / A0 + 0.5 * KV * (V - V0) ** 2
            e.backward()
            E += e.detach()
        return E, r.grad, alpha.grad


def _philox(v, step, stream, seed):
    """Philox4x32-10 of counters (v, step, 0, stream) and key (seed, 0): four words per vertex."""
    c = [v.astype(np.uint64), np.full(v.shape, step, np.uint64), np.zeros(v.shape, np.uint64), stream.astype(np.uint64)]
    k0, k1, low = seed & 0xFFFFFFFF, seed >> 32, np.uint64(0xFFFFFFFF)
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & low, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & low]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _normals(v, step, stream, seed, wide):
    """Three Box-Muller normals per vertex: from 53-bit uniforms of two draws (wide), else from 24-bit ones of one."""
    sh = np.uint64
    o = _philox(v, step, stream, seed)
    if wide:
        def u53(a, b):
            return (((a >> sh(5)) << sh(26)) | (b >> sh(6))).astype(float) * 2.0 ** -53 + 2.0 ** -54
        q = _philox(v, step, stream | np.uint32(0x80000000), seed)
        u = [u53(o[0], o[1]), u53(o[2], o[3]), u53(q[0], q[1]), u53(q[2], q[3])]
    else:
        u = [((x >> sh(8)).astype(float) + 0.5) / 16777216.0 for x in o]
    a, b = np.sqrt(-2.0 * np.log(u[0])), np.sqrt(-2.0 * np.log(u[2]))
    return np.stack([a * np.cos(2 * np.pi * u[1]), a * np.sin(2 * np.pi * u[1]), b * np.cos(2 * np.pi * u[3])], 1)


def _trajectory(case, S, r, alpha, it, streams, vertex, minv=None, first=0):
    """(energies [steps, surfaces], r, p) after case["steps"] steps from r at rest, the noise from step `first` on."""
    dev = r.device
    AK, D, dt = it.time_step / AKMA_S, it.D, it.time_step
    mass = case.get("kind") == "ld_mass"
    wide = case["fp64"] or mass
    p, E = torch.zeros_like(r), []
    for k in range(first, first + case["steps"]):
        e, g, _ = S.energy_grad(r, alpha)
        E.append(e)
        xi = torch.from_numpy(_normals(vertex, k, streams, 17, wide)).to(dev)
        if it.kind == U.OVERDAMPED_BD:
            r = r - D * dt / KT * g + math.sqrt(2 * D * dt) * xi
        else:
            p = p - it.gamma * AK * p - g * AK + math.sqrt(2 * it.gamma * KT * AK) * xi
            r = r + AK * (minv @ p if mass else p)
    return torch.stack(E), r, p


def _tensor(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(_device())


def exact(case, seed):
    if case["op"] == "mass":
        st = prepare(case, seed)
        minv, x = _tensor(st["mesh"].mass_get()), st["x"]
        x = _tensor(x) if case["host"] else x
        return 0.5 * (minv @ x.view(-1, 3)).reshape(-1)
    if case["op"] == "batch":
        plans = _plans(case, seed)
        S = _Surfaces(plans)
        rs = [_state(case, plan, seed * 1013 + k) for k, (plan, _) in enumerate(plans)]
        r = _tensor(np.concatenate([x[:-3].reshape(-1, 3) for x in rs]))
        alpha = torch.ones(len(rs), 3, dtype=torch.float64, device=r.device)
        vertex = np.concatenate([np.arange(p.nv) for p, _ in plans])
        streams = np.repeat(np.arange(len(plans)), [p.nv for p, _ in plans]).astype(np.uint32)
        # the batch has taken case["steps"] steps by the first pass, which starts from r_in with the noise after them
        E, r, _ = _trajectory(case, S, r, alpha, _integrator(case), streams, vertex, first=case["steps"])
        out = [torch.cat([r[S.off[j]:S.off[j + 1]].reshape(-1), alpha[j]]) for j in range(S.n)]
        return {"r": torch.cat(out), "E": E[-1]}
    if case["op"] == "run":
        minv = it = None
        if case["kind"] == "ld_mass":
            st = prepare(case, seed)
            plans, it, minv = st["plans"], st["it"], _tensor(st["mesh"].mass_get())
        else:
            plans = _plans(case, seed)
            it = _integrator(case)
        plan = plans[0][0]
        S, r0 = _Surfaces(plans), _state(case, plan, seed)
        r = _tensor(r0[:-3].reshape(-1, 3))
        alpha = torch.ones(1, 3, dtype=torch.float64, device=r.device)
        E, r, p = _trajectory(case, S, r, alpha, it, np.full(plan.nv, 1, np.uint32), np.arange(plan.nv), minv)
        got = {"E": E[:, 0], "r": torch.cat([r.reshape(-1), alpha[0]])}
        return got if case["kind"] == "bd" else got | {"p": p.reshape(-1)}
    plans = _plans(case, seed)
    S, r0 = _Surfaces(plans), _state(case, plans[0][0], seed)
    r, alpha = _tensor(r0[:-3].reshape(-1, 3)), _tensor(r0[None, -3:])
    restraint = None
    if case["restrained"]:
        with torch.no_grad():
            A0, V0 = S.area_volume(_tensor(plans[0][0].positions()[:-3].reshape(-1, 3)), alpha)
        restraint = (0.2, A0, 0.01, V0)
    E, g, ga = S.energy_grad(r, alpha, restraint)
    return {"E": E[0] if case["host"] else E, "g": torch.cat([g.reshape(-1), ga[0]])}
