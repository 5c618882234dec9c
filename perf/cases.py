"""The solver's workloads as measurable cases: inputs, one pass through the public entry points, the
work a pass cannot do without, and its result in 64 bits.

Four kinds of pass, each what a program that uses the library does in its loop:
  frame    one vbd_solver_step (VBDsolver::step) and the new positions and velocities, read into
           tensors on the GPU; with `energy_every`, the energy history VBDsolver::step fills as well
  batch    the same for many independent meshes in one solver (vbd_solver_init_batch)
  train    one iteration of a material fit: new per-tet materials, the initial state, recorded steps,
           the loss gradient on the host, the backward pass with its gradients
  wrapper  one VBD_GPU_Solver frame of the reference's driver: the inertial target from host memory,
           solveVBD with that solver's own arithmetic, the positions back to host memory
"""
from __future__ import annotations

import math

import numpy as np
import torch

from vbd_tetmesh_b200 import _capi, build_batch_solver, build_solver, meshgen
from vbd_tetmesh_b200.material_id import beams

GRAVITY = (0.0, -9.8, 0.0)


def _frame(name, lx, ly, lz, **kw):
    c = dict(kind="frame", lx=lx, ly=ly, lz=lz, cell=0.05, jitter=0.2, E=1e5, nu=0.3, sigma=0.0, pin="x0", vel=0.1,
             dt=1.0 / 60.0, substeps=1, iterations=20, accel=True, rho=0.9, energy_every=0, walk=0)
    c.update(kw)
    return dict(c, name=name) if name else c


def _cube(name, n):
    """The benchmark's cube (unit cube, E = 1e6, nu = 0.4, bottom face pinned) of n^3 cells."""
    return _frame(name, n, n, n, cell=1.0 / n, E=1e6, nu=0.4, pin="y0", vel=0.5, dt=1.0 / 120.0, iterations=50)


def listed():
    return [
        # the smallest simulation in use: the reference's CPU-sized beam, one frame of an interactive loop
        _frame("beam_frame", 16, 4, 4, jitter=0.0, rho=0.95),
        # the same beam with the single-cluster walk that the documentation names for small meshes
        _frame("beam_frame_walk", 16, 4, 4, jitter=0.0, rho=0.95, walk=2),
        # a small ragged block, per-tet materials, sub-stepped, without acceleration
        _frame("block_substeps", 13, 7, 5, sigma=0.2, pin="z1", substeps=2, iterations=15, accel=False),
        # a character-sized body (4,913 vertices)
        _cube("cube16_frame", 16),
        # a mid-sized block with the energy history that VBDsolver::step keeps every 10 iterations
        _frame("block_monitored", 40, 21, 19, iterations=30, energy_every=10),
        # a scene-sized body (35,937 vertices)
        _cube("cube32_frame", 32),
        # the benchmark's workload (274,625 vertices, 1,572,864 tets)
        _cube("cube64_frame", 64),
        # many independent bodies at once: the batched configuration's distribution, 128 meshes
        dict(name="batch128_frame", kind="batch", meshes=128, lo=4, hi=24, dt=1.0 / 60.0, iterations=20, rho=0.9),
        # differentiable simulation of one body with per-tet materials, by the single-cluster walk
        dict(name="train_beam", kind="train", meshes=0, lx=32, ly=8, lz=8, sigma=0.2, steps=6, checkpoint=3,
             iterations=30, adjoint_iterations=50, rho=0.95, walk=2),
        # the material identification's batch of 64 beams, one loss-and-gradient evaluation
        dict(name="train_batch", kind="train", meshes=64, lx=0, ly=0, lz=0, sigma=0.0, steps=4, checkpoint=2,
             iterations=100, adjoint_iterations=50, rho=0.95, walk=0),
        # the reference driver's GPU loop on host buffers, a small and an ordinary body
        dict(name="wrapper_beam", kind="wrapper", lx=16, ly=4, lz=4, cell=0.05, E=1e5, nu=0.3, dt=1.0 / 60.0,
             iterations=20, rho=0.95),
        dict(name="wrapper_cube32", kind="wrapper", lx=32, ly=32, lz=32, cell=1.0 / 32.0, E=1e6, nu=0.4,
             dt=1.0 / 120.0, iterations=50, rho=0.9),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("frame", "frame", "frame", "frame", "batch", "train", "train", "wrapper"))
    E, nu = 10.0 ** rng.uniform(4.0, 6.0), rng.uniform(0.2, 0.45)
    if kind == "batch":
        return dict(kind=kind, meshes=_log_int(rng, 4, 120), lo=rng.randint(2, 6), hi=rng.randint(8, 24), dt=1.0 / 60.0,
                    iterations=rng.choice((10, 20, 30)), rho=0.9)
    if kind == "train":
        many = rng.random() < 0.5
        return dict(kind=kind, meshes=_log_int(rng, 2, 64) if many else 0, lx=0 if many else rng.randint(8, 40),
                    ly=0 if many else rng.randint(3, 8), lz=0 if many else rng.randint(3, 8), sigma=0.0 if many else 0.2,
                    steps=rng.randint(2, 5), checkpoint=rng.randint(1, 3), iterations=rng.choice((20, 30, 60)),
                    adjoint_iterations=rng.choice((25, 50)), rho=rng.choice((0.9, 0.95)),
                    walk=0 if many else rng.choice((0, 2)))
    # cells spread over their logarithm, from the beam's number to the 64^3 cube's, in ragged shapes
    cells = math.exp(rng.uniform(math.log(150.0), math.log(262144.0 if kind == "frame" else 32768.0)))
    lx = max(3, min(96, int(cells ** (1.0 / 3.0) * math.exp(rng.uniform(-0.6, 0.6)))))
    ly = max(3, min(96, int(math.sqrt(cells / lx) * math.exp(rng.uniform(-0.4, 0.4)))))
    lz = max(2, min(96, int(cells / (lx * ly))))
    if kind == "wrapper":
        return dict(kind=kind, lx=lx, ly=ly, lz=lz, cell=0.05, E=E, nu=nu, dt=1.0 / 60.0,
                    iterations=rng.choice((10, 20, 50)), rho=0.9)
    small = (lx + 1) * (ly + 1) * (lz + 1) <= 4000
    return _frame(None, lx, ly, lz, E=E, nu=nu, sigma=rng.choice((0.0, 0.2)), jitter=rng.choice((0.0, 0.2)),
                  pin=rng.choice(("x0", "x1", "y0", "y1", "z0", "z1")), dt=rng.choice((1.0 / 60.0, 1.0 / 120.0)),
                  substeps=rng.choice((1, 1, 2)), iterations=rng.choice((10, 20, 25)), accel=rng.random() < 0.75,
                  energy_every=rng.choice((0, 0, 10)), walk=rng.choice((0, 2)) if small else 0)


def _meshes(case, seed):
    """The case's meshes with their initial velocities.  A batch's shapes and materials are those of the
    repository's configurations (their own seeds); everything else comes from the seed."""
    rng = np.random.default_rng(seed)
    if case["kind"] == "batch":
        ms = meshgen.batched_blocks(case["meshes"], lo=case["lo"], hi=case["hi"])
        for m in ms:
            m.v[m.fixed == 0] = rng.normal(0.0, 0.1, (int((m.fixed == 0).sum()), 3))
        return ms
    if case["kind"] == "train" and case["meshes"]:
        return beams(case["meshes"])[0]
    if case["kind"] in ("train", "wrapper"):
        c = _frame(None, case["lx"], case["ly"], case["lz"], sigma=case.get("sigma", 0.0), cell=case.get("cell", 0.05),
                   E=case.get("E", 1e5), nu=case.get("nu", 0.3), jitter=0.0 if case["kind"] == "train" else 0.2)
    else:
        c = case
    m = meshgen.jittered_block(c["lx"], c["ly"], c["lz"], cell=c["cell"], jitter=c["jitter"], E=c["E"], nu=c["nu"],
                               seed=seed, pin_face=c["pin"], per_tet_sigma=c["sigma"])
    if case["kind"] != "train":
        m.v[m.fixed == 0] = rng.normal(0.0, c["vel"], (int((m.fixed == 0).sum()), 3))
    return [m]


def _inputs(case, seed):
    """The meshes and the arrays a pass reads besides them."""
    ms = _meshes(case, seed)
    rng = np.random.default_rng(seed + 1)
    extra = {}
    if case["kind"] == "train":
        n, t = sum(m.num_verts for m in ms), sum(m.num_tets for m in ms)
        rest = np.concatenate([m.rest for m in ms])
        extra["target"] = rest + rng.normal(0.0, 0.01, (n, 3)).astype(np.float32)
        scale = np.exp(rng.normal(0.0, 0.1, t)).astype(np.float32)
        extra["mu"] = np.concatenate([m.mu for m in ms]) * scale
        extra["lam"] = np.concatenate([m.lam for m in ms]) * scale
    elif case["kind"] == "wrapper":
        m = ms[0]
        y = m.x + np.float32(case["dt"]) * m.v + rng.normal(0.0, 1e-3, m.x.shape).astype(np.float32)
        y[m.fixed != 0] = m.x[m.fixed != 0]
        extra["y"] = y.astype(np.float32)
    return ms, extra


def prepare(case, seed):
    ms, extra = _inputs(case, seed)
    batch = case["kind"] == "batch" or case.get("meshes", 0) > 0
    b = meshgen.concat(ms)
    s = build_batch_solver(b) if batch else build_solver(ms[0])
    if case.get("walk"):
        s.set_option(_capi.OPT_PERSISTENT, case["walk"])
    if case.get("energy_every"):
        s.set_option(_capi.OPT_ENERGY_EVERY, case["energy_every"])
    if case["kind"] == "wrapper":
        s.set_option(_capi.OPT_SEMANTICS, _capi.SEMANTICS_GPU_WRAPPER)
    st = dict(case=case, solver=s, rest=b.rest, zero=np.zeros_like(b.rest), **extra)
    if case["kind"] in ("frame", "batch"):
        st["x"] = torch.empty(s.num_verts, 3, device="cuda")
        st["v"] = torch.empty(s.num_verts, 3, device="cuda")
    return st


def run(state):
    c, s = state["case"], state["solver"]
    if c["kind"] in ("frame", "batch"):
        s.step(c["dt"], c["iterations"], GRAVITY, c.get("accel", True), c["rho"], c.get("substeps", 1))
        s.get_positions(state["x"].data_ptr())
        s.get_velocities(state["v"].data_ptr())
        out = {"x": state["x"], "v": state["v"]}
        if c.get("energy_every"):
            out["energy"] = s.energy_history()
        return out
    if c["kind"] == "wrapper":
        s.update_inertia_from_cpu(state["y"])
        s.solve_vbd(c["iterations"], 1.0 / (c["dt"] * c["dt"]), True, c["rho"], _capi.INIT_FROM_INERTIA)
        return {"x": s.get_positions()}
    s.set_materials(state["mu"], state["lam"])
    s.set_positions(state["rest"])
    s.set_velocities(state["zero"])
    s.record(c["checkpoint"])
    for _ in range(c["steps"]):
        s.step(1.0 / 60.0, c["iterations"], GRAVITY, True, c["rho"])
    x = s.get_positions()
    gx, gv, gmu, glam = s.backward(2.0 * (x - state["target"]), None, c["adjoint_iterations"], c["rho"])
    return {"x": x, "gx": gx, "gv": gv, "gmu": gmu, "glam": glam}


def _sizes(case):
    """(vertices, tets) of the case; a batch's expected ones."""
    if case.get("meshes"):
        if case["kind"] == "batch":
            e = np.arange(case["lo"], case["hi"] + 1)
            return case["meshes"] * float(np.mean(e + 1.0)) ** 3, case["meshes"] * 6 * float(np.mean(e)) ** 3
        e, f = np.arange(3.0, 9.0), 24.0
        return case["meshes"] * (f + 1) * float(np.mean((e + 1) ** 2)), case["meshes"] * 6 * f * float(np.mean(e * e))
    lx, ly, lz = case["lx"], case["ly"], case["lz"]
    return (lx + 1) * (ly + 1) * (lz + 1), 6 * lx * ly * lz


def work(case):
    """Each tet's ids, Dm^-1, volume and materials and each vertex's state read once, the results
    written once; per iteration the element blocks of the four vertices of every tet (about 70
    operations each; about 140 in the adjoint, 450 in the corotated model) and one 3x3 solve a vertex."""
    n, t = _sizes(case)
    its = case["iterations"] * case.get("substeps", 1) * case.get("steps", 1)
    per_inc = 450.0 if case["kind"] == "wrapper" else 70.0
    flops = its * (4.0 * t * per_inc + 60.0 * n)
    nbytes = 64.0 * t + 28.0 * n + (12.0 if case["kind"] == "wrapper" else 24.0) * n
    if case["kind"] == "train":
        flops += case["adjoint_iterations"] * case["steps"] * (4.0 * t * 140.0 + 60.0 * n)
        nbytes += 16.0 * t + 24.0 * n
    return {"bytes": nbytes, "flops": flops}


# ---- the same passes in 64 bits, with plain torch operations --------------------------------------


def _greedy(n, tets):
    """Greedy vertex colouring in id order: the smallest colour no coloured neighbour holds."""
    pairs = np.concatenate([tets[:, [a, b]] for a in range(4) for b in range(4) if a > b]).astype(np.int64)
    hi, lo = pairs.max(1), pairs.min(1)
    key = np.unique(hi * n + lo)
    hi, lo = key // n, (key % n).tolist()
    off = np.searchsorted(hi, np.arange(n + 1)).tolist()
    colour = [0] * n
    for v in range(n):
        used = 0
        for u in lo[off[v]:off[v + 1]]:
            used |= 1 << colour[u]
        colour[v] = ((~used) & (used + 1)).bit_length() - 1
    return np.array(colour)


class _Exact:
    """The vertex block Gauss-Seidel on the concatenated meshes."""

    def __init__(self, ms, mu=None, lam=None, corotated=False):
        f8 = dict(dtype=torch.float64, device="cuda")
        off = np.cumsum([0] + [m.num_verts for m in ms])
        tets = np.concatenate([m.tets.astype(np.int64) + o for m, o in zip(ms, off)])
        self.n, self.corotated = int(off[-1]), corotated
        rest = torch.tensor(np.concatenate([m.rest for m in ms]), **f8)
        self.x = torch.tensor(np.concatenate([m.x for m in ms]), **f8)
        self.v = torch.tensor(np.concatenate([m.v for m in ms]), **f8)
        fixed = np.concatenate([m.fixed for m in ms]) != 0
        self.free = torch.tensor(~fixed, device="cuda")[:, None]
        self.mu = torch.tensor(np.concatenate([m.mu for m in ms]) if mu is None else mu, **f8)
        self.lam = torch.tensor(np.concatenate([m.lam for m in ms]) if lam is None else lam, **f8)
        self.tets = torch.tensor(tets, device="cuda")
        p = rest[self.tets]
        D = (p[:, 1:] - p[:, :1]).transpose(1, 2)
        self.V = torch.linalg.det(D).abs() / 6.0
        self.Dinv = torch.linalg.inv(D)
        self.Q = torch.cat([-self.Dinv.sum(1, keepdim=True), self.Dinv], 1)
        self.m = torch.zeros(self.n, **f8)
        rho_v = torch.tensor(np.concatenate([np.full(m.num_tets, m.density) for m in ms]), **f8) * self.V / 4.0
        for k in range(4):
            self.m.index_add_(0, self.tets[:, k], rho_v)
        colour = _greedy(self.n, tets)
        flat = tets.reshape(-1)
        self.sweeps = []
        for c in range(int(colour.max()) + 1):
            verts = np.flatnonzero((colour == c) & ~fixed)
            if not len(verts):
                continue
            slot = np.full(self.n, -1)
            slot[verts] = np.arange(len(verts))
            inc = np.flatnonzero(slot[flat] >= 0)
            g = lambda a: torch.tensor(a, device="cuda")  # noqa: E731
            self.sweeps.append((g(verts), g(inc // 4), g(inc % 4), g(slot[flat[inc]])))

    @staticmethod
    def mul(a, b):
        return (a[..., :, :, None] * b[..., None, :, :]).sum(-2)

    @staticmethod
    def cof(F):
        return torch.stack([torch.linalg.cross(F[:, 1], F[:, 2]), torch.linalg.cross(F[:, 2], F[:, 0]),
                            torch.linalg.cross(F[:, 0], F[:, 1])], 1)

    def kinematics(self, x, t):
        p = x[self.tets[t]]
        F = self.mul((p[:, 1:] - p[:, :1]).transpose(1, 2), self.Dinv[t])
        C = self.cof(F)
        return F, C, (F[:, 0] * C[:, 0]).sum(1)

    @staticmethod
    def solve3(H, f, guard):
        A = torch.stack([torch.linalg.cross(H[:, 1], H[:, 2]), torch.linalg.cross(H[:, 2], H[:, 0]),
                         torch.linalg.cross(H[:, 0], H[:, 1])], 2)
        det = (H[:, 0] * A[:, :, 0]).sum(1)
        ok = det.abs() > guard
        return torch.where(ok[:, None], (A * f[:, None, :]).sum(2) / torch.where(ok, det, 1.0)[:, None], 0.0)

    def block(self, x, t, n):
        """Gradient and diagonal block of tets t at their local vertices n."""
        F, C, J = self.kinematics(x, t)
        q, V, mu, lam = self.Q[t, n], self.V[t][:, None], self.mu[t][:, None], self.lam[t][:, None]
        qq = (q * q).sum(1)[:, None, None]
        eye = torch.eye(3, dtype=torch.float64, device="cuda")
        Fq = (F * q[:, None, :]).sum(2)
        if self.corotated:
            R = F.clone()
            for _ in range(5):
                CR = self.cof(R)
                det = (R[:, 0] * CR[:, 0]).sum(1)[:, None, None]
                R = torch.where(det.abs() < 1e-8, R, 0.5 * (R + CR / det))
            tr = ((R * F).sum((1, 2)) - 3.0)[:, None]
            Rq = (R * q[:, None, :]).sum(2)
            g = V * (2.0 * mu * (Fq - Rq) + lam * tr * Rq)
            return g, V[:, None] * (2.0 * mu[:, None] * qq * eye + lam[:, None] * Rq[:, :, None] * Rq[:, None, :])
        Cq = (C * q[:, None, :]).sum(2)
        g = V * (mu * (Fq - Cq) + lam * (J[:, None] - 1.0) * Cq)
        return g, V[:, None] * (mu[:, None] * qq * eye + lam[:, None] * Cq[:, :, None] * Cq[:, None, :])

    def omegas(self, iters, accel, rho):
        rho, w, out = float(np.float32(rho)), 1.0, []
        for k in range(1, iters + 1):
            w = 1.0 if k == 1 else (2.0 / (2.0 - rho * rho) if k == 2 else 4.0 / (4.0 - rho * rho * w))
            out.append(w if accel else 1.0)
        return out

    def iterate(self, x, y, dtsr, iters, accel, rho, each=None):
        reg = 1.000001 if self.corotated else 1.0
        eye = torch.eye(3, dtype=torch.float64, device="cuda")
        pp = x.clone()
        for k, w in enumerate(self.omegas(iters, accel, rho)):
            before = x.clone()
            for verts, t, n, slot in self.sweeps:
                g, H = self.block(x, t, n)
                cm = (self.m[verts] * dtsr)[:, None]
                f = (cm * (y[verts] - x[verts])).index_add_(0, slot, g, alpha=-1.0)
                A = (cm[:, None] * reg * eye).index_add_(0, slot, H)
                x[verts] += self.solve3(A, f, 1e-8)
            if w > 1.0:
                x = torch.where(self.free, w * (x - pp) + pp, x)
            pp = before
            if each:
                each(k, x)
        return x

    def energy(self, x):
        F, _, J = self.kinematics(x, slice(None))
        lj = torch.log(J.abs())
        return float((self.V * (0.5 * self.mu * ((F * F).sum((1, 2)) - 3.0) - self.mu * lj + 0.5 * self.lam * lj * lj)).sum())

    def step(self, dt, iters, accel, rho, substeps=1, energy_every=0, energies=None):
        h = float(np.float32(np.float32(dt) / np.float32(substeps)))
        g = torch.tensor([float(np.float32(a)) for a in GRAVITY], dtype=torch.float64, device="cuda")
        each = (lambda k, x: energies.append(self.energy(x)) if k % energy_every == 0 else None) if energy_every else None
        for _ in range(substeps):
            prev = self.x.clone()
            self.v = torch.where(self.free, self.v + h * g, self.v)
            y = torch.where(self.free, prev + h * self.v, prev)
            self.x = self.iterate(self.x.clone(), y, 1.0 / (h * h), iters, accel, rho, each)
            self.v = torch.where(self.free, (self.x - prev) / h * 0.999, self.v)
        return h

    def adjoint(self, states, h, ax, sweeps, rho):
        """Gradients of the final positions' loss gradient ax through the steps that ended at `states`."""
        c, dtsr = 0.999 / h, 1.0 / (h * h)
        lam, lpp = torch.zeros_like(ax), torch.zeros_like(ax)
        av = torch.zeros_like(ax)
        gmu, glam = torch.zeros_like(self.mu), torch.zeros_like(self.lam)
        eye = torch.eye(3, dtype=torch.float64, device="cuda")

        def coupling(x, t, n, L):
            """V dP(sum over the other three vertices of lam q^T) q_n of tets t at local vertices n."""
            F, C, J = self.kinematics(x, t)
            l4 = L[self.tets[t]].clone()
            l4[torch.arange(len(n), device="cuda"), n] = 0.0
            dF = (l4[:, :, :, None] * self.Q[t][:, :, None, :]).sum(1)
            dC = torch.stack([torch.linalg.cross(dF[:, i], F[:, j]) + torch.linalg.cross(F[:, i], dF[:, j])
                              for i, j in ((1, 2), (2, 0), (0, 1))], 1)
            dJ = (C * dF).sum((1, 2))[:, None, None]
            mu, la, q = self.mu[t][:, None, None], self.lam[t][:, None, None], self.Q[t, n]
            dP = mu * (dF - dC) + la * (dJ * C + (J[:, None, None] - 1.0) * dC)
            return self.V[t][:, None] * (dP * q[:, None, :]).sum(2)

        pinned = torch.nonzero(~self.free[:, 0])[:, 0]
        at = torch.full((self.n,), -1, device="cuda")
        at[pinned] = torch.arange(len(pinned), device="cuda")
        inc = torch.nonzero(at[self.tets.reshape(-1)] >= 0)[:, 0]
        for x in reversed(states):
            G = torch.where(self.free, ax + c * av, 0.0)
            for w in self.omegas(sweeps, rho > 0.0, rho):
                before = lam.clone()
                for verts, t, n, slot in self.sweeps:
                    _, H = self.block(x, t, n)
                    A = ((self.m[verts] * dtsr)[:, None, None] * eye).index_add_(0, slot, H)
                    f = G[verts].index_add_(0, slot, coupling(x, t, n, lam), alpha=-1.0)
                    lam[verts] = self.solve3(A, f, 1e-30)
                if w > 1.0:
                    lam = w * (lam - lpp) + lpp
                lpp = before
            F, C, J = self.kinematics(x, slice(None))
            lt = lam[self.tets]
            Fq = (F[:, None] * self.Q[:, :, None, :]).sum(3)
            Cq = (C[:, None] * self.Q[:, :, None, :]).sum(3)
            gmu -= self.V * (lt * (Fq - Cq)).sum((1, 2))
            glam -= self.V * (J - 1.0) * (lt * Cq).sum((1, 2))
            if len(inc):
                ax = ax.index_add(0, self.tets.reshape(-1)[inc], coupling(x, inc // 4, inc % 4, lam), alpha=-1.0)
            yt = (self.m * dtsr)[:, None] * lam
            ax, av = torch.where(self.free, yt - c * av, ax), torch.where(self.free, h * yt, av)
        return ax, av, gmu, glam


def exact(case, seed):
    ms, extra = _inputs(case, seed)
    if case["kind"] == "wrapper":
        e = _Exact(ms, corotated=True)
        y = torch.tensor(extra["y"], dtype=torch.float64, device="cuda")
        dtsr = float(np.float32(1.0 / (case["dt"] * case["dt"])))
        return {"x": e.iterate(y.clone(), y, dtsr, case["iterations"], True, case["rho"])}
    if case["kind"] == "train":
        e = _Exact(ms, extra["mu"], extra["lam"])
        e.v.zero_()
        states = []
        for _ in range(case["steps"]):
            h = e.step(1.0 / 60.0, case["iterations"], True, case["rho"])
            states.append(e.x)
        ax = 2.0 * (e.x - torch.tensor(extra["target"], dtype=torch.float64, device="cuda"))
        rho = float(np.float32(case["rho"]))
        gx, gv, gmu, glam = e.adjoint(states, h, ax, case["adjoint_iterations"], rho)
        return {"x": e.x, "gx": gx, "gv": gv, "gmu": gmu, "glam": glam}
    e = _Exact(ms)
    energies = []
    e.step(case["dt"], case["iterations"], case.get("accel", True), case["rho"], case.get("substeps", 1),
           case.get("energy_every", 0), energies)
    out = {"x": e.x, "v": e.v}
    if case.get("energy_every"):
        out["energy"] = np.array(energies)
    return out
