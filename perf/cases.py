"""Performance cases of the solver: what a program that uses this library has it do.

A case is one workload through a public entry point:

* ``step``    -- a solver handle advances its state by CFL steps (``Solver.step``)
                 and hands the new state to a device tensor;
* ``rhs``     -- one right-hand side on device fields (``Solver.rhs_device``), as a
                 program with its own time integrator calls it;
* ``adjoint`` -- ``adjoint.evolve`` forward and backward: the state at T and the
                 gradient of a final-time misfit with respect to the initial state;
* ``batch``   -- many independent advection meshes advanced together
                 (``BatchSolver``).

Meshes are periodic boxes of nx x ny x nz cells, six tetrahedra each; the states
are smooth, seeded fields (and seeded advection velocities).  Meshes depend on
the sizes alone and are built once per process; the handle, its upload and the
state are made by ``prepare``.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from exadglm_b200 import adjoint, capi
from exadglm_b200.mesh import Mesh3D, UniformBox
from exadglm_b200.problem import Problem, advection_gaussian

GAMMA = 1.4
TAU_SCALE = 1.2
CFL = {"euler": 0.4, "advection": 0.5}
RKA = (0.0, -567301805773 / 1357537059087, -2404267990393 / 2016746695238,
       -3550918686646 / 2091501179385, -1275806237668 / 842570457699)
RKB = (1432997174477 / 9575080441755, 5161836677717 / 13612068292357,
       1720146321549 / 2090206949498, 3134564353537 / 4481467310338,
       2277821191437 / 14882151754819)


def np_of(N):
    return (N + 1) * (N + 2) * (N + 3) // 6


def nfp_of(N):
    return (N + 1) * (N + 2) // 2


def _step(name, physics, N, n, steps=1, precision="fp64"):
    return {"name": name, "kind": "step", "physics": physics, "N": N, "nx": n[0], "ny": n[1],
            "nz": n[2], "precision": precision, "steps": steps}


def listed():
    return [
        # the benchmark workload: one time step of a production-size Euler run
        _step("euler_n4_k196608", "euler", 4, (32, 32, 32)),
        # the same run in the split-TF32 mode
        _step("euler_n4_tf32_k196608", "euler", 4, (32, 32, 32), precision="tf32x3"),
        # the precision study's order: a high-order Euler run, FP64 and split BF16
        _step("euler_n6_k82944", "euler", 6, (24, 24, 24)),
        _step("euler_n6_bf16_k82944", "euler", 6, (24, 24, 24), precision="bf16x3"),
        # a lower order on a box with unequal sides
        _step("euler_n3_k110970", "euler", 3, (27, 25, 27), steps=2),
        # the notebooks' order on their own small mesh: an interactive run
        _step("euler_n5_k1296", "euler", 5, (6, 6, 6), steps=10),
        # linear advection on the smallest configured mesh: launches and latency
        _step("advection_n3_k3072", "advection", 3, (8, 8, 8), steps=20),
        # linear advection at the notebooks' order, production size, odd sides
        _step("advection_n5_k93750", "advection", 5, (25, 25, 25), steps=2),
        # a caller's own time integrator asking for a right-hand side
        {"name": "rhs_euler_n4_k25194", "kind": "rhs", "physics": "euler", "N": 4, "nx": 19,
         "ny": 17, "nz": 13, "precision": "fp64"},
        # gradient of a final-time misfit on the gradient-check mesh
        {"name": "adjoint_euler_n4_k24576", "kind": "adjoint", "N": 4, "nx": 16, "ny": 16,
         "nz": 16, "steps": 6, "every": 3},
        # an ensemble of small advection problems of mixed size and order
        {"name": "batch_48", "kind": "batch", "count": 48, "nmin": 4, "nmax": 12, "steps": 5},
    ]


def _box(rng, K):
    """Cells per side of a box of about K tetrahedra with unequal, often odd sides."""
    c = max(2.0, (K / 6) ** (1 / 3))
    s = [max(2, int(round(c * rng.uniform(0.75, 1.3)))) for _ in range(2)]
    return s[0], s[1], max(2, int(round(K / 6 / (s[0] * s[1]))))


def draw(rng):
    kind = rng.choice(["step"] * 5 + ["mixed"] + ["rhs"] + ["adjoint"] + ["batch"])
    if kind == "batch":
        nmax = rng.randint(5, 12)
        return {"kind": "batch", "count": rng.randint(8, 48), "nmin": rng.randint(2, nmax - 2),
                "nmax": nmax, "steps": rng.randint(1, 5)}
    if kind == "adjoint":
        nx, ny, nz = _box(rng, math.exp(rng.uniform(math.log(200), math.log(24000))))
        steps = rng.randint(2, 6)
        return {"kind": "adjoint", "N": rng.randint(2, 4), "nx": nx, "ny": ny, "nz": nz,
                "steps": steps, "every": rng.randint(1, steps)}
    physics = "euler" if kind == "mixed" else rng.choice(["euler", "euler", "advection"])
    N = rng.randint(4, 6) if kind == "mixed" else rng.randint(2, 6)
    nvar = 5 if physics == "euler" else 1
    kmax = min(190000.0, 2.4e7 / (nvar * np_of(N)))
    nx, ny, nz = _box(rng, math.exp(rng.uniform(math.log(200), math.log(kmax))))
    c = {"kind": "rhs" if kind == "rhs" else "step", "physics": physics, "N": N, "nx": nx,
         "ny": ny, "nz": nz,
         "precision": rng.choice(["tf32x3", "bf16x3"]) if kind == "mixed" else "fp64"}
    if c["kind"] == "step":
        small = nx * ny * nz < 2000
        c["steps"] = rng.randint(1, 20) if small else 1
    return c


# ---------------------------------------------------------------- inputs


@functools.lru_cache(maxsize=None)
def _mesh(N, nx, ny, nz):
    return Mesh3D(N, UniformBox(nx + 1, ny + 1, nz + 1), high_order=False)


def _problem(physics, N, nx, ny, nz, seed):
    """A Problem with smooth fields of seeded phases and amplitudes."""
    mesh = _mesh(N, nx, ny, nz)
    rng = np.random.default_rng(seed)
    x, y, z = (torch.from_numpy(p).cuda().view(-1) for p in (mesh.PX, mesh.PY, mesh.PZ))

    def wave(amplitude):
        k = rng.integers(-2, 3, 3).tolist()
        return amplitude * torch.sin(
            2 * math.pi * (k[0] * x + k[1] * y + k[2] * z + rng.uniform()))

    if physics == "euler":
        rho = 1.0 + wave(0.2) + wave(0.05)
        v = [c + wave(0.1) for c in rng.uniform(-1.0, 1.0, 3).tolist()]
        p = 1.0 + wave(0.1)
        u0 = torch.stack([rho, rho * v[0], rho * v[1], rho * v[2], p / (GAMMA - 1) +
                          0.5 * rho * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2)]).cpu().numpy()
        vel = None
    else:
        u0 = (wave(0.5) + wave(0.5) + wave(0.25))[None, :].cpu().numpy()
        vel = np.broadcast_to(rng.uniform(-1.0, 1.0, 3)[:, None], (3, x.numel()))
    return Problem(physics, N, mesh, u0, vel, cfl=CFL[physics], gamma=GAMMA,
                   tau_scale=TAU_SCALE, tmax=1e6)


def _batch_problems(case, seed):
    """Advection instances whose sizes and orders (2..6) follow from the case, and
    whose velocities, centres and widths follow from the seed."""
    sizes, rng = np.random.default_rng(case["count"]), np.random.default_rng(seed)
    out = []
    for _ in range(case["count"]):
        n, N = int(sizes.integers(case["nmin"], case["nmax"] + 1)), int(sizes.integers(2, 7))
        out.append(advection_gaussian(n, N, v=rng.uniform(-1.0, 1.0, 3),
                                      center=rng.uniform(0.2, 0.8, 3),
                                      width2=float(rng.uniform(0.05, 0.2)) ** 2,
                                      tmax=1e6, mesh=_mesh(N, n, n, n)))
    return out


def _case_problem(case, seed):
    return _problem(case.get("physics", "euler"), case["N"], case["nx"], case["ny"], case["nz"],
                    seed)


def _target(p):
    """Density target of the misfit: the initial density shifted by a constant."""
    return p.u0[0] * 0.95


def _rows(t):
    return [r.data_ptr() for r in t]


def prepare(case, seed):
    if case["kind"] == "batch":
        problems = _batch_problems(case, seed)
        b = capi.BatchSolver(problems)
        out = [torch.empty(p.K * p.Np, dtype=torch.float64, device="cuda") for p in problems]
        return {"kind": "batch", "batch": b, "steps": case["steps"], "out": out}
    p = _case_problem(case, seed)
    s = {"kind": case["kind"], "solver": capi.Solver(p, precision=case.get("precision", "fp64")),
         "u": torch.from_numpy(p.u0).cuda()}
    if case["kind"] == "adjoint":
        s.update(steps=case["steps"], every=case["every"],
                 target=torch.from_numpy(_target(p)).cuda())
    else:
        s.update(steps=case.get("steps", 0), out=torch.empty_like(s["u"]))
    return s


def run(state):
    kind = state["kind"]
    if kind == "step":
        state["solver"].step(state["steps"])
        state["solver"].get_state_device(_rows(state["out"]))
        return state["out"]
    if kind == "rhs":
        state["solver"].rhs_device(_rows(state["u"]), _rows(state["out"]))
        return state["out"]
    if kind == "adjoint":
        u0 = state["u"].detach().requires_grad_(True)
        uT = adjoint.evolve(u0, state["solver"], state["steps"], checkpoint_every=state["every"])
        adjoint.density_misfit(uT, state["target"]).backward()
        return {"uT": uT.detach(), "grad": u0.grad}
    b = state["batch"]
    b.step(state["steps"])
    for i, o in enumerate(state["out"]):
        capi.check(b.L.dglm_batch_get_state(b.h, i, o.data_ptr(), 1))
    # the instances end to end, in one array
    return torch.cat(state["out"])


# ---------------------------------------------------------------- work


def _stage_work(physics, N, K):
    """Bytes and operations of one Runge-Kutta stage: state and register read and
    written, the geometry, the face penalty and the neighbour map read; the four
    dense operator applications."""
    nv = 5 if physics == "euler" else 1
    Np, Nfp = np_of(N), nfp_of(N)
    per = 4 * nv * Np * 8 + 29 * 8 + 16 * Nfp + (0 if physics == "euler" else 3 * Np * 8)
    return K * per, K * nv * (6 * Np * Np + 8 * Np * Nfp)


def work(case):
    if case["kind"] == "batch":
        b = f = 0
        for p in _batch_problems(case, 0):
            # the velocity of an instance is three numbers
            x, y = _stage_work("advection", p.N, p.K)
            b, f = b + x - p.K * p.Np * 24, f + y
        return {"bytes": 5 * case["steps"] * b, "flops": 5 * case["steps"] * f}
    physics = case.get("physics", "euler")
    K, Np = 6 * case["nx"] * case["ny"] * case["nz"], np_of(case["N"])
    b, f = _stage_work(physics, case["N"], K)
    if case["kind"] == "rhs":
        # no register: state in, right-hand side out
        return {"bytes": b - K * (5 if physics == "euler" else 1) * Np * 16, "flops": f}
    if case["kind"] == "adjoint":
        # forward, and per reverse stage the adjoint pair and the stage's input state
        back = K * (5 * 5 * Np * 8 + 29 * 8 + 16 * nfp_of(case["N"]))
        return {"bytes": 5 * case["steps"] * (b + back), "flops": 2 * 5 * case["steps"] * f}
    return {"bytes": 5 * case["steps"] * b, "flops": 5 * case["steps"] * f}


# ---------------------------------------------------------------- 64-bit values


class _Plain:
    """The scheme in plain torch float64: one element per row, fields (nvar, K, Np)."""

    def __init__(self, p):
        def dev(a, dtype=torch.float64):
            return torch.as_tensor(np.ascontiguousarray(a), device="cuda").to(dtype)

        m, ref = p.mesh, p.mesh.ref
        self.p, self.K, self.Np, self.Nfp, self.nv = p, p.K, p.Np, p.Nfp, p.nvar
        self.W = [dev(getattr(ref, n)).T.contiguous() for n in ("WDr", "WDs", "WDt")]
        self.L = dev(ref.LIFT).T.contiguous()
        self.geo = [[dev(getattr(m, d + q)).view(-1, 1) for q in "xyz"] for d in "rst"]
        self.n = [dev(a).view(-1, 4, 1) for a in (m.NX, m.NY, m.NZ)]
        self.fs = dev(m.Fscale).view(-1, 4, 1)
        self.fm = dev(ref.Fmask, torch.int64).view(-1)
        self.vmapP = dev(m.vmapP, torch.int64).view(-1)
        self.vmapF = dev(m.vmapF, torch.int64).view(-1)
        self.v = None if p.vel is None else dev(p.vel).view(3, self.K, self.Np)

    def trace(self, a):
        return a[:, self.fm].view(self.K, 4, self.Nfp)

    def flux(self, u, at_faces=False):
        """Physical fluxes F, G, W, each a list over the variables."""
        if self.v is not None:
            return [[(self.trace(c) if at_faces else c) * u[0]] for c in self.v]
        r, E = u[0], u[4]
        w = [u[i] / r for i in (1, 2, 3)]
        p = (self.p.gamma - 1) * (E - 0.5 * (u[1] * w[0] + u[2] * w[1] + u[3] * w[2]))
        out = []
        for d in range(3):
            f = [u[1 + d]] + [u[1 + i] * w[d] for i in range(3)] + [(E + p) * w[d]]
            f[1 + d] = f[1 + d] + p
            out.append(f)
        return out

    def maxv(self, u):
        if self.v is not None:
            v2 = self.trace(sum(c * c for c in self.v))
            return v2.amax(2).sqrt()
        t = [self.trace(a) for a in u]
        v2 = (t[1] ** 2 + t[2] ** 2 + t[3] ** 2) / t[0] ** 2
        pr = (self.p.gamma - 1) * (t[4] - 0.5 * t[0] * v2)
        return v2.amax(2).sqrt() + (self.p.gamma * pr / t[0]).abs().amax(2).sqrt()

    def tau(self, mv):
        return (0.25 * (mv.view(-1) + mv.view(-1)[self.vmapF]) * self.p.tau_scale).view(-1, 4, 1)

    def dt(self, mv):
        return float(self.p.cfl / (2 * self.p.N + 1) / (mv * self.fs[:, :, 0]).max())

    def rhs(self, u, tau):
        u = list(u)
        F = self.flux(u)
        um = [self.trace(a) for a in u]
        ub = [0.5 * (a + b.reshape(-1)[self.vmapP].view(self.K, 4, self.Nfp))
              for a, b in zip(um, u)]
        B = self.flux(ub, at_faces=True)
        out = []
        for q in range(self.nv):
            r = 0
            for g, W in zip(self.geo, self.W):
                r = r + (g[0] * F[0][q] + g[1] * F[1][q] + g[2] * F[2][q]) @ W
            nf = self.n[0] * B[0][q] + self.n[1] * B[1][q] + self.n[2] * B[2][q]
            out.append(r - ((nf - tau * (ub[q] - um[q])) * self.fs).reshape(self.K, -1) @ self.L)
        return torch.stack(out)

    def steps(self, u, n):
        for _ in range(n):
            with torch.no_grad():
                mv = self.maxv(u.detach())
                tau, dt = self.tau(mv), self.dt(mv)
            k = 0
            for a, b in zip(RKA, RKB):
                k = a * k + dt * self.rhs(u, tau)
                u = u + b * k
        return u


def exact(case, seed):
    if case["kind"] == "batch":
        got = []
        for p in _batch_problems(case, seed):
            s = _Plain(p)
            u = torch.as_tensor(p.u0, device="cuda").view(1, p.K, p.Np)
            got.append(s.steps(u, case["steps"]).reshape(-1))
        return torch.cat(got)
    p = _case_problem(case, seed)
    s = _Plain(p)
    u = torch.as_tensor(p.u0, device="cuda").view(p.nvar, p.K, p.Np)
    if case["kind"] == "rhs":
        return s.rhs(u, s.tau(s.maxv(u))).view(p.nvar, -1)
    if case["kind"] == "step":
        return s.steps(u, case["steps"]).view(p.nvar, -1)
    u = u.clone().requires_grad_(True)
    uT = s.steps(u, case["steps"])
    d = uT[0] - torch.as_tensor(_target(p), device="cuda").view(p.K, p.Np)
    (0.5 * (d * d).sum()).backward()
    return {"uT": uT.detach().view(p.nvar, -1), "grad": u.grad.view(p.nvar, -1)}
