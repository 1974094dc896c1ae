"""Timed cases of the framework's main paths, through its public Python entry points.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same ranges,
``prepare(case, seed)`` makes what a user's program holds before a call, ``run(state)`` is one
pass and returns its outputs, ``work(case)`` the bytes and operations a pass cannot do
without, ``exact(case, seed)`` the same outputs from plain torch in 64 bits.

All operators are the uniform lid-driven cavity's (``gip_b200.cavity``), the workload of this
repository's tests and benchmark.  Operators, solvers and engines are set up once per
configuration and kept, as a program that solves many right-hand sides or restarts many runs
on one mesh keeps them; what changes from state to state is the data: right-hand sides,
vectors, lid velocities.
"""
from __future__ import annotations

import collections
import math

import numpy as np
import torch

from gip_b200 import cavity
from gip_b200.adjoint import CavityAdjoint
from gip_b200.device import DeviceMatrix, DnsBatch, DnsEngine, PcgSolver, dns_params, host_loop_pcg
from gip_b200.formats import Csr

# At most this many set-up configurations are kept (the oldest goes first).
KEPT = 16
_kept: "collections.OrderedDict" = collections.OrderedDict()

# solver settings by name, as the benchmark and the tests use them
SOLVERS = {
    "fixed": dict(pcg_mode="fixed", maxit=100),                      # GIP's own: 100 iterations
    "tol": dict(pcg_mode="tol", maxit=20000, tol=1e-6),
    "mixed": dict(pcg_mode="mixed", maxit=20000, tol=1e-6, inner_tol=0.3, max_outer=400),
    "mixed_amg": dict(pcg_mode="mixed", maxit=20000, tol=1e-6, inner_tol=0.01, max_outer=400,
                      precond="amg"),
}
POISSON = {
    "tol": dict(mode="tol", maxit=20000, tol=1e-8),
    "mixed": dict(mode="mixed", maxit=20000, tol=1e-8, inner_tol=0.3, max_outer=400),
    "mixed_amg": dict(mode="mixed", maxit=20000, tol=1e-8, inner_tol=0.01, max_outer=400,
                      precond="amg"),
}


def listed():
    return [
        # one operator application on a small mesh (GIP_Matrix::spmv with alpha and beta, as the
        # drop-in's generic classes call it): latency
        {"name": "spmv_21", "kind": "spmv", "n": 21, "mode": 1},
        # the same on a large one, plain y = A x: the pressure operator of a 200^3 mesh
        {"name": "spmv_200", "kind": "spmv", "n": 200, "mode": 0},
        # GIP_LinearSolver's loop kept by the host over the fused entry points, 100 iterations,
        # at the size of GIP's shipped 97,521-cell mesh
        {"name": "host_loop_46", "kind": "host_loop", "n": 46, "iters": 100},
        # the pressure-Poisson benchmark, FP64 Jacobi-PCG to 1e-8
        {"name": "poisson_tol_128", "kind": "poisson", "n": 128, "solver": "tol"},
        # a smaller, odd-sized one in the mixed form with GIP's Jacobi
        {"name": "poisson_mixed_75", "kind": "poisson", "n": 75, "solver": "mixed"},
        # the pressure-Poisson benchmark in the mixed form with AMG
        {"name": "poisson_mixed_amg_128", "kind": "poisson", "n": 128, "solver": "mixed_amg"},
        # ten GIP timesteps (fixed 100 iterations) on a mesh of test size
        {"name": "steps_fixed_12", "kind": "steps", "n": 12, "re": 100.0, "solver": "fixed",
         "steps": 10, "permute": False},
        # the 48^3 Re 100 cavity, ten GIP timesteps
        {"name": "steps_fixed_48", "kind": "steps", "n": 48, "re": 100.0, "solver": "fixed",
         "steps": 10, "permute": False},
        # a mid-sized mesh in arbitrary cell order, renumbered by the engine, mixed form with AMG
        {"name": "steps_mixed_amg_63", "kind": "steps", "n": 63, "re": 400.0,
         "solver": "mixed_amg", "steps": 10, "permute": True},
        # the 256^3 Re 1000 cavity in the mixed form with AMG
        {"name": "steps_mixed_amg_256", "kind": "steps", "n": 256, "re": 1000.0,
         "solver": "mixed_amg", "steps": 3, "permute": False},
        # uneven cavities advanced together
        {"name": "batch_12", "kind": "batch", "count": 12, "lo": 24, "hi": 64, "pick": 5,
         "solver": "mixed_amg", "steps": 3},
        # kinetic energy and its gradient with respect to lid and viscosity
        {"name": "adjoint_32", "kind": "adjoint", "n": 32, "re": 400.0, "steps": 10, "every": 5},
    ]


def draw(rng):
    def edge(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["spmv", "host_loop", "poisson", "poisson", "steps", "steps", "steps",
                       "batch", "adjoint"])
    if kind == "spmv":
        return {"kind": kind, "n": edge(12, 200), "mode": rng.choice([0, 1])}
    if kind == "host_loop":
        return {"kind": kind, "n": edge(10, 100), "iters": 100}
    if kind == "poisson":
        return {"kind": kind, "n": edge(16, 144), "solver": rng.choice(sorted(POISSON))}
    if kind == "steps":
        solver = rng.choice(sorted(SOLVERS))
        return {"kind": kind, "n": edge(10, 128), "re": rng.choice([100.0, 400.0, 1000.0]),
                "solver": solver, "steps": rng.randint(2, 8) if solver == "tol" else 10,
                "permute": rng.choice([False, True])}
    if kind == "batch":
        lo = edge(12, 32)
        return {"kind": kind, "count": rng.randint(3, 16), "lo": lo, "hi": lo + rng.randint(4, 32),
                "pick": rng.randint(0, 999), "solver": rng.choice(["mixed_amg", "mixed"]),
                "steps": rng.randint(1, 4)}
    return {"kind": kind, "n": edge(10, 40), "re": rng.choice([100.0, 400.0]),
            "steps": rng.randint(3, 12), "every": rng.randint(2, 6)}


# ------------------------------------------------------------------------------- set-up
def _keep(key, make):
    if key not in _kept:
        while len(_kept) >= KEPT:
            _kept.popitem(last=False)
        _kept[key] = make()
    return _kept[key]


def _pressure(n):
    """The cavity's pressure operator without ghost columns (host CSR)."""
    L = cavity.generate(n, ghost_cols=False)[0].ops["L"]
    return Csr(L.nrows, L.nrows, L.rowptr, L.col, L.val)


def _gpu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _rhs(n, seed):
    """A right-hand side U[-1, 1] with its mean removed, as the Poisson benchmark has it."""
    b = np.random.default_rng(seed).uniform(-1.0, 1.0, n ** 3)
    return b - b.mean()


def _lid(n, seed):
    """Lid velocity profile: unit speed with 1% noise."""
    return 1.0 + np.random.default_rng(seed).normal(0.0, 0.01, n * n)


def _cavity(c):
    return cavity.generate(c["n"], re=c["re"], permute_seed=1234 if c["permute"] else None)


def _engine(c):
    # arbitrary cell orders and large meshes are renumbered for locality
    E = DnsEngine(_cavity(c)[0], gamma=1.0 / c["re"], reorder=c["permute"] or c["n"] >= 128,
                  **SOLVERS[c["solver"]])
    E.advance(1)      # the first step, from rest
    E.snapshot()      # where every run restarts
    torch.cuda.synchronize()
    return E


def _members(c):
    """Edges and Reynolds numbers of a batch's cavities."""
    rng = np.random.default_rng(c["pick"])
    edges = [int(n) for n in rng.integers(c["lo"], c["hi"] + 1, c["count"])]
    res = [float(r) for r in np.exp(rng.uniform(math.log(100.0), math.log(1000.0), c["count"]))]
    return edges, res


def _batch(c):
    edges, res = _members(c)
    cases = [cavity.generate(n, re=r)[0] for n, r in zip(edges, res)]
    B = DnsBatch(cases, [dns_params(gamma=1.0 / r, reorder=True, **SOLVERS[c["solver"]])
                         for r in res])
    B.advance(1)
    for e in B.instances:
        e.snapshot()
    torch.cuda.synchronize()
    return B


def _adjoint(c):
    case, meta = cavity.generate(c["n"], re=c["re"])
    A = CavityAdjoint(case, meta.lid_ghosts, np.full(case.n_inner, meta.h ** 3),
                      nu0=1.0 / c["re"], gamma=1.0 / c["re"], tol=1e-12,
                      checkpoint_every=c["every"], precond="amg")
    A.forward(np.ones(c["n"] ** 2), 1.0 / c["re"], c["steps"])  # records the CFL time steps
    return A


def prepare(case, seed):
    k, n = case["kind"], case.get("n")
    if k == "spmv":
        A = _keep(("L", n), lambda: DeviceMatrix(_pressure(n)))
        g = torch.Generator(device="cuda").manual_seed(seed)
        x, y = torch.randn(2, n ** 3, dtype=torch.float64, device="cuda", generator=g)
        return {"case": case, "A": A, "x": x.contiguous(), "y": y.contiguous()}
    if k == "host_loop":
        def make():
            L = _pressure(n)
            rows = np.repeat(np.arange(L.nrows), np.diff(L.rowptr))
            diag = np.zeros(L.nrows)
            diag[rows[rows == L.col]] = 1.0 / L.val[rows == L.col]
            D = Csr(L.nrows, L.nrows, np.arange(L.nrows + 1, dtype=np.int32),
                    np.arange(L.nrows, dtype=np.int32), diag)
            return DeviceMatrix(L), DeviceMatrix(D), _gpu(diag)

        A, D, dinv = _keep(("loop", n), make)
        return {"case": case, "A": A, "D": D, "dinv": dinv, "b": _gpu(_rhs(n, seed)),
                "x": torch.zeros(n ** 3, dtype=torch.float64, device="cuda"),
                "x0": torch.zeros(n ** 3, dtype=torch.float64, device="cuda")}
    if k == "poisson":
        S = _keep((k, n, case["solver"]),
                  lambda: PcgSolver(DeviceMatrix(_pressure(n)), **POISSON[case["solver"]]))
        return {"case": case, "S": S, "b": _gpu(_rhs(n, seed)),
                "x": torch.zeros(n ** 3, dtype=torch.float64, device="cuda"),
                "x0": torch.zeros(n ** 3, dtype=torch.float64, device="cuda")}
    if k == "steps":
        E = _keep((k, n, case["re"], case["solver"], case["permute"]), lambda: _engine(case))
        return {"case": case, "E": E, "lid": torch.from_numpy(_lid(n, seed)).pin_memory()}
    if k == "batch":
        B = _keep(tuple(case[q] for q in ("kind", "count", "lo", "hi", "pick", "solver")),
                  lambda: _batch(case))
        edges, _ = _members(case)
        return {"case": case, "B": B, "edges": edges,
                "lids": [torch.from_numpy(_lid(m, seed + 1000003 * i)).pin_memory()
                         for i, m in enumerate(edges)]}
    A = _keep((k, n, case["re"], case["steps"], case["every"]), lambda: _adjoint(case))
    nu = (1.0 + 0.05 * float(np.random.default_rng(seed + 1).uniform(-1.0, 1.0))) / case["re"]
    return {"case": case, "A": A, "lid": torch.from_numpy(_lid(n, seed)).requires_grad_(),
            "nu": torch.tensor(nu, dtype=torch.float64, requires_grad=True)}


# ---------------------------------------------------------------------------------- run
FIELDS = ("u", "v", "w", "p", "mf")


def _restart(E, n, lid):
    """Back to the kept state with new lid velocities (the lid's ghosts end the ghost cells)."""
    E.snapshot(restore=True)
    E.set_field("u", lid.numpy(), offset=n ** 3 + 5 * n * n)


def _fields(E, names):
    return {f: E.copy_field(f, torch.empty(E.n_faces if f == "mf" else E.n_owned,
                                           dtype=torch.float64, device="cuda")) for f in names}


def run(state):
    c = state["case"]
    k = c["kind"]
    if k == "spmv":
        if c["mode"]:  # y = alpha A x + beta y
            return state["A"].spmv(state["x"], state["y"].clone(), 0.5, -0.25, 1)
        return state["A"].spmv(state["x"], torch.empty_like(state["y"]))
    if k == "host_loop":
        host_loop_pcg(state["A"], state["D"], state["dinv"], state["b"], state["x"], state["x0"],
                      c["iters"])
        return state["x"]
    if k == "poisson":
        state["S"].solve(state["b"], state["x"], state["x0"])
        return state["x"]
    if k == "steps":
        _restart(state["E"], c["n"], state["lid"])
        state["E"].advance(c["steps"])
        return _fields(state["E"], FIELDS)
    if k == "batch":
        B = state["B"]
        for e, n, lid in zip(B.instances, state["edges"], state["lids"]):
            _restart(e, n, lid)
        B.advance(c["steps"])
        return [_fields(e, ("u", "v", "w", "p")) for e in B.instances]
    J = state["A"].energy(state["lid"], state["nu"], c["steps"])
    g = torch.autograd.grad(J, (state["lid"], state["nu"]))
    return {"J": J.detach(), "lid": g[0], "nu": g[1]}


# --------------------------------------------------------------------------------- work
def _step_work(n, iters):
    """Bytes and flops of one timestep on n^3 cells: its operators (12 bytes a nonzero), its
    face and cell fields once in and once out; `iters` solver iterations' arithmetic."""
    cells, faces = n ** 3, 3 * (n + 1) * n * n
    nnz = (7 + 7 + 6 + 6 + 6 + 12) * cells + 12 * faces  # L, D, Mres, M, G, Ec; SO and SF
    return 12.0 * nnz + 8.0 * (20 * cells + 2 * faces), 2.0 * (nnz + 14 * cells +
                                                                iters * 12 * cells)


def work(case):
    k, n = case["kind"], case.get("n")
    if k == "batch":
        got = [_step_work(m, 20) for m in _members(case)[0]]
        return {"bytes": case["steps"] * sum(g[0] for g in got),
                "flops": case["steps"] * sum(g[1] for g in got)}
    cells = n ** 3
    if k == "spmv":  # operator, x, y in and out
        return {"bytes": 12.0 * 7 * cells + (24.0 if case["mode"] else 16.0) * cells,
                "flops": 14.0 * cells}
    if k in ("host_loop", "poisson"):  # operator, b, x0 in; x out; the iterations' arithmetic
        iters = case.get("iters", 20 if case.get("solver") == "mixed_amg" else 9 * n)
        return {"bytes": 12.0 * 7 * cells + 24.0 * cells, "flops": 26.0 * cells * iters}
    iters = {"fixed": 100, "tol": 3 * n, "mixed": 3 * n}.get(case.get("solver"), 20)
    b, f = _step_work(n, iters)
    times = case["steps"] * (3 if k == "adjoint" else 1)  # forward, replay, backward
    return {"bytes": times * b, "flops": times * f}


# -------------------------------------------------------------------------------- exact
class _Rows:
    """A CSR operator on the GPU in plain torch; rows without nonzeros are known."""

    def __init__(self, m):
        self.nrows = m.nrows
        rp = torch.from_numpy(np.asarray(m.rowptr, np.int64)).cuda()
        self.some = rp[1:] > rp[:-1]
        self.row = torch.repeat_interleave(torch.arange(m.nrows, device="cuda"), rp[1:] - rp[:-1])
        self.col = torch.from_numpy(np.asarray(m.col, np.int64)).cuda()
        self.val = torch.from_numpy(np.asarray(m.val, np.float64)).cuda()

    def __call__(self, x, val=None):
        y = torch.zeros(self.nrows, dtype=torch.float64, device="cuda")
        return y.index_add(0, self.row, (self.val if val is None else val) * x[self.col])


class _Neumann:
    """The cavity's pinned pressure system solved by cosine transforms: the rows of L but the
    pin's sum to zero, so sum(b) = pin x_p, and the rest is the Neumann Laplacian."""

    def __init__(self, n, perm=None):
        i = np.arange(n)
        q = np.cos(np.pi * (i[:, None] + 0.5) * i[None, :] / n) * math.sqrt(2.0 / n)
        q[:, 0] = math.sqrt(1.0 / n)
        lam = (2.0 - 2.0 * np.cos(np.pi * i / n)) / n  # face area over distance: 1 / n
        lam3 = lam[:, None, None] + lam[None, :, None] + lam[None, None, :]
        lam3[0, 0, 0] = np.inf
        self.n, self.q, self.lam = n, _gpu(q), _gpu(lam3)
        self.cell = (n // 2) * (1 + n + n * n)
        self.pin = 6.0 / n / 101.0
        self.perm = None if perm is None else torch.from_numpy(np.asarray(perm, np.int64)).cuda()

    def _modes(self, a, t):
        q = self.q.T if t else self.q
        a = torch.einsum("ia,abc->ibc", q, a)
        a = torch.einsum("jb,ibc->ijc", q, a)
        return torch.einsum("kc,ijc->ijk", q, a)

    def __call__(self, b):
        if self.perm is not None:
            b = b[self.perm]
        total = b.sum()
        e = torch.zeros_like(b)
        e[self.cell] = 1.0
        f = (b - total * e).reshape(self.n, self.n, self.n)
        x = self._modes(self._modes(f, True) / self.lam, False).reshape(-1)
        x = x + (total / self.pin - x[self.cell])
        if self.perm is not None:
            x = torch.zeros_like(x).index_copy(0, self.perm, x)
        return x


def _jacobi_cg(A, dinv, b, x, iters):
    """GIP_LinearSolver's Jacobi-PCG: exactly `iters` iterations."""
    r = b - A(x)
    p = dinv * r
    rz = r @ p
    for _ in range(iters):
        q = A(p)
        alpha = rz / (p @ q)
        x = x + alpha * p
        r = r - alpha * q
        z = dinv * r
        old, rz = rz, r @ z
        p = z + (rz / old) * p
    return x


class _Timestep:
    """GIP_DNS's timestep in plain torch (rho = 1)."""

    def __init__(self, case, gamma, solve):
        self.N, self.NO = case.n_inner, case.n_owned
        self.op = {k: _Rows(case.ops[k]) for k in case.ops}
        self.gamma, self.solve = gamma, solve
        f = {k: _gpu(case.fields[k]) for k in ("u", "v", "w", "dxs")}
        self.vel = [f["u"], f["v"], f["w"]]
        self.dx = f["dxs"][:self.N]
        self.a0 = [torch.zeros(self.N, dtype=torch.float64, device="cuda") for _ in range(3)]
        self.mf = torch.zeros(case.n_faces, dtype=torch.float64, device="cuda")
        self.p0 = torch.zeros(self.N, dtype=torch.float64, device="cuda")
        self.p = None
        self.nu = 1.0
        self.dt = None

    def cfl(self):
        speed = torch.stack([x[:self.N].abs() for x in self.vel]).amax(0)
        dt = torch.minimum(0.25 * self.dx / speed, 0.2 * self.dx * self.dx / self.gamma).min()
        return min(0.8 * float(dt), 0.1)

    def step(self, dt=None):
        op, N = self.op, self.N
        if dt is None:
            dt = self.dt if self.dt is not None else self.cfl()
        cval = torch.where(op["Ec"].some, op["Ec"](self.mf), op["D"].val)
        a = [self.nu * op["D"](x) - op["D"](x, cval) for x in self.vel]
        star = [torch.cat([x[:N] + 1.5 * dt * f - 0.5 * dt * g, x[N:]])
                for x, f, g in zip(self.vel, a, self.a0)]
        self.a0 = a
        rhs = (op["Mx"](star[0]) + op["My"](star[1]) + op["Mz"](star[2])) / dt
        p = self.solve(self, rhs)
        self.p0 = p
        full = torch.cat([p, torch.zeros(self.NO - N, dtype=torch.float64, device="cuda")])
        full = full + op["Lb"](full)
        self.p = full
        gp = [op["G" + d](full) for d in "xyz"]
        self.vel = [torch.cat([x[:N] - dt * g[:N], x[N:]]) for x, g in zip(star, gp)]
        mf = torch.where(op["SO"].some, -dt * op["SO"](full), self.mf)
        for d, g, x in zip("xyz", gp, self.vel):
            mf = mf + dt * op["SF" + d](g)
        for d, x in zip("xyz", self.vel):
            mf = mf + op["SF" + d](x)
        self.mf = mf
        self.dt = self.cfl() if not torch.is_grad_enabled() else None
        return dt


def _exact_steps(n, re, solver, steps, lid, permute):
    case, meta = cavity.generate(n, re=re, permute_seed=1234 if permute else None)
    if solver == "fixed":
        L = _Rows(case.ops["L"])
        dinv = torch.zeros(case.n_inner, dtype=torch.float64, device="cuda")
        on = L.row == L.col
        dinv[L.row[on]] = 1.0 / L.val[on]
        ghosts = torch.zeros(case.n_owned - case.n_inner, dtype=torch.float64, device="cuda")

        def solve(t, b):
            return _jacobi_cg(lambda x: L(torch.cat([x, ghosts])), dinv, b, t.p0, 100)
    else:
        direct = _Neumann(n, meta.cell_perm)

        def solve(t, b):
            return direct(b)
    T = _Timestep(case, 1.0 / re, solve)
    T.step()
    at = n ** 3 + 5 * n * n
    T.vel[0] = T.vel[0].clone()
    T.vel[0][at:at + n * n] = _gpu(lid)
    for _ in range(steps):
        T.step()
    return {"u": T.vel[0], "v": T.vel[1], "w": T.vel[2], "p": T.p, "mf": T.mf}


def exact(case, seed):
    k, n = case["kind"], case.get("n")
    if k == "adjoint":
        return _exact_adjoint(case, seed)
    with torch.no_grad():
        if k == "batch":
            edges, res = _members(case)
            out = []
            for i, (m, r) in enumerate(zip(edges, res)):
                f = _exact_steps(m, r, case["solver"], case["steps"], _lid(m, seed + 1000003 * i),
                                 False)
                out.append({q: f[q] for q in ("u", "v", "w", "p")})
            return out
        if k == "steps":
            if n > 144:
                return None  # its operators alone take most of the time there is
            return _exact_steps(n, case["re"], case["solver"], case["steps"], _lid(n, seed),
                                case["permute"])
        if k == "poisson":
            return _Neumann(n)(_gpu(_rhs(n, seed)))
        A = _Rows(_pressure(n))
        if k == "spmv":
            g = torch.Generator(device="cuda").manual_seed(seed)
            x, y = torch.randn(2, n ** 3, dtype=torch.float64, device="cuda", generator=g)
            return 0.5 * A(x) - 0.25 * y if case["mode"] else A(x)
        on = A.row == A.col
        dinv = torch.zeros(n ** 3, dtype=torch.float64, device="cuda")
        dinv[A.row[on]] = 1.0 / A.val[on]
        b = _gpu(_rhs(n, seed))
        return _jacobi_cg(A, dinv, b, torch.zeros_like(b), case["iters"])


def _exact_adjoint(case, seed):
    n, re, steps = case["n"], case["re"], case["steps"]
    cav, meta = cavity.generate(n, re=re)
    direct = _Neumann(n)
    at = n ** 3 + 5 * n * n

    def simulate(lid, nu_scale, dts):
        T = _Timestep(cav, 1.0 / re, lambda t, b: direct(b))
        u = T.vel[0]
        T.vel[0] = torch.cat([u[:at], lid, u[at + n * n:]])
        T.nu = nu_scale
        used = [T.step(dts[i] if dts else None) for i in range(steps)]
        return T, used

    with torch.no_grad():
        _, dts = simulate(torch.ones(n * n, dtype=torch.float64, device="cuda"), 1.0, None)
    lid = _gpu(_lid(n, seed)).requires_grad_()
    nu = (1.0 + 0.05 * float(np.random.default_rng(seed + 1).uniform(-1.0, 1.0))) / re
    nu = torch.tensor(nu, dtype=torch.float64, device="cuda", requires_grad=True)
    T, _ = simulate(lid, nu * re, dts)
    J = 0.5 * meta.h ** 3 * sum((x[:n ** 3] ** 2).sum() for x in T.vel)
    g = torch.autograd.grad(J, (lid, nu))
    return {"J": J.detach(), "lid": g[0], "nu": g[1]}
