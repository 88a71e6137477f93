"""The work this solver is used for, as cases that can be timed and checked.

Every case goes through the package's public surface (`solver.Solver`, `Integrator`, `Batch`, the
C ABI they bind) on a rotated simple wave (gamma = 3) of seeded amplitude and phase, scaled by a
smooth seeded perturbation: the states that the speed protocol, the accuracy runs, the uneven
batch and the adjoint configuration of this repository solve for.

Kinds:
  residual  one evaluation of the frozen-speed DG residual R(u)
  jv, jtw   the matrix-free J v and its adjoint J^T w at a linearised state
  adjoint   one J^T GMRES solve of the discrete adjoint (the factors are kept, as they are there)
  factor    FP64 block Jacobi: linearise, assemble, factor every cell block, apply it once
  condense  FP64 HDG condensation: residual, condense, condensed right-hand side, one Schur apply,
            one recovery
  newton    one backward-Euler Newton update from the start of a stage (linearise, factor or
            condense, GMRES, line search)
  advance   time steps of the full integrator on a host state, copies included
  batch     one Newton update of every member of an uneven batch
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

GAMMA = 3.0
SAFETY = 1.1
DIRK_A = 0.24169426078821
DIRK_B, DIRK_E = DIRK_A / 4, 0.12915286960590
STAGES = {
    "be": ([[1.0]], [1.0]),
    "ssp-dirk3": ([[DIRK_A], [-DIRK_A, DIRK_A], [0, 1 - DIRK_A, DIRK_A],
                   [DIRK_B, DIRK_E, 0.5 - DIRK_B - DIRK_E - DIRK_A, DIRK_A]], [0, 1 / 6, 1 / 6, 2 / 3]),
}


def listed():
    return [
        # the command-line default mesh (8 x 8, k = 3): a single small call, all launch latency
        dict(name="residual_8_k3", kind="residual", nx=8, ny=8, k=3, quad=0),
        # the operator of every DG Krylov step at the speed-protocol size
        dict(name="jv_256_k8", kind="jv", nx=256, ny=256, k=8, quad=0),
        # the over-integrated volume rule, an option of every 2D run, on an odd mesh
        dict(name="residual_75x53_k5_q8", kind="residual", nx=75, ny=53, k=5, quad=8),
        # one stage solve of the discrete adjoint (k = 4, CFL 2) on a quarter of its 128 x 128 mesh
        dict(name="adjoint_64_k4", kind="adjoint", nx=64, ny=64, k=4, cfl=2.0, restart=20),
        # the FP64 block-Jacobi factorisation at the protocol's degree, ragged against any grid of CTAs
        dict(name="factor_fp64_50x45_k8", kind="factor", nx=50, ny=45, k=8),
        # the FP64 condensation at a middle degree on an odd mesh
        dict(name="condense_fp64_61x43_k6", kind="condense", nx=61, ny=43, k=6),
        # ordinary implicit steps: FP32 factors on a ragged mesh, and the all-FP64 condensed form
        dict(name="newton_dg_mixed_97x61_k5", kind="newton", method="dg", precision="mixed", condense32=0, nx=97, ny=61,
             k=5, cfl=5.0, restart=20, graph=False),
        dict(name="newton_hdg_fp64_64_k4", kind="newton", method="hdg", precision="fp64", condense32=0, nx=64, ny=64, k=4,
             cfl=5.0, restart=20, graph=False),
        # the speed protocol's two headline updates
        dict(name="newton_dg_mixed16_256_k8", kind="newton", method="dg", precision="mixed16", condense32=0, nx=256,
             ny=256, k=8, cfl=5.0, restart=20, graph=True),
        dict(name="newton_hdg_mixed32_256_k8", kind="newton", method="hdg", precision="mixed", condense32=1, nx=256,
             ny=256, k=8, cfl=5.0, restart=20, graph=True),
        # one SSP-DIRK3 step of the accuracy runs (64 x 64, k = 2, CFL 2): launch-bound whole calls
        dict(name="advance_dirk3_64_k2", kind="advance", dim=2, integrator="ssp-dirk3", method="dg", nx=64, ny=64, k=2,
             cfl=2.0, restart=20, steps=1),
        # an uneven batch: several degrees, meshes and methods advanced together
        dict(name="batch_5", kind="batch", members="k8n32dg k4n64hdg k6n48dg k2n64dg k8n32hdg", cfl=5.0,
             restart=30, graph=True),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def mesh(k, most_cells, lo=8, hi=256):
        while True:
            nx, ny = log_int(lo, hi), log_int(lo, hi)
            if nx * ny <= most_cells:
                return dict(nx=nx, ny=ny, k=k)

    k = rng.randint(1, 8)
    m2 = (4 * (k + 1) ** 2) ** 2
    kind = rng.choice(["residual", "jv", "jtw", "adjoint", "factor", "condense", "newton", "newton", "newton", "advance",
                       "batch"])
    if kind in ("residual", "jv", "jtw"):
        quad = 0 if rng.random() < 0.75 else rng.randint(k + 2, min(16, 2 * k + 3))
        return dict(kind=kind, quad=quad, **mesh(k, 65536 if not quad else 10000))
    if kind == "adjoint":
        return dict(kind=kind, cfl=2.0, restart=20, **mesh(k, int(1.5e8 / m2) + 64, hi=128))
    if kind in ("factor", "condense"):
        return dict(kind=kind, **mesh(k, int(2.5e8 / m2) + 64, hi=160))
    if kind == "newton":
        method = rng.choice(["dg", "hdg"])
        precision = rng.choice(["fp64", "mixed", "mixed16"] if method == "dg" else ["fp64", "mixed"])
        return dict(kind=kind, method=method, precision=precision,
                    condense32=1 if method == "hdg" and precision == "mixed" and rng.random() < 0.6 else 0,
                    cfl=5.0, restart=rng.choice([20, 30]), graph=rng.random() < 0.5,
                    **mesh(k, int(3e8 / m2) + 64, hi=160))
    if kind == "advance":
        if rng.random() < 0.4:
            return dict(kind=kind, dim=1, integrator=rng.choice(["ssp-dirk3", "be"]), method=rng.choice(["dg", "hdg"]),
                        nx=log_int(16, 256), ny=1, k=rng.randint(1, 4), cfl=2.0, restart=20, steps=rng.randint(1, 3))
        return dict(kind=kind, dim=2, integrator=rng.choice(["ssp-dirk3", "be"]), method=rng.choice(["dg", "hdg"]),
                    cfl=2.0, restart=20, steps=1, **mesh(rng.randint(1, 4), 4096, hi=96))
    members = " ".join("k%dn%d%s" % (rng.choice([2, 4, 6, 8]), rng.choice([16, 24, 32, 48]), rng.choice(["dg", "hdg"]))
                       for _ in range(rng.randint(2, 5)))
    return dict(kind=kind, members=members, cfl=5.0, restart=30, graph=rng.random() < 0.5)


# ---- inputs ---------------------------------------------------------------------------------------
def _device():
    return torch.device("cuda", 0) if torch.cuda.is_available() else torch.device("cpu")


def _t(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device=_device())


def _state(nx, ny, k, seed, dim=2):
    """Nodal values of the perturbed simple wave in the solver's layout ([cell][variable][node])."""
    r = np.random.RandomState(seed)
    amp, phase = 0.8 + 0.2 * r.rand(), 2 * math.pi * r.rand()
    bump, px, py = 0.05 + 0.2 * r.rand(), 2 * math.pi * r.rand(), 2 * math.pi * r.rand()
    xi = _t(np.polynomial.legendre.leggauss(k + 1)[0])
    pi = math.pi
    X = (torch.arange(nx, device=_device(), dtype=torch.float64)[:, None] + (xi + 1) / 2) / nx  # [cx][i]
    if dim == 1:
        s = 2 * X - 1
        factor = 1 + bump * torch.sin(2 * pi * X + px)
    else:
        Y = (torch.arange(ny, device=_device(), dtype=torch.float64)[:, None] + (xi + 1) / 2) / ny  # [cy][j]
        s = 2 * X[None, :, None, :] + 2 * Y[:, None, :, None] - 2
        factor = 1 + bump * torch.sin(2 * pi * X + px)[None, :, None, :] * torch.sin(2 * pi * Y + py)[:, None, :, None]
    jm = amp * torch.sin(pi * s + phase)
    speed, sound = (2 + jm) / 2, (2 - jm) / 2
    rho = sound / math.sqrt(GAMMA)
    energy = rho ** 3 / (GAMMA - 1) + 0.5 * rho * speed * speed
    if dim == 1:
        u = torch.stack([rho, rho * speed, energy], dim=1) * factor[:, None]  # [cell][v][i]
    else:
        c = math.sqrt(0.5)
        u = torch.stack([rho, rho * speed * c, rho * speed * c, energy], dim=2) * factor[:, :, None]  # [cy][cx][v][j][i]
    return u.reshape(-1).contiguous()


def _direction(n, seed):
    return _t(np.random.RandomState(seed + 7919).standard_normal(n))


def _members(case):
    out = []
    for text in case["members"].split():
        k, rest = text[1:].split("n", 1)
        method = "hdg" if rest.endswith("hdg") else "dg"
        out.append((int(k), int(rest[:-len(method)]), method))
    return out


def prepare(case, seed):
    from dg_hdg_euler_cpp_b200.solver import Batch, Integrator, Solver

    kind = case["kind"]
    st = {"case": case, "seed": seed}
    if kind == "batch":
        members = _members(case)
        st["batch"] = Batch([dict(nx=n, ny=n, k=k, cfl=case["cfl"], integrator="be", steps=1, restart=case["restart"],
                                  max_linear=1500, method=method, precision="mixed") for k, n, method in members])
        st["batch"].gmres_graph(case["graph"])
        st["states"] = [_state(n, n, k, seed + 101 * i).cpu().numpy() for i, (k, n, _) in enumerate(members)]
        return st
    nx, ny, k = case["nx"], case["ny"], case["k"]
    if kind == "advance":
        st["solver"] = Solver(dim=case["dim"], nx=nx, ny=max(ny, 3), k=k, cfl=case["cfl"], integrator=case["integrator"],
                              steps=case["steps"], method=case["method"], restart=case["restart"])
        st["host"] = _state(nx, ny, k, seed, case["dim"]).cpu().numpy()
        return st
    u = st["u"] = _state(nx, ny, k, seed)
    if kind == "newton":
        s = Solver(nx=nx, ny=ny, k=k, cfl=case["cfl"], integrator="be", steps=1, method=case["method"],
                   precision=case["precision"], condense32=case["condense32"], restart=case["restart"], max_linear=1500,
                   safety=SAFETY)
        s.gmres_graph(case["graph"])
        st["solver"], st["integrator"] = s, Integrator(s, case["method"])
        return st
    s = st["solver"] = Solver(nx=nx, ny=ny, k=k, quad=case.get("quad", 0), cfl=case.get("cfl", 5.0),
                              method="hdg" if kind == "condense" else "dg", restart=case.get("restart", 1),
                              precision="mixed16" if kind in ("residual", "jv", "jtw") and not case["quad"] else "fp64",
                              safety=SAFETY)
    rate = s.freeze(u)
    old = _state(nx, ny, k, seed + 1)
    s.set_stage(old, case.get("cfl", 5.0) / rate)
    if kind != "residual" and kind != "condense":
        s.dg_refresh(u)
    if kind == "adjoint":
        s.precond_refresh("dg")
    st["v"] = _direction(s.trace_size if kind == "condense" else s.size, seed)
    return st


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "batch":
        b = state["batch"]
        b.stage_begin(state["states"])
        b.update()
        return [b.state(i) for i in range(b.count)]
    s = state["solver"]
    if kind == "advance":
        return s.advance(case["method"], state["host"], max_updates=256)[0]
    if kind == "newton":
        it = state["integrator"]
        it.stage_begin(state["u"])
        it.update()
        out = torch.empty(s.size, dtype=torch.float64, device=s.device)
        p = ctypes.c_void_p(it.state_ptr())
        s.lib.dgh_axpby(s.h, ctypes.c_double(1.0), p, ctypes.c_double(0.0), p, ctypes.c_void_p(out.data_ptr()), s.size)
        s.lib.dgh_sync(s.h)
        return out
    if kind == "residual":
        return s.residual(state["u"])
    if kind == "jv":
        return s.dg_apply(state["v"])
    if kind == "jtw":
        return s.dg_apply_T(state["v"])
    if kind == "adjoint":
        return s.gmres("dg_t", state["v"], 1500, 1e-12)[0]
    if kind == "factor":
        s.dg_refresh(state["u"])
        s.precond_refresh("dg")
        return s.precond_apply("dg", state["v"])
    s.hdg_refresh_projected(state["u"], s.residual(state["u"]))
    return {"rhs": s.hdg_rhs(), "schur": s.hdg_apply(state["v"]), "du": s.hdg_recover(state["v"])}


# ---- the work of one pass -------------------------------------------------------------------------
def _newton_work(cells, n, method, fbytes, sbytes, krylov, restart):
    """Bytes and flops of one Newton update with `krylov` GMRES steps: the factors or Schur blocks
    written once and read once a step, the operator's vectors, the CGS2 sweeps, the factorisation."""
    m, fw, t = 4 * n * n, 4 * n, 16 * n
    basis = min(krylov, restart) / 2 + 1
    lu = 2 / 3 * m ** 3
    if method == "dg":
        N, op_bytes = cells * m, 8 * 2.75 * cells * m
        pre, flops = fbytes * m * m * cells, lu * cells
        step_flops = 2 * m * m * cells + N * (4 * n + 60)
    else:
        N, op_bytes = 2 * cells * fw, sbytes * t * t * cells
        pre, flops = fbytes * fw * fw * 2 * cells, (lu + 2 * m * m * (t + 1)) * cells
        step_flops = 2 * t * t * cells + 2 * fw * fw * 2 * cells
    step = pre + op_bytes + 8 * N * (3 * basis + 5)
    return {"bytes": pre + (op_bytes if method == "hdg" else 0) + krylov * step + 8 * 8 * cells * m,
            "flops": flops + krylov * (step_flops + 6 * basis * N)}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        parts = [_newton_work(n * n, k + 1, method, 4, 8, 60, case["restart"]) for k, n, method in _members(case)]
        return {key: sum(p[key] for p in parts) for key in ("bytes", "flops")}
    n = case["k"] + 1
    cells = case["nx"] * case["ny"]
    m, fw, t = 4 * n * n, 4 * n, 16 * n
    N, speeds = cells * m, 4 * cells * n
    if kind in ("residual", "jv", "jtw"):
        q = case["quad"] or n
        volume = N * (4 * n + 60) if q == n else 4 * cells * (4 * n * q * (n + q)) * 2 + 60 * cells * q * q
        return {"bytes": 8 * (3 * N + speeds), "flops": volume + 60 * 4 * cells * n}
    if kind == "factor":
        return {"bytes": cells * 16 * m * m + 8 * 3 * N, "flops": cells * (2 / 3 * m ** 3 + 2 * m * m)}
    if kind == "condense":
        return {"bytes": cells * 8 * (2 * t * t + 2 * m * t) + 8 * 4 * N + 8 * 4 * 2 * cells * fw,
                "flops": cells * (2 / 3 * m ** 3 + 2 * m * m * (t + 1) + 2 * t * t + 2 * m * t)}
    if kind == "adjoint":
        w = _newton_work(cells, n, "dg", 8, 8, 60, case["restart"])
        return {"bytes": w["bytes"] - 8 * m * m * cells, "flops": w["flops"] - 2 / 3 * m ** 3 * cells}
    if kind == "advance":
        if case["dim"] == 1:
            m, N = 3 * n, 3 * n * cells
            solves = (16 if case["integrator"] == "ssp-dirk3" else 4) * case["steps"]
            return {"bytes": solves * 20 * 8 * cells * (m * m + 20 * m), "flops": solves * cells * (m ** 3 + 40 * m * m)}
        solves = (16 if case["integrator"] == "ssp-dirk3" else 5) * case["steps"]
        w = _newton_work(cells, n, case["method"], 8, 8, 25, case["restart"])
        return {"bytes": solves * w["bytes"], "flops": solves * w["flops"]}
    half = {"fp64": 8, "mixed": 4, "mixed16": 2}[case["precision"]]
    face = 8 if case["precision"] == "fp64" else 4
    krylov = 200 if cells > 30000 else 100
    return _newton_work(cells, n, case["method"], half if case["method"] == "dg" else face,
                        4 if case["condense32"] else 8, krylov, case["restart"])


# ---- the same in 64-bit torch, from the scheme's definition ----------------------------------------
class _Scheme:
    """The DG scheme on an nx x ny periodic mesh of tensor-product Gauss cells (dim 2), or its 1D
    form, as differentiable torch functions of the nodal state u [ny][nx][4][n][n] ([nx][3][n])."""

    def __init__(self, nx, ny, k, quad=0, dim=2):
        self.dim, self.nx, self.ny, self.n = dim, nx, ny, k + 1
        self.q = quad or k + 1
        n = k + 1
        x, w = np.polynomial.legendre.leggauss(n)
        qx, qw = (x, w) if self.q == n else np.polynomial.legendre.leggauss(self.q)
        bary = np.array([1 / np.prod([x[i] - x[j] for j in range(n) if j != i]) for i in range(n)])

        def lagrange(y):
            return np.array([np.prod([(y - x[j]) for j in range(n) if j != i]) * bary[i] for i in range(n)])

        D = np.array([[0.0 if i == j else bary[j] / (bary[i] * (x[i] - x[j])) for j in range(n)] for i in range(n)])
        D -= np.diag(D.sum(1))
        V = np.eye(n) if self.q == n else np.array([lagrange(y) for y in qx])
        self.w, self.V, self.qw = _t(w), _t(V), _t(qw)
        self.wd = _t(qw[:, None] * (V @ D))   # [q][i] = qw_q l_i'(x_q)
        self.eL, self.eR = _t(lagrange(-1.0)), _t(lagrange(1.0))
        self.nvar = 4 if dim == 2 else 3
        self.m = self.nvar * n ** dim
        if dim == 2:
            self.shape = (ny, nx, 4, n, n)
            self.hx, self.hy = 2 * math.sqrt(2.0) / nx, 2 * math.sqrt(2.0) / ny
            self.fwx, self.fwy = 0.5 * self.hy * self.w, 0.5 * self.hx * self.w
            self.mass = 0.25 * self.hx * self.hy * self.w[:, None] * self.w[None, :]
        else:
            self.shape = (nx, 3, n)
            self.hx = 2.0 / nx
            self.mass = 0.5 * self.hx * self.w

    @staticmethod
    def primitive(u, dim):
        """velocities, pressure, enthalpy; u has its variables in dimension 2 (2D) or 1 (1D)."""
        ax = 2 if dim == 2 else 1
        c = u.unbind(ax)
        vel = [c[1 + a] / c[0] for a in range(dim)]
        p = (GAMMA - 1) * (c[-1] - 0.5 * sum(c[1 + a] * vel[a] for a in range(dim)))
        return c, vel, p, (c[-1] + p) / c[0]

    def flux(self, u, axis):
        c, vel, p, _ = self.primitive(u, self.dim)
        f = [c[1 + axis]] + [c[1 + a] * vel[axis] + (p if a == axis else 0) for a in range(self.dim)]
        return torch.stack(f + [(c[-1] + p) * vel[axis]], dim=2 if self.dim == 2 else 1)

    # restrictions of every cell to its faces: (left, right[, bottom, top])
    def traces(self, u):
        if self.dim == 1:
            return u @ self.eL, u @ self.eR
        return u @ self.eL, u @ self.eR, torch.einsum("yxvji,j->yxvi", u, self.eL), torch.einsum("yxvji,j->yxvi", u, self.eR)

    def speeds(self, u):
        """Frozen Einfeldt bounds (a, b) per face node, each face owned by the cell below it."""
        t, out = self.traces(u), []
        for axis in range(self.dim):
            l = t[2 * axis + 1]
            r = self.next(t[2 * axis], axis)
            cl, vl, pl, hl = self.primitive(l, self.dim)
            cr, vr, pr, hr = self.primitive(r, self.dim)
            sl, sr = cl[0].sqrt(), cr[0].sqrt()
            v = [(sl * a + sr * b) / (sl + sr) for a, b in zip(vl, vr)]
            H = (sl * hl + sr * hr) / (sl + sr)
            c = ((GAMMA - 1) * (H - 0.5 * sum(a * a for a in v))).sqrt()
            sndl, sndr = (GAMMA * pl / cl[0]).sqrt(), (GAMMA * pr / cr[0]).sqrt()
            a = SAFETY * torch.maximum((sndl - vl[axis]).clamp_min(0), c - v[axis])
            b = SAFETY * torch.maximum((vr[axis] + sndr).clamp_min(0), v[axis] + c)
            ax = 2 if self.dim == 2 else 1
            out.append((a.unsqueeze(ax), b.unsqueeze(ax)))
        return out

    def next(self, t, axis):
        return torch.roll(t, -1, 1 if self.dim == 2 and axis == 0 else 0)

    def prev(self, t, axis):
        return torch.roll(t, 1, 1 if self.dim == 2 and axis == 0 else 0)

    def points(self, u):
        if self.q == self.n:
            return u
        return u @ self.V.T if self.dim == 1 else torch.einsum("pj,yxvji,qi->yxvpq", self.V, u, self.V)

    def rate(self, u, sp):
        z = self.points(u)
        c, vel, p, _ = self.primitive(z, self.dim)
        snd, total = (GAMMA * p / c[0]).sqrt(), 0
        for axis in range(self.dim):
            s = torch.maximum(sp[axis][0], sp[axis][1])
            s = torch.maximum(s, self.prev(s, axis)).flatten(self.dim).amax(-1)
            total = total + torch.maximum(s, (vel[axis].abs() + snd).flatten(self.dim).amax(-1)) / (self.hx if axis == 0 else self.hy)
        return float(total.max())

    def volume(self, u):
        """minus the weak volume term"""
        z = self.points(u)
        if self.dim == 1:
            return -(self.flux(z, 0) @ self.wd)
        wv = self.qw[:, None] * self.V
        out = 0.5 * self.hy * torch.einsum("pj,yxvpq,qi->yxvji", wv, self.flux(z, 0), self.wd)
        return -(out + 0.5 * self.hx * torch.einsum("pj,yxvpq,qi->yxvji", self.wd, self.flux(z, 1), wv))

    def lift(self, f, side):
        e = self.eR if side % 2 else self.eL
        if self.dim == 1:
            return f[..., None] * e
        return f[..., :, None] * e if side < 2 else f[..., None, :] * e[:, None]

    def weight(self, axis):
        return 1.0 if self.dim == 1 else (self.fwx if axis == 0 else self.fwy)

    def residual(self, u, old, inv_tau, sp, other=None):
        """R(u); with `other` the neighbours' restrictions are held at those of that state."""
        r = self.mass * (u - old) * inv_tau
        if self.n > 1:
            r = r + self.volume(u)
        own = self.traces(u)
        ext = own if other is None else other
        for axis in range(self.dim):
            a, b = sp[axis]
            w, lo, hi = self.weight(axis), 2 * axis, 2 * axis + 1

            def hll(l, r_):
                return w * (b * self.flux(l, axis) + a * self.flux(r_, axis) + a * b * (l - r_)) / (a + b)

            up = hll(own[hi], self.next(ext[lo], axis))
            r = r + self.lift(up, hi)
            if other is None:
                down = self.prev(up, axis)
            else:
                ap, bp = self.prev(a, axis), self.prev(b, axis)
                left = self.prev(ext[hi], axis)
                down = w * (bp * self.flux(left, axis) + ap * self.flux(own[lo], axis) + ap * bp * (left - own[lo])) / (ap + bp)
            r = r - self.lift(down, lo)
        return r

    def taus(self, sp):
        """per side: the stabilisation of the face seen from the cell"""
        out = []
        for axis in range(self.dim):
            out += [self.prev(sp[axis][1], axis), sp[axis][0]]
        return out

    def local(self, u, inv_tau, sp):
        """the cell equation of the condensed form without its trace terms"""
        r = self.mass * u * inv_tau
        if self.n > 1:
            r = r + self.volume(u)
        for side, (t, tau) in enumerate(zip(self.traces(u), self.taus(sp))):
            r = r + self.lift(self.weight(side // 2) * ((1 if side % 2 else -1) * self.flux(t, side // 2) + tau * t), side)
        return r

    def blocks(self, f, u):
        """the m x m diagonal blocks of the Jacobian of f (cell-local in u) at u"""
        cells, eye = u.numel() // self.m, torch.eye(self.m, dtype=torch.float64, device=u.device)
        out = torch.empty(cells, self.m, self.m, dtype=torch.float64, device=u.device)
        column = torch.func.vmap(lambda v: torch.func.jvp(f, (u,), (v.expand(self.shape),))[1])
        some = max(1, min(self.m, 40_000_000 // u.numel()))
        for j in range(0, self.m, some):
            v = eye[j:j + some].reshape(-1, *self.shape[self.dim:])
            out[:, :, j:j + some] = column(v).reshape(-1, cells, self.m).permute(1, 2, 0)
        return out


def _gmres(mul, pre, b, tol=3e-15, restart=60, limit=900):
    """Restarted right-preconditioned GMRES in 64 bits (two Gram-Schmidt passes)."""
    x, r, norm, done, best = torch.zeros_like(b), b.clone(), float(b.norm()), 0, math.inf
    while done < limit:
        beta = float(r.norm())
        if beta <= tol * norm or beta > 0.5 * best:
            break
        best = beta
        basis = torch.empty(restart + 1, b.numel(), dtype=b.dtype, device=b.device)
        basis[0] = r / beta
        H, g, turns = np.zeros((restart + 1, restart)), np.zeros(restart + 1), []
        g[0] = beta
        for j in range(restart):
            w = mul(pre(basis[j]))
            h = basis[:j + 1] @ w
            w = w - h @ basis[:j + 1]
            h2 = basis[:j + 1] @ w
            w = w - h2 @ basis[:j + 1]
            last = w.norm()
            col = torch.cat([h + h2, last[None]]).cpu().numpy()
            basis[j + 1] = w / last
            done += 1
            for i, (c, s) in enumerate(turns):
                col[i], col[i + 1] = c * col[i] + s * col[i + 1], c * col[i + 1] - s * col[i]
            size = math.hypot(col[j], col[j + 1])
            turns.append((col[j] / size, col[j + 1] / size))
            H[:j + 1, j], H[j, j] = col[:j + 1], size
            g[j], g[j + 1] = turns[j][0] * g[j], -turns[j][1] * g[j]
            if abs(g[j + 1]) <= 0.3 * tol * norm:
                break
        y = np.linalg.solve(H[:j + 1, :j + 1], g[:j + 1])
        x = x + pre(_t(y) @ basis[:j + 1])
        r = b - mul(x)
    return x


class _Solve:
    """J(u)^{-1} (or J^{-T}) of the DG residual by GMRES over exact cell blocks."""

    def __init__(self, S, u, old, inv_tau, sp, transpose=False, lu=None):
        if lu is None:
            frozen = S.traces(u)
            A = S.blocks(lambda x: S.residual(x, old, inv_tau, sp, frozen), u)
            lu = torch.linalg.lu_factor(A.transpose(1, 2).contiguous() if transpose else A)
        self.lu, self.cells, self.m = lu, u.numel() // S.m, S.m
        f = lambda x: S.residual(x, old, inv_tau, sp)  # noqa: E731
        if transpose:
            back = torch.func.vjp(f, u)[1]
            self.mul = lambda v: back(v.reshape(S.shape))[0].reshape(-1)
        else:
            self.mul = lambda v: torch.func.jvp(f, (u,), (v.reshape(S.shape),))[1].reshape(-1)

    def pre(self, v):
        return torch.linalg.lu_solve(*self.lu, v.reshape(self.cells, self.m, 1)).reshape(-1)

    def __call__(self, b, tol=3e-15):
        return _gmres(self.mul, self.pre, b.reshape(-1), tol)


def _one_update(nx, ny, k, cfl, u):
    """The state after one backward-Euler Newton update from u: the full step, halved while it is
    inadmissible or the residual does not fall."""
    S = _Scheme(nx, ny, k)
    u = u.reshape(S.shape)
    sp = S.speeds(u)
    inv_tau = S.rate(u, sp) / cfl
    r = S.residual(u, u, inv_tau, sp)
    du = _Solve(S, u, u, inv_tau, sp)(-r).reshape(S.shape)

    def dual(x):
        return float((x * x / S.mass).sum().sqrt())

    def physical(x):
        c, _, p, _ = S.primitive(x, 2)
        return float(torch.minimum(c[0], p).min()) > 1e-13

    size, theta = dual(r), 1.0
    round_off = 128 * np.finfo(float).eps * (2 * float((u * u * S.mass).sum().sqrt()) * inv_tau + size)
    for _ in range(30):
        trial = u + theta * du
        if all(physical(x) for x in (trial, *S.traces(trial))):
            if dual(S.residual(trial, u, inv_tau, sp)) <= (1 - 1e-4 * theta) * size + round_off:
                break
        theta /= 2
    return trial.reshape(-1)


def _advance(case, u):
    S = _Scheme(case["nx"], case["ny"], case["k"], dim=case["dim"])
    A, B = STAGES[case["integrator"]]
    u = u.reshape(S.shape)
    for _ in range(case["steps"]):
        sp, lu = S.speeds(u), None
        step = case["cfl"] / S.rate(u, sp)
        slopes, x = [], u
        for i, row in enumerate(A):
            base = u + sum((step * a * s for a, s in zip(row, slopes)), torch.zeros_like(u))
            if i:
                sp = S.speeds(x)
            inv_tau = 1 / (row[i] * step)
            last = math.inf
            for _ in range(20):  # Newton with loose solves, to round-off; one preconditioner a step
                r = S.residual(x, base, inv_tau, sp)
                size = float(r.norm())
                if size > 0.1 * last:
                    break
                last = size
                solve = _Solve(S, x, base, inv_tau, sp, lu=lu)
                x, lu = x + solve(-r, 1e-4).reshape(S.shape), solve.lu
            slopes.append((x - base) * inv_tau)
        u = x if case["integrator"] == "be" else u + sum(step * b * s for b, s in zip(B, slopes))
    return u.reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        if sum(n * n * (4 * (k + 1) ** 2) ** 2 for k, n, _ in _members(case)) > 1.2e9:
            return None
        return [_one_update(n, n, k, case["cfl"], _state(n, n, k, seed + 101 * i)).cpu().numpy()
                for i, (k, n, _) in enumerate(_members(case))]
    nx, ny, k = case["nx"], case["ny"], case["k"]
    m = 4 * (k + 1) ** 2
    if kind == "advance":
        if nx * ny * m * m > 4e7:
            return None
        return _advance(case, _state(nx, ny, k, seed, case["dim"])).cpu().numpy()
    if kind not in ("residual", "jv", "jtw") and nx * ny * m * m > 6e8:
        return None
    u = _state(nx, ny, k, seed)
    if kind == "newton":
        return _one_update(nx, ny, k, case["cfl"], u)
    S = _Scheme(nx, ny, k, case.get("quad", 0))
    u, old = u.reshape(S.shape), _state(nx, ny, k, seed + 1).reshape(S.shape)
    sp = S.speeds(u)
    inv_tau = S.rate(u, sp) / case.get("cfl", 5.0)
    if kind == "residual":
        return S.residual(u, old, inv_tau, sp).reshape(-1)
    if kind == "condense":
        return _exact_condense(S, u, old, inv_tau, sp, seed)
    v = _direction(u.numel(), seed)
    f = lambda x: S.residual(x, old, inv_tau, sp)  # noqa: E731
    if kind == "jv":
        return torch.func.jvp(f, (u,), (v.reshape(S.shape),))[1].reshape(-1)
    if kind == "jtw":
        return torch.func.vjp(f, u)[1](v.reshape(S.shape))[0].reshape(-1)
    solve = _Solve(S, u, old, inv_tau, sp, transpose=kind == "adjoint")
    return solve(v) if kind == "adjoint" else solve.pre(v)


def _exact_condense(S, u, old, inv_tau, sp, seed):
    lam = _direction(2 * S.nx * S.ny * 4 * S.n, seed)
    faces = lam.reshape(2, S.ny, S.nx, 4, S.n)
    r = S.residual(u, old, inv_tau, sp)
    lu = torch.linalg.lu_factor(S.blocks(lambda x: S.local(x, inv_tau, sp), u))
    taus = S.taus(sp)
    side = [S.prev(faces[0], 0), faces[0], S.prev(faces[1], 1), faces[1]]
    B = sum(-S.lift(S.weight(i // 2) * taus[i] * side[i], i) for i in range(4))  # B lambda per cell
    both = torch.stack([B.reshape(-1, S.m), r.reshape(-1, S.m)], dim=2)
    X, y = (z.reshape(S.shape) for z in torch.linalg.lu_solve(*lu, both).unbind(2))

    def couple(x):
        """C x: the derivative of the cell's trace equations, per side"""
        t, dt = S.traces(u), S.traces(x)
        out = []
        for i in range(4):
            df = torch.func.jvp(lambda z: S.flux(z, i // 2), (t[i],), (dt[i],))[1]
            out.append(S.weight(i // 2) * ((1 if i % 2 else -1) * df + taus[i] * dt[i]))
        return out

    def gather(c):
        return [c[2 * a + 1] + S.next(c[2 * a], a) for a in range(2)]

    cx, cy = gather(couple(X)), gather(couple(y))
    diag = [-S.weight(a) * (sp[a][0] + sp[a][1]) for a in range(2)]
    return {"rhs": torch.stack(cy).reshape(-1), "schur": torch.stack([diag[a] * faces[a] - cx[a] for a in range(2)]).reshape(-1),
            "du": (-X - y).reshape(-1)}
