"""What is timed: solves through the library's public entry points, from one
step's latency on a few thousand triangles to a million-triangle mesh.

A case is a dict of plain values.  Its "kind" says which entry points it runs:

  solve     rkdg_set_state, rkdg_advance(steps), rkdg_get_state: one request of
            a solve, its state in pinned host memory before and after;
  steps     rkdg_set_state, then a loop of rkdg_step that reads dt and the
            residual monitor back every step, as the reference's loop does,
            then rkdg_get_state;
  residual  rkdg_set_state, rkdg_residual: one R(U) of a given state;
  batch     the rkdg_batch_* pack of uneven solves of mixed order;
  serve     requests submitted to a running rkdg_server_* loop and waited for.

Meshes come from meshgen with the seeds of its defaults; the initial state
(vortex strength, direction and place, shock position, perturbations) comes
from the seed.  Every result is the whole state (FP64 forms as doubles, FP32
forms as the floats they are computed in).
"""
import functools
import math

import numpy as np
import torch

from rkdg_heter_calculate_b200 import CUDARkdgSolver, capi, meshgen
from rkdg_heter_calculate_b200.batch import Batch
from rkdg_heter_calculate_b200.serve import Server

GAMMA = 1.4
MACH3 = (1.4, 3.0, 0.0, 1.0)  # (rho, u, v, p) of the wind-tunnel inflow
TVB_M = 50.0


# ------------------------------------------------------------------ cases --
def _solve(name, mesh, n, order, precision, steps, kind="solve", flux="hllc", nq=6, rk=3, cfl=0.2,
           limiter=False, basis="native"):
    nq, ng = (3, 2) if order == 1 else (nq, 3)
    return dict(name=name, kind=kind, mesh=mesh, n=n, order=order, nq=nq, ng=ng, flux=flux, rk=rk, cfl=cfl,
                limiter=limiter, precision=precision, steps=steps, basis=basis)


def listed():
    return [
        # the plain method on its own configuration: P1, LLF, SSP-RK2, 100 steps
        _solve("plain_p1_3200", "structured", 40, 1, "fp64", 100, flux="llf", rk=2, cfl=0.3),
        # the drop-in use: the reference's only method and basis, far field and
        # slip walls, on a mesh the size of its NACA 0012 input
        _solve("dropin_p2_9240", "obstacle", 68, 2, "fp64", 100, flux="llf", nq=7, cfl=0.18, basis="reference"),
        # a host loop that wants dt and the residual monitor after every step
        _solve("monitored_p2_28800", "structured", 120, 2, "fp64", 20, kind="steps", flux="llf", nq=7, cfl=0.18),
        # one residual evaluation, for callers with their own time integrator
        _solve("residual_p2_64800", "structured", 180, 2, "fp64", 1, kind="residual", flux="llf", nq=7,
               basis="reference"),
        # FP32 on a mesh that fits the device's caches, odd lattice
        _solve("vortex_p2_fp32_20402", "delaunay", 101, 2, "fp32", 200),
        # an ordinary FP64 solve, odd lattice (a ragged last tile)
        _solve("vortex_p2_fp64_132098", "delaunay", 257, 2, "fp64", 60),
        # the unstructured vortex at full size, FP64 and the compensated FP32 form
        _solve("vortex_p2_fp64_980000", "delaunay", 700, 2, "fp64", 40),
        _solve("vortex_p2_fp32c_980000", "delaunay", 700, 2, "fp32c", 200),
        # the Mach-3 step with the TVB limiter: FP64 coarse, FP32 with FP64 geometry and dt
        _solve("mach3_p1_fp64_32256", "step", 80, 1, "fp64", 100, flux="llf", cfl=0.3, limiter=True),
        _solve("mach3_p1_fp32_806400", "step", 400, 1, "fp32", 100, flux="llf", cfl=0.3, limiter=True),
        # uneven solves of both orders packed into one launch per stage
        dict(name="batch_24_mixed_fp32c", kind="batch", solves=24, n_min=50, n_max=225, precision="fp32c",
             steps=100),
        # requests of both orders and fluxes, with and without the limiter, in
        # flight together on a serving loop
        dict(name="serve_8_mixed_fp32", kind="serve", requests=8, n_min=32, n_max=120, precision="fp32", steps=96),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["vortex", "vortex", "vortex", "obstacle", "mach3", "mach3", "steps", "residual", "batch",
                       "serve"])
    order = rng.choice([1, 2, 2])
    precision = rng.choice(["fp64", "fp32", "fp32c"])
    flux = rng.choice(["llf", "hllc"])
    nq = rng.choice([6, 7])
    rk = rng.choice([2, 3, 3])
    steps = rng.randrange(20, 61)
    if what == "batch":
        return dict(kind="batch", solves=rng.randrange(3, 25), n_min=rng.randrange(30, 60),
                    n_max=rng.randrange(90, 226), precision=precision, steps=rng.randrange(20, 61))
    if what == "serve":
        return dict(kind="serve", requests=rng.randrange(2, 9), n_min=rng.randrange(24, 40),
                    n_max=rng.randrange(60, 121), precision=rng.choice(["fp32", "fp32c", "fp64"]),
                    steps=rng.randrange(40, 97))
    if what == "mach3":
        # the lattice spacing 1/n divides the step's height and place; in FP32
        # mesh sizes and lengths where the limiter's thresholds leave a result
        # that rounding does not decide
        n = 5 * (_log_int(rng, 6, 40) if precision == "fp64" else _log_int(rng, 30, 50))
        steps = steps if precision == "fp64" else rng.randrange(10, 31)
        c = _solve("", "step", n, 1, precision, steps, flux="llf", cfl=0.3, limiter=True)
    elif what == "obstacle":
        c = _solve("", "obstacle", 2 * _log_int(rng, 12, 90), order, precision, steps, flux=flux, nq=nq, cfl=0.18,
                   basis="reference")
    elif what == "steps":
        c = _solve("", "structured", _log_int(rng, 20, 350), order, precision, rng.randrange(5, 31), kind="steps",
                   flux=flux, nq=nq, rk=rk, limiter=rng.random() < 0.3)
    elif what == "residual":
        c = _solve("", "structured", _log_int(rng, 20, 500), order, "fp64", 1, kind="residual", flux=flux, nq=nq,
                   basis=rng.choice(["native", "reference"]))
    else:
        c = _solve("", rng.choice(["structured", "structured", "delaunay"]), _log_int(rng, 24, 500), order,
                   precision, steps, flux=flux, nq=nq, rk=rk, limiter=rng.random() < 0.25)
    del c["name"]
    return c


# ----------------------------------------------------------------- inputs --
@functools.lru_cache(maxsize=64)
def _mesh(kind, n):
    """The mesh a user's program has read: by its kind and size alone."""
    if kind == "structured":
        return meshgen.periodic_structured(n, n, jitter=0.15, seed=5)
    if kind == "delaunay":
        return meshgen.periodic_delaunay(n, jitter=0.3, seed=2)
    if kind == "obstacle":
        return meshgen.box_with_obstacle(n, seed=7)
    return meshgen.forward_step(1.0 / n, jitter=0.3, seed=3)


def _conservative(rho, u, v, p):
    return torch.stack([rho, rho * u, rho * v, p / (GAMMA - 1) + 0.5 * rho * (u * u + v * v)])


def _flow(mesh_kind, n, seed):
    """(far-field state, the initial flow as a function of points) of a seed."""
    r = np.random.default_rng(seed)
    if mesh_kind in ("structured", "delaunay"):  # an isentropic vortex on [0, 10]^2
        beta, th = r.uniform(1.0, 5.0), r.uniform(0.0, 2 * math.pi)
        xc, yc = r.uniform(3.0, 7.0, 2)
        u0, v0 = math.sqrt(2) * math.cos(th), math.sqrt(2) * math.sin(th)

        def f(x, y):
            dx, dy = x - xc, y - yc
            e = torch.exp(0.5 * (1.0 - dx * dx - dy * dy))
            t = 1.0 - (GAMMA - 1) * beta * beta / (8 * GAMMA * math.pi ** 2) * e * e
            rho = t ** (1 / (GAMMA - 1))
            k = beta / (2 * math.pi)
            return _conservative(rho, u0 - k * dy * e, v0 + k * dx * e, rho ** GAMMA)
        prim = (1.0, u0, v0, 1.0)
    elif mesh_kind == "obstacle":  # Mach 0.4 past a block, with a pulse on its way
        al = math.radians(5.0)
        ut = 0.4 * math.sqrt(GAMMA)
        prim = (1.0, ut * math.cos(al), ut * math.sin(al), 1.0)
        xc, yc = r.uniform(-6.0, -3.0), r.uniform(-2.0, 2.0)
        amp = r.uniform(0.02, 0.1, 4)

        def f(x, y):
            e = torch.exp(-((x - xc) ** 2 + (y - yc) ** 2) / 4.0)
            return _conservative(prim[0] * (1 + amp[0] * e), prim[1] + amp[1] * e, prim[2] - amp[2] * e,
                                 prim[3] * (1 + amp[3] * e))
    else:  # Mach-3 inflow meeting a normal shock ahead of the step, wavy along y
        prim = MACH3
        xs, a, ph = r.uniform(0.3, 0.5), r.uniform(0.01, 0.05), r.uniform(0.0, 2 * math.pi)
        jump = (1.4 * 27 / 7, 7.0 / 9.0, 0.0, 31.0 / 3.0)  # Rankine-Hugoniot at Mach 3

        def f(x, y):
            s = 0.5 * (1 + torch.tanh((x - xs - a * torch.sin(2 * math.pi * y + ph)) * (0.5 * n)))
            q = [p0 + (p1 - p0) * s for p0, p1 in zip(prim, jump)]
            return _conservative(q[0], q[1], q[2], q[3])
    rho, u, v, p = prim
    return (rho, rho * u, rho * v, p / (GAMMA - 1) + 0.5 * rho * (u * u + v * v)), f


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


@functools.lru_cache(maxsize=4)
def _tables(order, nq, ng):
    return _Tables(order, nq, ng, _device())


def _initial(mesh, flow, order, basis):
    """Coefficients [4][nb][T] (doubles on the device) of the projected flow."""
    tb = _tables(order, 6 if order == 2 else 3, 3 if order == 2 else 2)
    geo = _Geometry(mesh, _device())
    xi = torch.as_tensor(tb.vol_pts, device=geo.c.device)
    c = geo.c
    x = c[:, 0, 0] + xi[:, :1] * (c[:, 1, 0] - c[:, 0, 0]) + xi[:, 1:] * (c[:, 2, 0] - c[:, 0, 0])
    y = c[:, 0, 1] + xi[:, :1] * (c[:, 1, 1] - c[:, 0, 1]) + xi[:, 1:] * (c[:, 2, 1] - c[:, 0, 1])
    U = torch.matmul((tb.phi * tb.vw[:, None]).T, flow(x, y))
    return _from_native(U, geo, order) if basis == "reference" else U


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=torch.cuda.is_available())
    h.copy_(t)
    return h


def _ptr(t):
    return capi.dptr(t.numpy())


def _members(case):
    """The solves of a batch or the requests of a serving case: sizes log-uniform, orders alternating."""
    k = case["solves"] if case["kind"] == "batch" else case["requests"]
    lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
    got = []
    for i in range(k):
        n = int(round(math.exp(lo + (hi - lo) * ((0.5 + i * 0.6180339887) % 1.0))))
        if case["kind"] == "serve" and i % 2:  # P1, LLF, with the limiter
            got.append(dict(mesh="structured", n=n, order=1, flux="llf", limiter=True, steps=case["steps"]))
        else:
            order = 1 if (case["kind"] == "batch" and i % 2) else 2
            got.append(dict(mesh="structured", n=n, order=order, flux="hllc", limiter=False, steps=case["steps"]))
    for m in got:
        m.update(rk=3, cfl=0.2, **(dict(nq=3, ng=2) if m["order"] == 1 else dict(nq=6, ng=3)))
    return got


def _member_inputs(case, seed):
    got = []
    for i, m in enumerate(_members(case)):
        mesh = _mesh(m["mesh"], m["n"])
        far, flow = _flow(m["mesh"], m["n"], 1000 * seed + i)
        got.append((m, mesh, far, _initial(mesh, flow, m["order"], "native")))
    return got


def prepare(case, seed):
    if case["kind"] in ("batch", "serve"):
        members = _member_inputs(case, seed)
        s = {"case": case, "U0": [_pinned(U) for _, _, _, U in members], "members": [m for m, _, _, _ in members],
             "far": [far for _, _, far, _ in members], "meshes": [mesh for _, mesh, _, _ in members]}
        if case["kind"] == "batch":
            s["batch"] = Batch(s["meshes"], [m["order"] for m in s["members"]], precision=case["precision"],
                               flux="hllc", rk=3, nq=6, gamma=GAMMA, cfl=0.2, farfields=s["far"])
            if len(set(m["order"] for m in s["members"])) == 2:
                s["batch"].set_shape(0, 2)  # the two orders as concurrent launches
        else:
            s["server"] = Server(1 << 30, max_slots=16, precision=case["precision"], flux="llf", rk=3, gamma=GAMMA,
                                 cfl=0.2, tvb_m=TVB_M)
            s["t_final"] = [(m["steps"] - 0.5) * _Plain(mesh, m, far, _device()).dt(U) for m, mesh, far, U in members]
        outs = s["U0"]
    else:
        mesh = _mesh(case["mesh"], case["n"])
        far, flow = _flow(case["mesh"], case["n"], seed)
        U0 = _pinned(_initial(mesh, flow, case["order"], case["basis"]))
        solver = CUDARkdgSolver(mesh, order=case["order"], nq=case["nq"], ng=case["ng"], flux=case["flux"],
                                limiter="tvb" if case["limiter"] else None, rk=case["rk"],
                                precision=case["precision"], gamma=GAMMA, cfl=case["cfl"], tvb_m=TVB_M,
                                farfield=far)
        basis = capi.BASIS_REFERENCE if case["basis"] == "reference" else capi.BASIS_NATIVE
        s = {"case": case, "U0": U0, "solver": solver, "basis": basis}
        outs = [U0]
    s["out"] = [_pinned(torch.zeros_like(u)) for u in outs]
    # the FP32 forms' results as the floats they are computed in
    s["out32"] = None if case["precision"] == "fp64" else [torch.zeros(u.shape, dtype=torch.float32) for u in outs]
    return s


# -------------------------------------------------------------- the passes --
def _results(s):
    if s["out32"] is None:
        return s["out"]
    for a, b in zip(s["out32"], s["out"]):
        a.copy_(b)
    return s["out32"]


def run(s):
    case, L = s["case"], capi.lib()
    if case["kind"] == "batch":
        b = s["batch"]
        for i, U in enumerate(s["U0"]):
            capi.check(L.rkdg_batch_set_state(b.h, i, _ptr(U), b.T[i]))
        b.advance(case["steps"])
        for i, U in enumerate(s["out"]):
            capi.check(L.rkdg_batch_get_state(b.h, i, _ptr(U), b.T[i]))
        return _results(s)
    if case["kind"] == "serve":
        srv = s["server"]
        ids = [srv.submit(mesh, m["order"], U.numpy(), tf, farfield=far, limiter=m["limiter"], flux=m["flux"])
               for mesh, m, U, tf, far in zip(s["meshes"], s["members"], s["U0"], s["t_final"], s["far"])]
        got = [srv.wait(i).state for i in ids]
        return got if s["out32"] is None else [u.astype(np.float32) for u in got]
    sv = s["solver"]
    capi.check(L.rkdg_set_state(sv.h, _ptr(s["U0"]), sv.T, s["basis"]))
    if case["kind"] == "residual":
        capi.check(L.rkdg_residual(sv.h, _ptr(s["out"][0]), sv.T, s["basis"]))
        return _results(s)
    history = []
    if case["kind"] == "steps":
        for _ in range(case["steps"]):
            dt, monitor = sv.step()
            history.append((dt, monitor[0], monitor[1]))
    else:
        sv.advance(case["steps"])
    capi.check(L.rkdg_get_state(sv.h, _ptr(s["out"][0]), sv.T, s["basis"]))
    if not history:
        return _results(s)
    return [*_results(s), np.array(history, dtype=np.float64 if s["out32"] is None else np.float32)]


# -------------------------------------------------------------------- work --
def _elements(case):
    n = case["n"]
    if case["mesh"] in ("structured", "delaunay"):
        return 2 * n * n
    if case["mesh"] == "obstacle":
        return 2 * n * n - 8
    return 2 * (round(3 * n) * n - round(2.4 * n) * round(0.2 * n))


def _work(case):
    """Per element and stage: the stage input read and the output written, U^n
    read where the stage combines with it, J^-1 (32 B) and the edges' sources
    and lists (24 B); the means' low parts in fp32c.  Plus the state in and out."""
    T, nb = _elements(case), 3 if case["order"] == 1 else 6
    nq, ng, rk = case["nq"], case["ng"], case["rk"]
    steps = case["steps"]
    host = 2 * 8 * 4 * nb * T
    w = 8 if case["precision"] == "fp64" else 4
    rows = 4 * nb * w + (16 if case["precision"] == "fp32c" else 0)
    volume = nq * (8 * nb + 40 + 8 * (2 * nb - 3))
    edges = 3 * ng * 8 * nb + 1.5 * ng * (110 if case["flux"] == "hllc" else 70) + 3 * ng * 8 * nb
    stage = volume + edges + 16 * nb + (60 if case["limiter"] else 0)
    if case["kind"] == "residual":
        return {"bytes": T * (2 * rows + 56) + host, "flops": T * stage}
    return {"bytes": steps * T * (rk * (2 * rows + 56) + (rk - 1) * rows) + host, "flops": steps * rk * T * stage}


def work(case):
    if case["kind"] in ("batch", "serve"):
        got = [_work(dict(m, kind="solve", precision=case["precision"])) for m in _members(case)]
        return {k: sum(g[k] for g in got) for k in ("bytes", "flops")}
    return _work(case)


# ------------------------------------- the same in 64 bits, in plain torch --
_REF_EDGE = (((1.0, 0.0), (0.0, 1.0)), ((0.0, 1.0), (0.0, 0.0)), ((0.0, 0.0), (1.0, 0.0)))


def _rule(nq):
    if nq == 7:
        a, b, c, d = 0.797426985353087, 0.101286507323456, 0.059715871789770, 0.470142064105115
        pts = [(1 / 3, 1 / 3), (b, b), (a, b), (b, a), (d, d), (c, d), (d, c)]
        return pts, [0.225] + [0.125939180544827] * 3 + [0.132394152788506] * 3
    if nq == 6:
        a, b = 0.44594849091596488631832925388305, 0.09157621350977074345957146340220
        wa, wb = 0.22338158967801146569500700843312, 0.10995174365532186763832632490021
        pts = [p for c in (a, b) for p in ((c, c), (1 - 2 * c, c), (c, 1 - 2 * c))]
        return pts, [wa] * 3 + [wb] * 3
    return [(1 / 6, 1 / 6), (2 / 3, 1 / 6), (1 / 6, 2 / 3)], [1 / 3] * 3


class _Tables:
    """Values of the reference-element orthonormal basis at the rules' points."""

    def __init__(self, order, nq, ng, dev):
        nb = 3 if order == 1 else 6
        ex = ((0, 0), (1, 0), (0, 1), (2, 0), (1, 1), (0, 2))
        f = math.factorial
        gram = np.array([[2 * f(a[0] + b[0]) * f(a[1] + b[1]) / f(a[0] + b[0] + a[1] + b[1] + 2) for b in ex]
                         for a in ex])
        K = np.linalg.inv(np.linalg.cholesky(gram))

        def psi(p):
            x, y = p[:, 0], p[:, 1]
            return (np.stack([np.ones_like(x), x, y, x * x, x * y, y * y], 1) @ K.T)[:, :nb]

        def grad(p):
            x, y = p[:, 0], p[:, 1]
            z, o = np.zeros_like(x), np.ones_like(x)
            return ((np.stack([z, o, z, 2 * x, y, z], 1) @ K.T)[:, :nb],
                    (np.stack([z, z, o, z, x, 2 * y], 1) @ K.T)[:, :nb])
        pts, w = _rule(nq)
        pts, w = np.array(pts), np.array(w)
        if ng == 3:
            cp = 0.5 + math.sqrt(15.0) / 10.0
            s, ew = np.array([1 - cp, 0.5, cp]), np.array([0.55555555555556, 0.88888888888889, 0.55555555555556]) / 2
        else:
            s, ew = np.array([0.5 - math.sqrt(3.0) / 6, 0.5 + math.sqrt(3.0) / 6]), np.array([0.5, 0.5])
        on_edges = np.array([[(1 - g) * np.array(a) + g * np.array(b) for g in s] for a, b in _REF_EDGE])
        e = psi(on_edges.reshape(-1, 2))
        m = psi(np.array([[0.5, 0.5], [0.0, 0.5], [0.5, 0.0]]))[:, 1:3]

        def t(a):
            return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)
        self.nb, self.ng = nb, ng
        self.vol_pts, self.vw, self.phi = pts, t(w), t(psi(pts))
        gx, gy = grad(pts)
        self.dx_w, self.dy_w = t((gx * w[:, None]).T), t((gy * w[:, None]).T)
        self.edge, self.edge_w = t(e), t((e.reshape(3, ng, nb) * ew[None, :, None]).reshape(3 * ng, nb).T)
        self.mid, self.mid_inv = t(m), t(np.linalg.solve(m.T @ m, m.T))


class _Geometry:
    def __init__(self, mesh, dev):
        self.c = torch.as_tensor(mesh.vertices[mesh.tris], device=dev)
        a, b = self.c[:, 1] - self.c[:, 0], self.c[:, 2] - self.c[:, 0]
        det = a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0]
        self.r0 = (b[:, 1] / det, -b[:, 0] / det)
        self.r1 = (-a[:, 1] / det, a[:, 0] / det)
        self.area = 0.5 * det
        # edge normals over the area, their lengths over the area, unit normals
        nx = torch.stack([2 * (self.r0[0] + self.r1[0]), -2 * self.r0[0], -2 * self.r1[0]])
        ny = torch.stack([2 * (self.r0[1] + self.r1[1]), -2 * self.r0[1], -2 * self.r1[1]])
        self.len = torch.sqrt(nx * nx + ny * ny)
        self.nx, self.ny = nx / self.len, ny / self.len


def _basis_change(geo, order):
    """C [T][i][j]: the reference's per-element basis function i (Gram-Schmidt
    of 1, X, Y, X^2, XY, Y^2 in centred coordinates over sqrt(area), not
    normalised) on the native functions j."""
    nb = 3 if order == 1 else 6
    tb = _tables(2, 6, 3)
    xi = torch.as_tensor(tb.vol_pts, device=geo.c.device)
    c = geo.c - geo.c.mean(dim=1, keepdim=True)
    s = 1 / torch.sqrt(geo.area)
    X = s[:, None] * (c[:, :1, 0] + xi[:, 0] * (c[:, 1:2, 0] - c[:, :1, 0]) + xi[:, 1] * (c[:, 2:, 0] - c[:, :1, 0]))
    Y = s[:, None] * (c[:, :1, 1] + xi[:, 0] * (c[:, 1:2, 1] - c[:, :1, 1]) + xi[:, 1] * (c[:, 2:, 1] - c[:, :1, 1]))
    m = torch.stack([torch.ones_like(X), X, Y, X * X, X * Y, Y * Y], dim=1)  # [T][6][q]
    chol = torch.linalg.cholesky(torch.matmul(m * tb.vw, m.transpose(1, 2)))
    phi = torch.linalg.solve_triangular(chol, m, upper=False) * torch.diagonal(chol, dim1=1, dim2=2)[:, :, None]
    return torch.matmul(phi * tb.vw, tb.phi)[:, :nb, :nb]


def _from_native(U, geo, order):
    C = _basis_change(geo, order)
    return torch.einsum("vjt,tij->vit", U, C / (C * C).sum(dim=2, keepdim=True)).contiguous()


def _to_native(U, geo, order):
    return torch.einsum("vit,tij->vjt", U, _basis_change(geo, order)).contiguous()


class _Plain:
    """The method as it is written down: one field at a time, in doubles."""

    def __init__(self, mesh, case, far, dev):
        self.tb, self.g, self.case = _tables(case["order"], case["nq"], case["ng"]), _Geometry(mesh, dev), case
        self.far = torch.tensor(far, dtype=torch.float64, device=dev)
        T, ng = len(mesh.tris), case["ng"]
        nb = mesh.neighbours.astype(np.int64)
        me = np.arange(T)
        se = np.zeros((3, T), dtype=np.int64)
        for k in range(3):
            for j in range(3):
                se[k][(nb[nb[:, k], j] == me) & (nb[:, k] >= 0)] = j
        src = np.where(nb.T < 0, me, nb.T)
        own = np.arange(3)[:, None]
        at = [np.where(nb.T < 0, (own * ng + g) * T + me, (se * ng + ng - 1 - g) * T + src) for g in range(ng)]
        self.nbr = torch.as_tensor(src, device=dev)
        self.other = torch.as_tensor(np.stack(at, 1), device=dev)  # [3][ng][T]
        self.tag = torch.as_tensor(np.where(nb.T < 0, mesh.bc.T, 0), device=dev)
        self.walls = bool((self.tag > 0).any())
        if case["limiter"]:
            self._limiter_geometry(se, nb)

    def _ghost(self, u, v, tag, nx, ny):
        """Across a boundary edge the far field, a copy or the mirrored state; u itself inside."""
        if not self.walls:
            return v
        far = self.far.reshape(4, *([1] * (u.dim() - 1)))
        mn = 2 * (u[1] * nx + u[2] * ny)
        wall = torch.stack([u[0], u[1] - mn * nx, u[2] - mn * ny, u[3]])
        return torch.where(tag == 0, v, torch.where(tag == 1, far, torch.where(tag == 2, u, wall)))

    @staticmethod
    def _pressure(u):
        return (GAMMA - 1) * (u[3] - 0.5 * (u[1] * u[1] + u[2] * u[2]) / u[0])

    def _normal(self, u, nx, ny):
        p = self._pressure(u)
        q = (u[1] * nx + u[2] * ny) / u[0]
        return torch.stack([u[0] * q, u[1] * q + p * nx, u[2] * q + p * ny, (u[3] + p) * q]), p, q

    def _flux(self, L, R, mL, mR, nx, ny):
        FL, pL, qL = self._normal(L, nx, ny)
        FR, pR, qR = self._normal(R, nx, ny)
        if self.case["flux"] == "llf":
            m = 0.5 * (mL + mR)
            a = ((m[1] * nx[:, 0] + m[2] * ny[:, 0]) / m[0]).abs() + torch.sqrt(GAMMA * self._pressure(m) / m[0])
            return 0.5 * (FL + FR - a[:, None] * (R - L))
        cL, cR = torch.sqrt(GAMMA * pL / L[0]), torch.sqrt(GAMMA * pR / R[0])
        SL, SR = torch.minimum(qL - cL, qR - cR), torch.maximum(qL + cL, qR + cR)
        dL, dR = L[0] * (SL - qL), R[0] * (SR - qR)
        SM = (pR - pL + dL * qL - dR * qR) / (dL - dR)
        left = SM >= 0
        S, d, p, q = (torch.where(left, a, b) for a, b in ((SL, SR), (dL, dR), (pL, pR), (qL, qR)))
        ps = p + d * (SM - q)
        star = (SM * (S * torch.where(left, L, R) - torch.where(left, FL, FR))
                + S * ps * torch.stack([torch.zeros_like(S), nx.expand_as(S), ny.expand_as(S), SM])) / (S - SM)
        return torch.where(SL >= 0, FL, torch.where(SR <= 0, FR, star))

    def rate(self, U):
        """dU/dt of native coefficients [4][nb][T]."""
        tb, g, ng = self.tb, self.g, self.case["ng"]
        w = torch.matmul(tb.phi, U)
        p = self._pressure(w)
        u, v = w[1] / w[0], w[2] / w[0]
        F = torch.stack([w[1], w[1] * u + p, w[2] * u, (w[3] + p) * u])
        G = torch.stack([w[2], w[1] * v, w[2] * v + p, (w[3] + p) * v])
        out = torch.matmul(tb.dx_w, F * g.r0[0] + G * g.r0[1]) + torch.matmul(tb.dy_w, F * g.r1[0] + G * g.r1[1])
        del w, F, G
        tr = torch.matmul(tb.edge, U)
        L = tr.reshape(4, 3, ng, -1)
        nx, ny = g.nx[:, None], g.ny[:, None]
        R = self._ghost(L, tr.reshape(4, -1)[:, self.other], self.tag[:, None], nx, ny)
        mean = U[:, :1].expand(4, 3, -1)
        far_mean = self._ghost(mean, U[:, 0][:, self.nbr], self.tag, g.nx, g.ny)
        f = self._flux(L, R, mean, far_mean, nx, ny) * g.len[:, None]
        return out - torch.matmul(tb.edge_w, f.reshape(4, 3 * ng, -1))

    def dt(self, U):
        m = U[:, 0]
        speed = torch.sqrt(m[1] ** 2 + m[2] ** 2) / m[0] + torch.sqrt(GAMMA * self._pressure(m) / m[0])
        return self.case["cfl"] / float((speed * self.g.len.sum(dim=0)).max())

    def _limiter_geometry(self, se, nb):
        """Cockburn and Shu's (alpha, beta) and pairing edge of every edge."""
        c = self.g.c.cpu().numpy()
        b0 = c.mean(axis=1)
        mids = np.stack([0.5 * (c[:, (k + 1) % 3] + c[:, (k + 2) % 3]) for k in range(3)])
        bk = np.empty_like(mids)
        for k in range(3):
            n, j = nb[:, k], se[k]
            inside = mids[k] + b0[n] - mids[j, n]
            e = c[:, (k + 2) % 3] - c[:, (k + 1) % 3]
            nrm = np.stack([e[:, 1], -e[:, 0]], 1) / np.linalg.norm(e, axis=1)[:, None]
            mirror = b0 + 2 * ((mids[k] - b0) * nrm).sum(1)[:, None] * nrm
            bk[k] = np.where((n >= 0)[:, None], inside, mirror)
        r, d = mids - b0, bk - b0
        ab, pair = np.zeros((3, 2, len(c))), np.zeros((3, len(c)), dtype=np.int64)
        for k in range(3):
            best = np.full(len(c), -1e300)
            for s in (1, 2):
                j = (k + s) % 3
                det = d[k][:, 0] * d[j][:, 1] - d[k][:, 1] * d[j][:, 0]
                al = (r[k][:, 0] * d[j][:, 1] - r[k][:, 1] * d[j][:, 0]) / det
                be = (d[k][:, 0] * r[k][:, 1] - d[k][:, 1] * r[k][:, 0]) / det
                better = np.minimum(al, be) > best + 1e-14
                best = np.where(better, np.minimum(al, be), best)
                ab[k, 0], ab[k, 1] = np.where(better, al, ab[k, 0]), np.where(better, be, ab[k, 1])
                pair[k] = np.where(better, j, pair[k])
        dev = self.g.c.device
        self.ab, self.pair = torch.as_tensor(ab, device=dev), torch.as_tensor(pair, device=dev)
        r = torch.as_tensor(r, device=dev)
        r2 = (r * r).sum(dim=2)
        self.dir, self.thr = (r / torch.sqrt(r2)[:, :, None]).permute(2, 0, 1), TVB_M * 4 * r2  # [2][3][T], [3][T]

    def limit(self, U):
        tb = self.tb
        mean = U[:, 0]
        tilde = torch.matmul(tb.mid, U[:, 1:3])  # [4][3][T]
        near = self._ghost(mean[:, None].expand(4, 3, -1), mean[:, self.nbr], self.tag, self.g.nx, self.g.ny)
        step = near - mean[:, None]
        dbar = 1.5 * (self.ab[:, 0] * step + self.ab[:, 1] * torch.gather(step, 1, self.pair.expand(4, 3, -1)))
        nx, ny = self.dir
        vx, vy = mean[1] / mean[0], mean[2] / mean[0]
        p = self._pressure(mean)
        c = torch.sqrt(GAMMA * p / mean[0])
        H, k2 = (mean[3] + p) / mean[0], 0.5 * (vx * vx + vy * vy)
        b1 = (GAMMA - 1) / (c * c)
        b2 = b1 * k2
        q, qt = vx * nx + vy * ny, vy * nx - vx * ny

        def chars(a):
            ac = a[1] * nx + a[2] * ny
            common = b2 * a[0] - b1 * (vx * a[1] + vy * a[2] - a[3])
            return torch.stack([0.5 * (common + (q * a[0] - ac) / c), a[0] - common,
                                -qt * a[0] - ny * a[1] + nx * a[2], 0.5 * (common - (q * a[0] - ac) / c)])
        wt, wd = chars(tilde), chars(dbar)
        minmod = torch.where((wt > 0) & (wd > 0), torch.minimum(wt, wd),
                             torch.where((wt < 0) & (wd < 0), torch.maximum(wt, wd), torch.zeros_like(wt)))
        w = torch.where(wt.abs() <= self.thr, wt, minmod)
        limited = (w != wt).any(dim=0).any(dim=0)
        both = w[0] + w[1] + w[3]
        delta = torch.stack([both, vx * both + c * nx * (w[3] - w[0]) - ny * w[2],
                             vy * both + c * ny * (w[3] - w[0]) + nx * w[2],
                             H * (w[0] + w[3]) + q * c * (w[3] - w[0]) + k2 * w[1] + qt * w[2]])
        pos, neg = delta.clamp(min=0).sum(dim=1), (-delta).clamp(min=0).sum(dim=1)
        tp = torch.where(pos > 0, (neg / pos).clamp(max=1), torch.ones_like(pos))
        tn = torch.where(neg > 0, (pos / neg).clamp(max=1), torch.ones_like(neg))
        fixed = tp[:, None] * delta.clamp(min=0) - tn[:, None] * (-delta).clamp(min=0)
        delta = torch.where((delta.sum(dim=1) != 0)[:, None], fixed, delta)
        new = torch.zeros_like(U)
        new[:, 0] = mean
        new[:, 1:3] = torch.matmul(tb.mid_inv, delta)
        return torch.where(limited, new, U)

    def step(self, U, dt):
        U0 = U
        for a in ((0.0, 0.5) if self.case["rk"] == 2 else (0.0, 0.75, 1 / 3)):
            U = a * U0 + (1 - a) * (U + dt * self.rate(U))
            if self.case["limiter"]:
                U = self.limit(U)
        return U


def exact(case, seed):
    dev = _device()
    if case["kind"] in ("batch", "serve"):
        got = []
        for m, mesh, far, U in _member_inputs(case, seed):
            s = _Plain(mesh, m, far, dev)
            if case["kind"] == "batch":
                for _ in range(case["steps"]):
                    U = s.step(U, s.dt(U))
            else:
                t, end = 0.0, (m["steps"] - 0.5) * s.dt(U)
                while t < end:
                    dt = min(s.dt(U), end - t)
                    U, t = s.step(U, dt), (end if dt >= end - t else t + dt)
            got.append(U)
        return got
    mesh = _mesh(case["mesh"], case["n"])
    far, flow = _flow(case["mesh"], case["n"], seed)
    U = _initial(mesh, flow, case["order"], case["basis"])
    s = _Plain(mesh, case, far, dev)
    ref = case["basis"] == "reference"
    if ref:
        U = _to_native(U, s.g, case["order"])
    if case["kind"] == "residual":
        R = s.rate(U) * s.g.area
        return [torch.einsum("vjt,tij->vit", R, _basis_change(s.g, case["order"])) if ref else R]
    history = []
    for _ in range(case["steps"]):
        dt = s.dt(U)
        new = s.step(U, dt)
        d = (new[:, 0] - U[:, 0]).abs().amax(dim=1)
        history.append((dt, float(d[0]), float(d[3])))
        U = new
    out = [_from_native(U, s.g, case["order"]) if ref else U]
    return out + [torch.tensor(history, dtype=torch.float64)] if case["kind"] == "steps" else out
