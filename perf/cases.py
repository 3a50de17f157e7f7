"""Timed cases of the quantum-dot framework: what its users have it do.

A case is a dict of plain values; ``kind`` names the call it makes:

``dot``       the drop-in ``CythonSchrodingerSolver(mesh, m*, V).solve(k)`` on one dot,
              host callbacks to host levels: the latency of one interactive call.
``sweep``     assembly and batched solve of many dots of uneven sizes (parameter sweeps,
              the framework's headline work); returns the levels.
``junction``  assembly and batched solve of one mesh under many bias potentials, the
              Schrodinger half of a self-consistent iteration; returns the levels.
``assemble``  H, M (and the absorbing term) of one mesh from nodal V and per-element 1/m*.
``batch``     H and M of a packed batch of dots (what a sweep assembles per step).
``poisson``   the Poisson half of a self-consistent iteration, one or many biases.
``products``  A X and M X of the open-system pencil for a block of complex vectors.
``open``      the open-system eigensolve: the k complex levels nearest a shift.
``interp``    a nodal field evaluated at many points (plots, resampling between meshes).
``adjoint``   gradients of a loss of the levels with respect to V and 1/m*, from
              eigenvectors in hand (inverse design).

The solves return their levels: at the tolerances that users solve to, single eigenvectors
are free in sign, free inside near-degenerate groups, and far less converged than levels.
What is computed from eigenvectors is covered by ``adjoint``, from given vectors.
"""
from __future__ import annotations

import math

import numpy as np
import torch

HBAR, M_E, Q_E = 1.054571817e-34, 9.1093837015e-31, 1.602176634e-19
C0 = HBAR * HBAR / (2.0 * M_E) / Q_E * 1e18        # hbar^2 / (2 m0) in eV nm^2
EPS0 = 8.854187817e-12
DEV = "cuda"


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # one dot through the drop-in call (P1 100 x 50 cells, 10 levels)
        dict(name="dot_p1", kind="dot", nx=100, ny=50, k=10),
        # a quarter of the 256-dot P2 sweep: nx ~ U{40..240}, ny = nx / 2, 8 levels
        dict(name="sweep_p2_64", kind="sweep", order=2, dots=64, lo=40, hi=240, k=8,
             precision="mixed"),
        # a few dots in the plain double-precision form, 8 levels
        dict(name="sweep_p2_fp64", kind="sweep", order=2, dots=8, lo=40, hi=120, k=8,
             precision="fp64"),
        # Schrodinger half of the p-n junction's iteration: 64 biases, 10 levels
        dict(name="junction_p1_64", kind="junction", nx=300, ny=100, biases=64, k=10),
        # the open-system pencil with its absorbing layer, P2 400 x 200 cells
        dict(name="assemble_p2_cap", kind="assemble", order=2, nx=400, ny=200, cap=True),
        # what the quarter sweep assembles
        dict(name="batch_p2_64", kind="batch", order=2, dots=64, lo=40, hi=240),
        # one right-hand side (the drop-in Poisson solve) and 64 biases
        dict(name="poisson_1", kind="poisson", nx=100, ny=50, nrhs=1),
        dict(name="poisson_64", kind="poisson", nx=300, ny=100, nrhs=64),
        # block products of the open system (48 complex columns, double precision)
        dict(name="products_fp64", kind="products", nx=400, ny=200, b=48, fp32=False),
        # the open-system solve at 200 x 100 cells, 20 levels
        dict(name="open_p2", kind="open", nx=200, ny=100, k=20, precision="mixed"),
        # 16.8M random points of one field, values only
        dict(name="interp_random", kind="interp", order=2, nx=400, ny=200, points=1 << 24,
             fields=1, ordered=False, gradient=False),
        # gradients of 4 levels on the P3 150 x 75-cell dot
        dict(name="adjoint_p3", kind="adjoint", order=3, nx=150, ny=75, states=4, open=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dot", "sweep", "junction", "assemble", "batch", "poisson", "poisson",
                       "products", "open", "interp", "interp", "adjoint"])
    if kind == "dot":
        nx = _log_int(rng, 40, 160)
        return dict(kind=kind, nx=nx, ny=rng.randint(max(20, nx // 3), nx), k=rng.randint(2, 12))
    if kind == "sweep":
        lo = rng.randint(40, 120)
        return dict(kind=kind, order=rng.choice([1, 2, 2, 3]), dots=_log_int(rng, 1, 24), lo=lo,
                    hi=lo + rng.randint(0, 60), k=rng.randint(4, 10),
                    precision=rng.choice(["mixed", "mixed", "fp64"]))
    if kind == "junction":
        nx = rng.randint(80, 300)
        return dict(kind=kind, nx=nx, ny=rng.randint(40, 100), biases=_log_int(rng, 1, 64),
                    k=rng.randint(4, 10))
    if kind == "assemble":
        order = rng.choice([1, 2, 3])
        nx = _log_int(rng, 40, 900 // order)
        return dict(kind=kind, order=order, nx=nx, ny=rng.randint(nx // 3, nx // 2),
                    cap=rng.choice([True, False]))
    if kind == "batch":
        lo = rng.randint(40, 120)
        return dict(kind=kind, order=rng.choice([1, 2, 3]), dots=_log_int(rng, 2, 24), lo=lo,
                    hi=lo + rng.randint(0, 60))
    if kind == "poisson":
        nx = _log_int(rng, 40, 300)
        return dict(kind=kind, nx=nx, ny=rng.randint(max(16, nx // 3), nx // 2),
                    nrhs=rng.choice([1, 1, _log_int(rng, 2, 64)]))
    if kind == "products":
        nx = _log_int(rng, 60, 400)
        return dict(kind=kind, nx=nx, ny=rng.randint(nx // 3, nx // 2), b=rng.randint(8, 48),
                    fp32=rng.choice([True, False]))
    if kind == "open":
        nx = rng.randint(80, 160)
        return dict(kind=kind, nx=nx, ny=nx // 2, k=rng.randint(10, 20),
                    precision=rng.choice(["mixed", "fp64"]))
    if kind == "interp":
        fields = rng.choice([1, 1, 2, 4])
        return dict(kind=kind, order=rng.choice([1, 2, 3]), nx=_log_int(rng, 40, 400),
                    ny=_log_int(rng, 20, 200), points=_log_int(rng, 1000, (1 << 24) // fields),
                    fields=fields, ordered=rng.choice([True, False]),
                    gradient=rng.choice([True, False]))
    order = rng.choice([1, 2, 3])
    nx = _log_int(rng, 40, 600 // order)
    return dict(kind=kind, order=order, nx=nx, ny=rng.randint(nx // 3, nx // 2),
                states=rng.randint(1, 10), open=rng.choice([True, False]))


# ---------------------------------------------------------------------------
# Inputs: meshes, potentials and masses, made from the seed (1 nm cells unless said)
# ---------------------------------------------------------------------------

LOCAL = {1: [(1, 0, 0), (0, 1, 0), (0, 0, 1)],
         2: [(2, 0, 0), (0, 2, 0), (0, 0, 2), (1, 1, 0), (0, 1, 1), (1, 0, 1)],
         3: [(3, 0, 0), (0, 3, 0), (0, 0, 3), (2, 1, 0), (1, 2, 0), (0, 2, 1), (0, 1, 2),
             (1, 0, 2), (2, 0, 1), (1, 1, 1)]}


def _lattice(p, nx, ny, Lx, Ly):
    """Node coordinates and element centroids of the order-p lattice (row-major nodes,
    two triangles per cell)."""
    ix, iy = np.meshgrid(np.arange(p * nx + 1), np.arange(p * ny + 1))
    x, y = ix.ravel() * (Lx / (p * nx)), iy.ravel() * (Ly / (p * ny))
    ci, cj = np.meshgrid(np.arange(nx), np.arange(ny))
    third = np.array([1.0, 2.0]) / 3.0
    cx = (ci.ravel()[:, None] + third).ravel() * (Lx / nx)
    cy = (cj.ravel()[:, None] + third).ravel() * (Ly / ny)
    return x, y, cx, cy


def _sweep_sizes(case):
    """Cells along x of each dot: the case's, whatever the seed."""
    return np.random.default_rng([20261203, case["lo"], case["hi"]]).integers(
        case["lo"], case["hi"] + 1, case["dots"])


def _wells(case, seed):
    """Per dot (nx, ny, Lx, Ly, c, V): a circular well of radius U[5, 20] nm and depth
    U[0.1, 0.5] eV, m* 0.041 m0 inside and 0.067 outside."""
    rng = np.random.default_rng([seed, 1])
    out = []
    for n in _sweep_sizes(case):
        nx, ny = int(n), int(n) // 2
        R, depth = rng.uniform(5.0, 20.0), rng.uniform(0.1, 0.5)
        wx, wy = nx / 2 + rng.uniform(-5.0, 5.0), ny / 2 + rng.uniform(-5.0, 5.0)
        x, y, cx, cy = _lattice(case["order"], nx, ny, float(nx), float(ny))
        V = np.where((x - wx) ** 2 + (y - wy) ** 2 < R * R, -depth, 0.0)
        m = np.where((cx - wx) ** 2 + (cy - wy) ** 2 < R * R, 0.041, 0.067)
        out.append((nx, ny, float(nx), float(ny), C0 / m, V))
    return out


def _gauss(seed, Lx, Ly):
    """Parameters of a Gaussian dot near the middle (nm, eV)."""
    rng = np.random.default_rng([seed, 2])
    return (Lx / 2 + rng.uniform(-0.1, 0.1) * Lx, Ly / 2 + rng.uniform(-0.1, 0.1) * Ly,
            rng.uniform(0.2, 0.4), rng.uniform(6.0, 12.0))


def _gauss_dot(case, seed, p=1):
    nx, ny = case["nx"], case["ny"]
    gx, gy, d, w = _gauss(seed, nx, ny)
    x, y, cx, cy = _lattice(p, nx, ny, float(nx), float(ny))
    well = lambda a, b: -d * np.exp(-((a - gx) ** 2 + (b - gy) ** 2) / (2 * w * w))  # noqa: E731
    return C0 / np.where(well(cx, cy) < -d / 2, 0.041, 0.067), well(x, y)


def _junction(case, seed):
    """Static potential (a 0.2 eV step and a Gaussian dot) less the bias ramps."""
    nx, ny, nb = case["nx"], case["ny"], case["biases"]
    rng = np.random.default_rng([seed, 3])
    x, y, cx, cy = _lattice(1, nx, ny, float(nx), float(ny))
    dot = lambda a, b: -0.3 * np.exp(-((a - nx / 2) ** 2 + (b - ny / 2) ** 2) / 128.0)  # noqa: E731
    c = C0 / np.where(dot(cx, cy) < -0.15, 0.041, 0.067)
    V0 = np.where(x < nx / 2, 0.2, 0.0) + dot(x, y)
    return c, [V0 - v * x / nx for v in np.sort(rng.uniform(0.0, 1.0, nb))]


def _open_dot(case, seed):
    """P2 on 200 x 100 nm: two Gaussian wells and an absorbing layer of 10 nm; depths and
    centres vary with the seed."""
    nx, ny, Lx, Ly = case["nx"], case["ny"], 200.0, 100.0
    rng = np.random.default_rng([seed, 4])
    x, y, cx, cy = _lattice(2, nx, ny, Lx, Ly)
    V, Vc = np.zeros_like(x), np.zeros_like(cx)
    for at, d, w in ((70.0, 0.29, 8.0), (125.0, 0.11, 11.0)):
        d *= rng.uniform(0.95, 1.05)
        gx, gy = at + rng.uniform(-5, 5), Ly / 2 + rng.uniform(-10, 10)
        V -= d * np.exp(-((x - gx) ** 2 + (y - gy) ** 2) / (2 * w * w))
        Vc -= d * np.exp(-((cx - gx) ** 2 + (cy - gy) ** 2) / (2 * w * w))
    depth = np.clip(10.0 - np.minimum(np.minimum(x, Lx - x), np.minimum(y, Ly - y)), 0.0, None)
    return C0 / np.where(Vc < -0.05, 0.041, 0.067), V, 0.05 * (depth / 10.0) ** 2


def _poisson(case, seed):
    """Permittivity per element and charge (C/m^3) per node and bias."""
    nx, ny, nrhs = case["nx"], case["ny"], case["nrhs"]
    rng = np.random.default_rng([seed, 5])
    x, y, cx, _ = _lattice(1, nx, ny, float(nx), float(ny))
    eps = np.where(np.abs(cx - nx / 2) < nx / 8, 15.15, 12.9)
    rho = np.empty((x.size, nrhs))
    for j in range(nrhs):
        gx, gy, w = nx * rng.uniform(0.3, 0.7), ny * rng.uniform(0.3, 0.7), rng.uniform(5.0, 15.0)
        rho[:, j] = 1.6e5 * (rng.uniform(0.5, 1.0) * np.exp(-((x - gx) ** 2 + (y - gy) ** 2)
                                                            / (2 * w * w)) - 0.1 * (x / nx))
    return eps, rho, np.sort(rng.uniform(0.0, 1.0, nrhs))


def _vectors(case, seed, n, cols, dtype):
    g = torch.Generator(device=DEV).manual_seed(seed)
    if dtype.is_complex:
        return torch.view_as_complex(torch.randn(n, cols, 2, generator=g, device=DEV,
                                                 dtype=torch.float64)).to(dtype)
    return torch.randn(n, cols, generator=g, device=DEV, dtype=dtype)


def _points(case, seed):
    """Query points (nm, 1 nm cells) and smooth nodal fields."""
    p, nx, ny = case["order"], case["nx"], case["ny"]
    g = torch.Generator(device=DEV).manual_seed(seed)
    u = lambda *s: torch.rand(*s, generator=g, device=DEV, dtype=torch.float64)  # noqa: E731
    x, y = u(case["points"]) * nx, u(case["points"]) * ny
    if case["ordered"]:
        at = torch.argsort(y.long().clamp(max=ny - 1) * nx + x.long().clamp(max=nx - 1))
        x, y = x[at].contiguous(), y[at].contiguous()
    X, Y = (torch.from_numpy(a).to(DEV) for a in _lattice(p, nx, ny, float(nx), float(ny))[:2])
    f = torch.zeros(case["fields"], X.numel(), device=DEV, dtype=torch.float64)
    for _ in range(6):
        a, q = u(case["fields"], 1) - 0.5, 40.0 * u(4)
        f += a * torch.sin(q[0] * X / nx + q[1]) * torch.cos(q[2] * Y / ny + q[3])
    return x, y, f


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------

def _dots(specs, order):
    from qdsim_b200.mesh import StructuredMesh
    from qdsim_b200.workloads import Dot
    return [Dot(StructuredMesh(order, nx, ny, Lx, Ly), c, V) for nx, ny, Lx, Ly, c, V in specs]


def _device_batch(dots):
    from qdsim_b200.batch import DeviceBatch, HostBatch
    db = DeviceBatch(HostBatch(dots), DEV)
    db.upload(non_blocking=False)
    return db


def prepare(case, seed):
    from qdsim_b200.mesh import SimpleMesh, StructuredMesh
    kind = case["kind"]
    if kind == "dot":
        nx, ny = case["nx"], case["ny"]
        gx, gy, d, w = (1e-9 * a if i != 2 else a for i, a in enumerate(_gauss(seed, nx, ny)))

        def V(x, y):
            return -d * Q_E * np.exp(-((x - gx) ** 2 + (y - gy) ** 2) / (2 * w * w))

        def m_star(x, y):
            return np.where(V(x, y) < -0.5 * d * Q_E, 0.041, 0.067) * M_E

        return dict(case=case, mesh=SimpleMesh(nx + 1, ny + 1, nx * 1e-9, ny * 1e-9), V=V, m=m_star)
    if kind == "sweep":
        return dict(case=case, db=_device_batch(_dots(_wells(case, seed), case["order"])))
    if kind == "batch":
        return dict(case=case, db=_device_batch(_dots(_wells(case, seed), case["order"])))
    if kind == "junction":
        c, Vs = _junction(case, seed)
        from qdsim_b200.workloads import Dot
        mesh = StructuredMesh(1, case["nx"], case["ny"], float(case["nx"]), float(case["ny"]))
        db = _device_batch([Dot(mesh, c, V) for V in Vs])
        db.set_shift(0.5)
        return dict(case=case, db=db)
    if kind == "assemble":
        from qdsim_b200.fem import FEMProblem
        p, nx, ny = case["order"], case["nx"], case["ny"]
        c, V = _gauss_dot(case, seed, p)
        t = lambda a: torch.from_numpy(a).to(DEV)  # noqa: E731
        W = t(_layer(case)) if case["cap"] else None
        return dict(case=case, prob=FEMProblem(StructuredMesh(p, nx, ny, float(nx), float(ny)),
                                               device=DEV), c=t(c), V=t(V), W=W)
    if kind == "poisson":
        from qdsim_b200.poisson import PoissonProblem
        eps, rho, Vn = _poisson(case, seed)
        mesh = StructuredMesh(1, case["nx"], case["ny"], float(case["nx"]), float(case["ny"]))
        return dict(case=case, prob=PoissonProblem(mesh, eps, device=DEV),
                    rho=torch.from_numpy(rho).to(DEV), Vn=Vn)
    if kind in ("products", "open"):
        from qdsim_b200.cap import CAPSolver
        c, V, W = _open_dot(case, seed)
        solver = CAPSolver(StructuredMesh(2, case["nx"], case["ny"], 200.0, 100.0), c, V, W,
                           device=DEV)
        if kind == "open":
            return dict(case=case, solver=solver)
        dtype = torch.complex64 if case["fp32"] else torch.complex128
        X = _vectors(case, seed, solver.prob.n, case["b"], dtype)
        return dict(case=case, prob=solver.prob, X=X, AX=torch.empty_like(X), MX=torch.empty_like(X))
    if kind == "interp":
        from qdsim_b200.interp import FieldInterpolator
        x, y, f = _points(case, seed)
        mesh = StructuredMesh(case["order"], case["nx"], case["ny"], float(case["nx"]),
                              float(case["ny"]))
        return dict(case=case, fi=FieldInterpolator(mesh, device=DEV), x=x, y=y, f=f)
    from qdsim_b200.fem import FEMProblem
    p, nx, ny = case["order"], case["nx"], case["ny"]
    prob = FEMProblem(StructuredMesh(p, nx, ny, float(nx), float(ny)), device=DEV)
    prob.node_adjacency()
    psi = _vectors(case, seed, prob.n, case["states"],
                   torch.complex128 if case["open"] else torch.float64)
    return dict(case=case, prob=prob, psi=psi, w=_weights(case, seed))


def _layer(case):
    x, y, _, _ = _lattice(case["order"], case["nx"], case["ny"], float(case["nx"]),
                          float(case["ny"]))
    edge = np.minimum(np.minimum(x, case["nx"] - x), np.minimum(y, case["ny"] - y))
    return 0.05 * (np.clip(10.0 - edge, 0.0, None) / 10.0) ** 2


def _weights(case, seed):
    rng = np.random.default_rng([seed, 6])
    w = rng.uniform(-1.0, 1.0, case["states"])
    return w + 1j * rng.uniform(-1.0, 1.0, case["states"]) if case["open"] else w


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "dot":
        from qdsim_b200.solvers import CythonSchrodingerSolver
        E, _ = CythonSchrodingerSolver(state["mesh"], state["m"], state["V"]).solve(case["k"])
        return {"E": E}
    if kind == "sweep":
        # the sweep's tuned configuration (a 12-column block for 8 levels)
        state["db"].assemble()
        b = max(8, (case["k"] + 4 + 3) // 4 * 4)
        return {"E": state["db"].solve(case["k"], b=b, precision=case["precision"], tol=1e-9,
                                       tol32=1e-7, chunk_rows=2048, max_iter=2000)[0]}
    if kind == "junction":
        # as the self-consistent loop calls it: levels near zero measured against 0.1 eV
        state["db"].assemble()
        b = max(8, (case["k"] + 4 + 3) // 4 * 4)
        return {"E": state["db"].solve(case["k"], b=b, precision="mixed", tol=1e-9, max_iter=4000,
                                       eig_scale=0.1)[0]}
    if kind == "assemble":
        return state["prob"].assemble(state["c"], state["V"], state["W"])
    if kind == "batch":
        state["db"].assemble()
        return {"H": state["db"].H, "M": state["db"].M}
    if kind == "poisson":
        return {"phi": state["prob"].solve(state["rho"], 0.0, state["Vn"])}
    if kind == "products":
        state["prob"].spmm(state["X"], state["AX"], state["MX"])
        return {"AX": state["AX"], "MX": state["MX"]}
    if kind == "open":
        nev = min(40, 2 * case["k"])
        return {"E": state["solver"].solve(k=case["k"], sigma=-0.05, nev=nev, b=nev + 8,
                                           precision=case["precision"], tol=1e-9).E}
    if kind == "interp":
        f = state["f"] if case["fields"] > 1 else state["f"][0]
        return state["fi"].evaluate(state["x"], state["y"], f, gradient=case["gradient"],
                                    element=case["gradient"])
    from qdsim_b200.adjoint import energy_gradients
    dV, dc = energy_gradients(state["prob"], state["psi"], state["w"])
    return {"dV": dV, "dc": dc}


# ---------------------------------------------------------------------------
# work: inputs read once, outputs written once
# ---------------------------------------------------------------------------

_ROW = {1: 6.9, 2: 11.4, 3: 16.9}      # nonzeros per row of the stiffness pattern
_K = {1: 3, 2: 6, 3: 10}


def _sizes(p, nx, ny):
    """(nodes, elements, interior rows, nonzeros)"""
    rows = (p * nx - 1) * (p * ny - 1)
    return (p * nx + 1) * (p * ny + 1), 2 * nx * ny, rows, rows * _ROW[p]


def work(case):
    kind = case["kind"]
    if kind in ("sweep", "batch", "junction"):
        p = case.get("order", 1)
        shapes = ([(case["nx"], case["ny"])] * case["biases"] if kind == "junction" else
                  [(int(n), int(n) // 2) for n in _sweep_sizes(case)])
        by = fl = 0.0
        for nx, ny in shapes:
            N, E, rows, nnz = _sizes(p, nx, ny)
            by += N * 24 + E * (_K[p] * 4 + 8) + nnz * 4
            by += rows * case["k"] * 8 if kind != "batch" else nnz * 16
            fl += E * _K[p] ** 2 * 20
        return {"bytes": by, "flops": fl}
    if kind == "dot":
        N, E, rows, nnz = _sizes(1, case["nx"], case["ny"])
        return {"bytes": N * 24 + E * 20 + nnz * 20 + rows * case["k"] * 8, "flops": 4 * nnz * case["k"]}
    if kind == "assemble":
        p = case["order"]
        N, E, rows, nnz = _sizes(p, case["nx"], case["ny"])
        return {"bytes": N * (32 if case["cap"] else 24) + E * (_K[p] * 4 + 8) + nnz * 4
                + nnz * (24 if case["cap"] else 16), "flops": E * _K[p] ** 2 * 20}
    if kind == "poisson":
        N = (case["nx"] + 1) * (case["ny"] + 1)
        return {"bytes": N * 7 * 24 + N * case["nrhs"] * 16, "flops": N * 7 * 4 * case["nrhs"]}
    if kind in ("products", "open"):
        N, E, rows, nnz = _sizes(2, case["nx"], case["ny"])
        s, b = (4 if case.get("fp32") else 8), case.get("b", case.get("k"))
        return {"bytes": nnz * (4 + 3 * s) + 3 * rows * b * 2 * s, "flops": nnz * b * 12}
    if kind == "interp":
        N = _sizes(case["order"], case["nx"], case["ny"])[0]
        per = 16 + 8 * case["fields"] * (3 if case["gradient"] else 1) + (4 if case["gradient"] else 0)
        return {"bytes": case["points"] * per + 8 * N * case["fields"],
                "flops": case["points"] * case["fields"] * _K[case["order"]] * 2}
    p = case["order"]
    N, E, rows, _ = _sizes(p, case["nx"], case["ny"])
    return {"bytes": rows * case["states"] * (16 if case["open"] else 8) + E * (_K[p] * 4 + 8) + N * 28,
            "flops": E * _K[p] ** 2 * 2 * case["states"]}


# ---------------------------------------------------------------------------
# exact: plain torch and numpy in 64 bits
# ---------------------------------------------------------------------------

def _rule(p):
    """Barycentric points and weights of the element quadrature."""
    if p == 1:
        a, b = 1 / 6, 2 / 3
        return np.array([(a, a, b), (a, b, a), (b, a, a)]), np.full(3, 1 / 3)
    if p == 2:
        a, b, c, d = 0.059715871789770, 0.470142064105115, 0.797426985353087, 0.101286507323456
        xe = [(1 / 3, 1 / 3), (a, b), (b, a), (b, b), (c, d), (d, c), (d, d)]
        w = [0.225] + [0.132394152788506] * 3 + [0.125939180544827] * 3
    else:
        a, b, c, d = 0.249286745170910, 0.501426509658179, 0.063089014491502, 0.873821971016996
        e, f, g = 0.310352451033785, 0.636502499121399, 0.053145049844816
        xe = [(a, a), (a, b), (b, a), (c, c), (c, d), (d, c), (e, f), (f, g), (g, e), (f, e),
              (e, g), (g, f)]
        w = [0.116786275726379] * 3 + [0.050844906370207] * 3 + [0.082851075618374] * 6
    xe, w = np.array(xe), np.array(w)
    return np.concatenate([1 - xe.sum(1, keepdims=True), xe], 1), w / w.sum()


def _shapes(p, lam):
    """Lagrange shape functions [.., K] and their derivatives [.., 3, K] along each
    barycentric coordinate, as products of one-dimensional factors."""
    one = lam[..., 0] * 0 + 1

    def factor(l, m):
        v, d = one, one * 0
        for s in range(m):
            v, d = v * (p * l - s) / (s + 1), (d * (p * l - s) + v * p) / (s + 1)
        return v, d

    lib = torch if isinstance(lam, torch.Tensor) else np
    phi, der = [], []
    for at in LOCAL[p]:
        f = [factor(lam[..., i], at[i]) for i in range(3)]
        phi.append(f[0][0] * f[1][0] * f[2][0])
        der.append(lib.stack([f[0][1] * f[1][0] * f[2][0], f[0][0] * f[1][1] * f[2][0],
                              f[0][0] * f[1][0] * f[2][1]], -1))
    return lib.stack(phi, -1), lib.stack(der, -1)


def _tables(p):
    lam, w = _rule(p)
    phi, d = _shapes(p, lam)
    dx, dy = d[:, 1] - d[:, 0], d[:, 2] - d[:, 0]
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
    return dict(M=t(np.einsum("q,qi,qj->ij", w, phi, phi)), xx=t(np.einsum("q,qi,qj->ij", w, dx, dx)),
                xy=t(np.einsum("q,qi,qj->ij", w, dx, dy) + np.einsum("q,qi,qj->ij", w, dy, dx)),
                yy=t(np.einsum("q,qi,qj->ij", w, dy, dy)),
                T=t(np.einsum("q,ql,qi,qj->lij", w, phi, phi, phi)))


def _elements(p, nx, ny):
    """Lattice coordinates (ix, iy) of each element's nodes, int64 [E, K] twice (element
    2 cell + t, triangles (v00, v10, v01) and (v10, v11, v01))."""
    ci = torch.arange(nx, device=DEV).repeat(ny)
    cj = torch.arange(ny, device=DEV).repeat_interleave(nx)
    ix = torch.empty(2 * nx * ny, _K[p], dtype=torch.int64, device=DEV)
    iy = torch.empty_like(ix)
    for t, tri in enumerate((((0, 0), (1, 0), (0, 1)), ((1, 0), (1, 1), (0, 1)))):
        for a, l in enumerate(LOCAL[p]):
            ix[t::2, a] = p * ci + sum(l[i] * tri[i][0] for i in range(3))
            iy[t::2, a] = p * cj + sum(l[i] * tri[i][1] for i in range(3))
    return ix, iy


def _stiff(p, nx, ny, hx, hy):
    """Stiffness of each of the two triangles of a cell with c = 1, [2, K, K], and A."""
    tb, out = _tables(p), []
    for v in (((0, 0), (hx, 0), (0, hy)), ((hx, 0), (hx, hy), (0, hy))):
        J = np.array([[v[1][0] - v[0][0], v[2][0] - v[0][0]], [v[1][1] - v[0][1], v[2][1] - v[0][1]]])
        G = np.linalg.inv(J) @ np.linalg.inv(J).T
        out.append(0.5 * hx * hy * (G[0, 0] * tb["xx"] + G[0, 1] * tb["xy"] + G[1, 1] * tb["yy"]))
    return torch.stack(out), 0.5 * hx * hy, tb


def _element_matrices(p, nx, ny, Lx, Ly, c, V, W=None):
    S, A, tb = _stiff(p, nx, ny, Lx / nx, Ly / ny)
    ix, iy = _elements(p, nx, ny)
    node = iy * (p * nx + 1) + ix
    t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=DEV)  # noqa: E731
    H = t(c)[:, None, None] * S.repeat(nx * ny, 1, 1)
    H += A * torch.einsum("el,lij->eij", t(V)[node], tb["T"])
    M = (A * tb["M"]).expand(2 * nx * ny, -1, -1)
    G = -A * torch.einsum("el,lij->eij", t(W)[node], tb["T"]) if W is not None else None
    return ix, iy, H, M, G


def _pairs(p, nx, ny, ix, iy):
    """Row and column (interior nodes, row-major) of each element-matrix entry, -1 outside."""
    wx, wy = p * nx - 1, p * ny - 1
    ins = (ix > 0) & (ix <= wx) & (iy > 0) & (iy <= wy)
    dof = torch.where(ins, (iy - 1) * wx + ix - 1, -1)
    r = dof[:, :, None].expand(-1, -1, dof.shape[1])
    q = dof[:, None, :].expand(-1, dof.shape[1], -1)
    keep = (r >= 0) & (q >= 0)
    return r[keep], q[keep], keep, wx * wy


def _csr_values(p, nx, ny, Lx, Ly, c, V, W=None):
    """Values of H, M (and the absorbing term) in row-then-column order, and the pattern."""
    ix, iy, H, M, G = _element_matrices(p, nx, ny, Lx, Ly, c, V, W)
    r, q, keep, n = _pairs(p, nx, ny, ix, iy)
    key, at = torch.unique(r * n + q, return_inverse=True)
    put = lambda m: torch.zeros(key.numel(), dtype=torch.float64, device=DEV).index_add_(  # noqa: E731
        0, at, m[keep])
    return put(H), put(M), put(G) if G is not None else None, key // n, key % n, n


class _Blocks:
    """Block-tridiagonal system of B lattice problems of one order, lines of nodes along x
    grouped p to a block, problems of different sizes padded with decoupled unknowns."""

    def __init__(self, p, specs, pad=1e3, closed_y=True):
        """specs: (nx, ny, Lx, Ly, c, V, W or None); closed_y: Dirichlet at y = 0, Ly too."""
        self.p, self.B = p, len(specs)
        off = 1 if closed_y else 0
        nxm, self.wy = max(s[0] for s in specs), max(p * s[1] + 1 - 2 * off for s in specs)
        self.nb, self.s = -(-(p * nxm - 1) // p), p * self.wy
        self.n = self.nb * self.s
        rows, cols, Hv, Mv, Gv = [], [], [], [], []
        used = torch.zeros(self.B * self.n, dtype=torch.bool, device=DEV)
        for k, (nx, ny, Lx, Ly, c, V, W) in enumerate(specs):
            ix, iy, H, M, G = _element_matrices(p, nx, ny, Lx, Ly, c, V, W)
            ins = (ix > 0) & (ix < p * nx) & (iy >= off) & (iy <= p * ny - off)
            dof = torch.where(ins, k * self.n + (ix - 1) * self.wy + iy - off, -1)
            r = dof[:, :, None].expand(-1, -1, dof.shape[1])
            q = dof[:, None, :].expand(-1, dof.shape[1], -1)
            keep = (r >= 0) & (q >= 0)
            rows.append(r[keep]), cols.append(q[keep]), Hv.append(H[keep]), Mv.append(M[keep])
            if G is not None:
                Gv.append(G[keep])
            used[r[keep]] = True
        gap = (~used).nonzero()[:, 0]
        rows.append(gap), cols.append(gap)
        Hv.append(torch.full((gap.numel(),), pad, dtype=torch.float64, device=DEV))
        Mv.append(torch.ones(gap.numel(), dtype=torch.float64, device=DEV))
        self.r, self.q = torch.cat(rows), torch.cat(cols)
        self.H, self.M = torch.cat(Hv), torch.cat(Mv)
        self.G = torch.cat(Gv + [torch.zeros_like(Mv[-1])]) if Gv else None

    def sparse(self, v):
        N = self.B * self.n
        return torch.sparse_coo_tensor(torch.stack([self.r, self.q]), v, (N, N)).coalesce().to_sparse_csr()

    def dense(self, v):
        """Diagonal blocks [nb, B, s, s] and the blocks right of them [nb, B, s, s]."""
        s = self.s
        k, i, j = self.r // self.n, self.r % self.n, self.q % self.n
        bi, bj = i // s, j // s
        D = torch.zeros(self.nb * self.B * s * s, dtype=v.dtype, device=DEV)
        U = torch.zeros_like(D)
        at = ((bi * self.B + k) * s + i % s) * s + j % s
        for T, m in ((D, bi == bj), (U, bj == bi + 1)):
            T.index_put_((at[m],), v[m], accumulate=True)
        return D.view(self.nb, self.B, s, s), U.view(self.nb, self.B, s, s)

    def factor(self, v):
        """Block LDL^T (plain transposes): inverses of the pivot blocks and the couplings."""
        D, self.U = self.dense(v)
        for j in range(self.nb):
            D[j] = torch.linalg.inv(D[j])
            if j + 1 < self.nb:
                D[j + 1] -= self.U[j].mT @ (D[j] @ self.U[j])
        self.D = D

    def solve(self, b):
        """b [B, n, q] -> the solution."""
        b = b.view(self.B, self.nb, self.s, -1).transpose(0, 1).clone()
        for j in range(1, self.nb):
            b[j] -= self.U[j - 1].mT @ (self.D[j - 1] @ b[j - 1])
        for j in reversed(range(self.nb)):
            if j + 1 < self.nb:
                b[j] -= self.U[j] @ b[j + 1]
            b[j] = self.D[j] @ b[j]
        return b.transpose(0, 1).reshape(self.B, self.n, -1)


def _levels(p, specs, k):
    """The k lowest levels of each problem by block Krylov iteration on a shifted inverse:
    first from below the spectrum, then from just above the k-th level found, with a new
    random block each time, until no level moves."""
    S = _Blocks(p, [(*s, None) for s in specs])
    H, M = S.sparse(S.H), S.sparse(S.M)
    mul = lambda A, X: (A @ X.reshape(-1, X.shape[2])).view(X.shape)  # noqa: E731
    g = torch.Generator(device=DEV).manual_seed(0)
    Q = X = None

    def expand(Z):
        for _ in range(2):
            if Q is not None:
                Z = Z - Q @ (Q.mT @ mul(M, Z))
            R = torch.linalg.cholesky(Z.mT @ mul(M, Z))
            Z = torch.linalg.solve_triangular(R, Z.mT, upper=False).mT.contiguous()
        return Z, Z if Q is None else torch.cat([Q, Z], 2)

    shift = torch.tensor([float(np.min(s[5])) - 0.01 for s in specs], device=DEV, dtype=torch.float64)
    E = torch.full((S.B, k), math.inf, device=DEV, dtype=torch.float64)
    for steps in (48, 20, 20, 20):
        S.factor(S.H - shift[S.r // S.n] * S.M)
        X, Q = expand(torch.randn(S.B, S.n, k + 6, generator=g, device=DEV, dtype=torch.float64))
        for _ in range(steps):
            X, Q = expand(S.solve(mul(M, X)))
        T = Q.mT @ mul(H, Q)
        old, (E, Y) = E, torch.linalg.eigh(0.5 * (T + T.mT))
        Q = (Q @ Y[:, :, :2 * k + 6]).contiguous()
        shift = 0.75 * E[:, k - 1] + 0.25 * E[:, k]
        E = E[:, :k]
        if float(((E - old).abs() / E.abs().amax(1, keepdim=True)).max()) < 1e-13:
            break
    return E


def _all_levels(p, specs, k):
    """_levels over groups of similar size, in the order given."""
    E = torch.empty(len(specs), k, dtype=torch.float64, device=DEV)
    order = sorted(range(len(specs)), key=lambda i: specs[i][0])
    for at in range(0, len(order), 16):
        g = order[at:at + 16]
        E[torch.tensor(g, device=DEV)] = _levels(p, [specs[i] for i in g], k)
    return E


def _open_levels(case, c, V, W, sigma=-0.05, steps=120):
    S = _Blocks(2, [(case["nx"], case["ny"], 200.0, 100.0, c, V, W)])
    A, Mv = torch.complex(S.H, S.G), S.M.to(torch.complex128)
    S.factor(A - sigma * Mv)
    A, M = S.sparse(A), S.sparse(Mv)
    g = torch.Generator(device=DEV).manual_seed(0)
    Q = torch.zeros(steps + 1, S.n, dtype=torch.complex128, device=DEV)
    q = torch.randn(S.n, generator=g, device=DEV, dtype=torch.complex128)
    Q[0] = q / torch.linalg.vector_norm(q)
    Hs = torch.zeros(steps + 1, steps, dtype=torch.complex128, device=DEV)
    for j in range(steps):
        w = S.solve((M @ Q[j][:, None]).view(1, S.n, 1)).view(-1)
        for _ in range(2):
            h = Q[:j + 1].conj() @ w
            w = w - h @ Q[:j + 1]
            Hs[:j + 1, j] += h
        Hs[j + 1, j] = torch.linalg.vector_norm(w)
        Q[j + 1] = w / Hs[j + 1, j]
    th, Y = np.linalg.eig(Hs[:steps].cpu().numpy())
    Y = Y[:, np.argsort(-np.abs(th))[:case["k"]]]
    X = Q[:steps].T @ torch.from_numpy(Y).to(DEV)
    E = ((X * (A @ X)).sum(0) / (X * (M @ X)).sum(0)).cpu().numpy()
    return E[np.argsort(np.abs(E - sigma))]


def _exact_poisson(case, seed):
    eps, rho, Vn = _poisson(case, seed)
    nx, ny = case["nx"], case["ny"]
    spec = (nx, ny, float(nx), float(ny), eps, np.zeros((nx + 1) * (ny + 1)), None)
    ix, iy, K, M, _ = _element_matrices(1, *spec)
    node = iy * (nx + 1) + ix
    N = (nx + 1) * (ny + 1)
    at = torch.stack([node[:, :, None].expand(-1, -1, 3).reshape(-1),
                      node[:, None, :].expand(-1, 3, -1).reshape(-1)])
    csr = lambda v: torch.sparse_coo_tensor(at, v.reshape(-1), (N, N)).coalesce().to_sparse_csr()  # noqa: E731
    phi = torch.zeros(ny + 1, nx + 1, case["nrhs"], dtype=torch.float64, device=DEV)
    phi[:, nx] = torch.from_numpy(Vn).to(DEV)
    b = csr(M) @ (-1e-18 / EPS0 * torch.from_numpy(rho).to(DEV)) - csr(K) @ phi.view(N, -1)
    S = _Blocks(1, [spec], closed_y=False)
    S.factor(S.H)
    free = b.view(ny + 1, nx + 1, -1)[:, 1:nx].transpose(0, 1).reshape(1, S.n, -1)
    x = S.solve(free)
    res = free - (S.sparse(S.H) @ x[0])[None]
    x = (x + S.solve(res)).view(nx - 1, ny + 1, -1)
    phi[:, 1:nx] = x.transpose(0, 1)
    phi = phi.view(N, -1)
    return {"phi": phi if case["nrhs"] > 1 else phi[:, 0]}


def _exact_interp(case, seed):
    x, y, f = _points(case, seed)
    p, nx, ny = case["order"], case["nx"], case["ny"]
    out = {k: torch.empty(case["fields"], x.numel(), dtype=torch.float64, device=DEV)
           for k in (("value", "grad_x", "grad_y") if case["gradient"] else ("value",))}
    el = torch.empty(x.numel(), dtype=torch.int32, device=DEV)
    ex, ey = _elements(p, nx, ny)
    node = ey * (p * nx + 1) + ex
    for at in range(0, x.numel(), 1 << 20):
        s = slice(at, at + (1 << 20))
        i, j = x[s].long().clamp(max=nx - 1), y[s].long().clamp(max=ny - 1)
        u, v = x[s] - i, y[s] - j                      # cells of 1 nm
        up = u + v > 1
        lam = torch.where(up[:, None], torch.stack([1 - v, u + v - 1, 1 - u], 1),
                          torch.stack([1 - u - v, u, v], 1))
        phi, d = _shapes(p, lam)
        e = 2 * (j * nx + i) + up
        fn = f[:, node[e]]
        out["value"][:, s] = torch.einsum("fpk,pk->fp", fn, phi)
        el[s] = e.to(torch.int32)
        if case["gradient"]:
            g = torch.einsum("fpk,pmk->fpm", fn, d)
            out["grad_x"][:, s] = torch.where(up, g[..., 1] - g[..., 2], g[..., 1] - g[..., 0])
            out["grad_y"][:, s] = torch.where(up, g[..., 1] - g[..., 0], g[..., 2] - g[..., 0])
    if case["fields"] == 1:
        out = {k: v[0] for k, v in out.items()}
    return {**out, "element": el} if case["gradient"] else out


def _exact_adjoint(case, seed):
    p, nx, ny = case["order"], case["nx"], case["ny"]
    S, A, tb = _stiff(p, nx, ny, 1.0, 1.0)
    ix, iy = _elements(p, nx, ny)
    wx, wy = p * nx - 1, p * ny - 1
    psi = _vectors(case, seed, wx * wy, case["states"],
                   torch.complex128 if case["open"] else torch.float64)
    full = torch.zeros(p * ny + 1, p * nx + 1, case["states"], dtype=psi.dtype, device=DEV)
    full[1:-1, 1:-1] = psi.view(wy, wx, -1)
    w = torch.from_numpy(_weights(case, seed)).to(DEV)
    a = full[iy, ix]                                   # [E, K, states]
    U = torch.einsum("eis,ejs,s->eij", a, a, w)
    U = U.real if case["open"] else U
    dc = (U * S.repeat(nx * ny, 1, 1)).sum((1, 2))
    dV = torch.zeros((p * nx + 1) * (p * ny + 1), dtype=torch.float64, device=DEV)
    dV.index_add_(0, (iy * (p * nx + 1) + ix).reshape(-1),
                  (A * torch.einsum("eij,lij->el", U, tb["T"])).reshape(-1))
    return {"dV": dV, "dc": dc}


def exact(case, seed):
    kind = case["kind"]
    if kind == "dot":
        nx, ny = case["nx"], case["ny"]
        c, V = _gauss_dot(case, seed)
        return {"E": _levels(1, [(nx, ny, float(nx), float(ny), c, V)], case["k"])[0].cpu().numpy() * Q_E}
    if kind == "sweep":
        return {"E": _all_levels(case["order"], _wells(case, seed), case["k"])}
    if kind == "junction":
        c, Vs = _junction(case, seed)
        nx, ny = case["nx"], case["ny"]
        return {"E": _all_levels(1, [(nx, ny, float(nx), float(ny), c, V) for V in Vs], case["k"])}
    if kind == "assemble":
        c, V = _gauss_dot(case, seed, case["order"])
        W = _layer(case) if case["cap"] else None
        H, M, G, *_ = _csr_values(case["order"], case["nx"], case["ny"], float(case["nx"]),
                                  float(case["ny"]), c, V, W)
        return {"H": H, "M": M, "Himag": G} if case["cap"] else {"H": H, "M": M}
    if kind == "batch":
        parts = [_csr_values(case["order"], *s)[:2] for s in _wells(case, seed)]
        return {"H": torch.cat([h for h, _ in parts]), "M": torch.cat([m for _, m in parts])}
    if kind == "poisson":
        return _exact_poisson(case, seed)
    if kind == "open":
        return {"E": _open_levels(case, *_open_dot(case, seed))}
    if kind == "products":
        H, M, G, r, q, n = _csr_values(2, case["nx"], case["ny"], 200.0, 100.0, *_open_dot(case, seed))
        dtype = torch.complex64 if case["fp32"] else torch.complex128
        X = _vectors(case, seed, n, case["b"], dtype).to(torch.complex128)
        csr = lambda v: torch.sparse_coo_tensor(torch.stack([r, q]), v, (n, n)).coalesce().to_sparse_csr()  # noqa: E731
        return {"AX": csr(torch.complex(H, G)) @ X, "MX": csr(M.to(torch.complex128)) @ X}
    if kind == "interp":
        return _exact_interp(case, seed)
    return _exact_adjoint(case, seed)
