"""Poisson step of the self-consistent loop on the GPU.

Same weak form and boundary conditions as
``qdsim_cython/solvers/poisson_solver.pyx`` (P1 stiffness with eps_r per
element, RHS = M (-rho), phi = V_p on x = 0 and V_n on x = Lx, natural
elsewhere), without its m^2-scale degenerate-area test that skips every
element of a nanometre mesh (:126).  Assembly uses the row-block kernel
(c = eps_r, V = 0); the solve is a batched PCG over any number of right-hand
sides (bias points) sharing the stiffness matrix: preconditioned by the
lattice's separable solver (``qd_poisson_lattice_solve``) where that is the
better form, else by the diagonal (``qd_pcg_solve``).

Units: node coordinates in nm, rho in C/m^3, phi in V.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from . import _native as N
from .fem import FEMProblem, stream_ptr
from .mesh import StructuredMesh

EPS0 = 8.854187817e-12     # qdsim_cython/solvers/poisson_solver.pyx:28


#: Largest condition number of the separably preconditioned operator for which
#: the lattice form is considered.  Its iterations grow with the square root of
#: this number and not with the mesh (lattice_pays).
LATTICE_KAPPA = 64.0
LATTICE_MAX_NX = 8000       # qd_poisson_lattice_solve's limits
LATTICE_MAX_NY = 16384
LATTICE_MAX_RHS = 256
#: Bytes that the plan of any problem may take.  Its cosine matrices take 8 ny^2
#: bytes whatever nx is: on a narrow mesh that is far more than the problem itself.
LATTICE_PLAN_BYTES = 256 << 20
NODE_BYTES = 200            # of a problem's mesh, pattern and matrices, about


def lattice_fits(nx, ny):
    """Whether an nx x ny lattice is within the separable solver's limits, and its
    plan no larger than LATTICE_PLAN_BYTES or than the problem's other data."""
    if nx > LATTICE_MAX_NX or ny > LATTICE_MAX_NY:
        return False
    nodes = (nx + 1) * (ny + 1)
    return 8 * ny * ny + 16 * nodes <= max(LATTICE_PLAN_BYTES, NODE_BYTES * nodes)


def on_lattice(mesh):
    """Whether the nodes of a P1 structured mesh lie on its uniform lattice (a mesh
    whose nodes were moved, e.g. graded towards a contact, is structured too)."""
    p = mesh.nodes.reshape(mesh.ny + 1, mesh.nx + 1, 2)
    x = np.arange(mesh.nx + 1) * (mesh.Lx / mesh.nx)
    y = np.arange(mesh.ny + 1) * (mesh.Ly / mesh.ny)
    return (np.abs(p[:, :, 0] - x).max() <= 1e-9 * mesh.Lx
            and np.abs(p[:, :, 1] - y[:, None]).max() <= 1e-9 * mesh.Ly)


def lattice_pays(mesh, kappa, nrhs):
    """Whether the lattice form is the faster one, by the iterations that either
    needs to 1e-12 and what an iteration takes (microseconds on a B200).

    Lattice: 8.5 to 12.5 sqrt(kappa) iterations where eps varies at random, one or
    two where the separable operator is the operator; five launches, a serial
    chain over the modes and one along the line, 300 bytes a value, and dense
    transforms at 23 TFLOP/s.  Diagonal: in proportion to nx, more on meshes that
    are long in y or fine in y, up to 11 nx; two launches, one thread's sum over the
    block's threads / nrhs, 88 bytes a value.  Over 278 pairs of meshes (4 x 4 to
    1000 x 1000, nx up to 7000, ny up to 4096), eps and 1 or 64 right-hand sides, the
    diagonal form was nowhere faster where this rule takes the lattice form.  It is
    where the rule takes it: 8 x 4096, eps in 1..30 at random, 64 right-hand sides
    7.8 against 85.9 ms; 8 x 512, 3.7 against 7.8 ms; 8 x 2048, one right-hand
    side, 10.2 against 16.0 ms.  At 300 x 100 and the same eps the lattice form takes
    12.1 ms for 64 right-hand sides where the diagonal one takes 71.8."""
    nx, ny = mesh.nx, mesh.ny
    hx, hy = mesh.Lx / nx, mesh.Ly / ny
    values = (nx + 1) * (ny + 1) * nrhs
    its = 2.0 if kappa < 1.001 else 9.0 * math.sqrt(kappa)
    lattice = its * (42.0 + 0.145 * ny + 0.025 * nx + 6e-5 * values
                     + 2.0 * ny * ny * (nx + 1) * nrhs / 23e6)
    its = nx * min(11.0, 5.5 * (mesh.Ly / mesh.Lx) ** 0.3) * math.sqrt(0.5 + 0.5 * (hx / hy) ** 2)
    diagonal = max(16.0, its) * (18.0 + 62.0 / nrhs + 1.8e-5 * values)
    return lattice <= diagonal


def lattice_means(mesh, eps):
    """Column means of the edge conductances of a P1 structured mesh: ``gx``
    [nx] over the x-edges between columns i and i + 1, ``gy`` [nx + 1] over the
    y-edges of column i (both divided by ny), and the condition number bound:
    the largest over the smallest ratio of an edge's conductance to what the
    separable operator gives it (mean, halved on the two boundary rows)."""
    nx, ny = mesh.nx, mesh.ny
    r = (mesh.Ly / ny) / (mesh.Lx / nx)
    e = np.asarray(eps, np.float64).reshape(ny, nx, 2)
    lo, up = e[:, :, 0], e[:, :, 1]          # triangles with the right angle at v00, v11
    ex = np.zeros((ny + 1, nx))              # conductance of the x-edge (i, i + 1) of row j
    ex[:-1] += 0.5 * r * lo
    ex[1:] += 0.5 * r * up
    ey = np.zeros((ny, nx + 1))
    ey[:, :-1] += 0.5 / r * lo
    ey[:, 1:] += 0.5 / r * up
    gx, gy = ex.sum(0) / ny, ey.sum(0) / ny
    w = np.ones(ny + 1)
    w[0] = w[-1] = 0.5
    with np.errstate(divide="ignore", invalid="ignore"):
        inner = ey[:, 1:-1] / gy[1:-1]       # the end columns are Dirichlet
        q = np.concatenate([(ex / (w[:, None] * gx)).ravel(), inner.ravel()])
    positive = gx.min() > 0.0 and gy.min() > 0.0 and q.min() > 0.0    # not with NaN
    kappa = float(q.max() / q.min()) if positive and np.isfinite(q.max()) else np.inf
    return gx, gy, kappa


class PoissonProblem:
    def __init__(self, mesh, eps_r_elem, device="cuda"):
        if mesh.order != 1:
            raise ValueError("the Poisson step is P1")
        self.mesh = mesh
        self.fem = FEMProblem(mesh, dirichlet=False, device=device)
        self.device = self.fem.device
        out = self.fem.assemble(np.asarray(eps_r_elem, float), np.zeros(mesh.num_nodes))
        self.K = out["H"]
        self.M = out["M"]
        x = mesh.nodes[:, 0]
        self.left = np.abs(x) < 1e-9 * mesh.Lx
        self.right = np.abs(x - mesh.Lx) < 1e-9 * mesh.Lx
        self.d_fixed = torch.from_numpy((self.left | self.right).astype(np.int32)).to(self.device)
        self._ws = None
        self._pays = {}        # right-hand sides: lattice_pays
        self._plan = self._lattice_plan(eps_r_elem)
        self.last_iters = 0
        self.last_relres = 0.0

    def _lattice_plan(self, eps):
        """Device plan of the separable preconditioner, or None where the
        diagonal form is taken (nodes not on a lattice, eps varying too much along
        y, a lattice beyond the kernel's limits or too narrow to pay)."""
        m = self.mesh
        if (not isinstance(m, StructuredMesh) or not lattice_fits(m.nx, m.ny)
                or not on_lattice(m)):
            return None
        gx, gy, self._kappa = lattice_means(m, eps)
        # one right-hand side is where the diagonal form's iteration costs most
        if not self._kappa <= LATTICE_KAPPA or not lattice_pays(m, self._kappa, 1):
            return None
        L = N.lib()
        nbytes = C.c_size_t()
        N.check(L.qd_poisson_lattice_plan_size(m.nx, m.ny, C.byref(nbytes)),
                "qd_poisson_lattice_plan_size")
        plan = torch.empty(nbytes.value, dtype=torch.uint8, device=self.device)
        g = torch.from_numpy(np.concatenate([gx, gy])).to(self.device)
        N.check(L.qd_poisson_lattice_plan(m.nx, m.ny, N.ptr(g), N.ptr(g[m.nx:]), N.ptr(plan),
                                          plan.numel(), stream_ptr()), "qd_poisson_lattice_plan")
        # solve() may run on any stream: the plan is complete when the problem is
        torch.cuda.current_stream().synchronize()
        return plan

    def _least_cap(self, tol):
        """The iteration cap from which the lattice form is taken.  It must be
        enough for that form, which needs at most sqrt(kappa) / 2 ln(2 / tol)
        iterations and a few more for the residual's scale; and below nx / 2 the
        call is left to end at its cap as the diagonal form does, whose iterations
        carry a contact's value one column further each."""
        digits = math.log(2.0 / min(tol, 1.0)) if tol > 0.0 else 0.0
        return max(1.0, self.mesh.nx / 2, 0.5 * math.sqrt(self._kappa) * (digits + 8.0))

    def rhs(self, rho):
        """(1e-18/eps0) M (-rho) on the device; rho [N] or [N, nrhs] (C/m^3)."""
        r = rho if isinstance(rho, torch.Tensor) else torch.from_numpy(np.asarray(rho, np.float64))
        r = r.to(self.device, torch.float64).reshape(self.mesh.num_nodes, -1).contiguous()
        b = torch.empty_like(r)
        n, nrhs = r.shape
        N.check(N.lib().qd_csr_spmv(n, nrhs, N.ptr(self.fem.d_rowptr), N.ptr(self.fem.d_col),
                                    N.ptr(self.M), N.ptr(r), N.ptr(b), -1e-18 / EPS0,
                                    stream_ptr()), "qd_csr_spmv")
        return b

    def solve(self, rho, V_p, V_n, tol=1e-12, max_iter=20000, x0=None):
        """phi (V) at every node, [N] or [N, nrhs] (device tensor)."""
        n = self.mesh.num_nodes
        if self._plan is not None and max_iter >= self._least_cap(tol):
            r = rho if isinstance(rho, torch.Tensor) else torch.from_numpy(np.asarray(rho, np.float64))
            r = r.to(self.device, torch.float64).reshape(n, -1).contiguous()
            nrhs = r.shape[1]
            if nrhs not in self._pays:
                self._pays[nrhs] = nrhs <= LATTICE_MAX_RHS and lattice_pays(self.mesh, self._kappa, nrhs)
            if self._pays[nrhs]:
                return self._solve_lattice(r, V_p, V_n, tol, max_iter, x0)
            rho = r
        b = self.rhs(rho)
        n, nrhs = b.shape
        vp = torch.as_tensor(np.broadcast_to(np.asarray(V_p, float), (nrhs,)).copy(),
                             device=self.device)
        vn = torch.as_tensor(np.broadcast_to(np.asarray(V_n, float), (nrhs,)).copy(),
                             device=self.device)
        X = (torch.zeros_like(b) if x0 is None
             else x0.to(self.device, torch.float64).reshape(n, nrhs).clone())
        X[torch.from_numpy(self.left).to(self.device)] = vp
        X[torch.from_numpy(self.right).to(self.device)] = vn
        L = N.lib()
        nbytes = C.c_size_t()
        N.check(L.qd_pcg_workspace_size(n, nrhs, C.byref(nbytes)), "qd_pcg_workspace_size")
        if self._ws is None or self._ws.numel() < nbytes.value:
            self._ws = torch.empty(nbytes.value, dtype=torch.uint8, device=self.device)
        iters = C.c_int32()
        relres = C.c_double()
        N.check(L.qd_pcg_solve(n, nrhs, N.ptr(self.fem.d_rowptr), N.ptr(self.fem.d_col),
                               N.ptr(self.K), N.ptr(b), N.ptr(X), N.ptr(self.d_fixed), float(tol),
                               int(max_iter), C.byref(iters), C.byref(relres), N.ptr(self._ws),
                               self._ws.numel(), stream_ptr()), "qd_pcg_solve")
        self.last_iters = iters.value
        self.last_relres = relres.value
        return X if nrhs > 1 else X[:, 0]

    def _solve_lattice(self, r, V_p, V_n, tol, max_iter, x0):
        n, nrhs = r.shape
        m, L = self.mesh, N.lib()
        vp = np.ascontiguousarray(np.broadcast_to(np.asarray(V_p, float), (nrhs,)))
        vn = np.ascontiguousarray(np.broadcast_to(np.asarray(V_n, float), (nrhs,)))
        X = torch.empty_like(r)
        if x0 is not None:
            x0 = x0.to(self.device, torch.float64).reshape(n, nrhs).contiguous()
        nbytes = C.c_size_t()
        N.check(L.qd_poisson_lattice_workspace_size(m.nx, m.ny, nrhs, C.byref(nbytes)),
                "qd_poisson_lattice_workspace_size")
        if self._ws is None or self._ws.numel() < nbytes.value:
            self._ws = torch.empty(nbytes.value, dtype=torch.uint8, device=self.device)
        iters = C.c_int32()
        relres = C.c_double()
        N.check(L.qd_poisson_lattice_solve(
            m.nx, m.ny, nrhs, N.ptr(self.fem.d_rowptr), N.ptr(self.fem.d_col), N.ptr(self.K),
            N.ptr(self.M), N.ptr(r), -1e-18 / EPS0, N.ptr(vp), N.ptr(vn), N.ptr(x0), N.ptr(X),
            N.ptr(self._plan), float(tol), int(max_iter), C.byref(iters), C.byref(relres),
            N.ptr(self._ws), self._ws.numel(), stream_ptr()), "qd_poisson_lattice_solve")
        self.last_iters = iters.value
        self.last_relres = relres.value
        return X if nrhs > 1 else X[:, 0]
