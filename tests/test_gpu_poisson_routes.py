"""Which form a Poisson problem takes, and that either gives the oracle's potential:
the lattice form (separable preconditioner) on structured meshes, the diagonal form
elsewhere."""
import ctypes as C

import numpy as np
import pytest

from oracle import fem as O, poisson as OP


def _mesh(nx, ny, hy=1.5):
    from qdsim_b200 import mesh as Mh
    om = O.structured_mesh(1, nx, ny, 2.0 * nx, hy * ny)
    return om, Mh.StructuredMesh(1, nx, ny, om.Lx, om.Ly)


def _solve(cuda, om, m, eps, nrhs, seed=0, **kw):
    """(problem, largest error over the largest potential) of one solve."""
    from qdsim_b200 import poisson as P
    rng = np.random.default_rng([seed, om.num_nodes, nrhs])
    R = 1.6e5 * rng.standard_normal((om.num_nodes, nrhs))
    vp, vn = rng.uniform(-0.2, 0.2, nrhs), rng.uniform(0.0, 1.0, nrhs)
    ref = OP.solve(om, eps, R, vp, vn).reshape(om.num_nodes, nrhs)
    prob = P.PoissonProblem(m, eps, device=cuda)
    got = prob.solve(R, vp, vn, tol=1e-12, **kw).cpu().numpy().reshape(om.num_nodes, nrhs)
    return prob, np.abs(got - ref).max() / np.abs(ref).max()


def test_plan_is_bounded():
    """The plan grows with ny^2: beyond 256 MB it may not exceed what the problem
    itself takes, and the library refuses ny beyond its own limit."""
    from qdsim_b200 import _native as N, poisson as P
    assert P.lattice_fits(300, 100) and P.lattice_fits(8, 4096) and P.lattice_fits(1000, 9000)
    assert not P.lattice_fits(8, 10000) and not P.lattice_fits(8000, 50000)
    assert not P.lattice_fits(8001, 10)
    size = C.c_size_t()
    L = N.lib()
    assert L.qd_poisson_lattice_plan_size(8, P.LATTICE_MAX_NY, C.byref(size)) == N.QD_OK
    assert L.qd_poisson_lattice_plan_size(8, P.LATTICE_MAX_NY + 1, C.byref(size)) != N.QD_OK
    assert L.qd_poisson_lattice_workspace_size(8, P.LATTICE_MAX_NY + 1, 1, C.byref(size)) != N.QD_OK


@pytest.mark.gpu
def test_a_tall_narrow_mesh_takes_the_diagonal_form(cuda):
    om, m = _mesh(4, 12000)
    eps = np.random.default_rng(1).uniform(10.0, 14.0, om.num_elements)
    prob, err = _solve(cuda, om, m, eps, 2)
    assert prob._plan is None and err <= 1e-9
