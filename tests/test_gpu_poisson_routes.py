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


@pytest.mark.filterwarnings("error")
def test_no_plan_without_positive_conductances():
    """The separable operator must be positive definite; zero, negative and non-finite
    columns leave the problem to the diagonal form, without a warning."""
    from qdsim_b200 import mesh as Mh, poisson as P
    m = Mh.StructuredMesh(1, 6, 4, 6.0, 4.0)
    for bad in (-3.0, 0.0, np.nan, np.inf):
        assert P.lattice_means(m, np.full(m.num_elements, bad))[2] == np.inf
        eps = np.full((4, 6, 2), 2.0)
        eps[:, 2] = bad
        assert P.lattice_means(m, eps.ravel())[2] == np.inf


# nx, ny, kappa, right-hand sides, whether the lattice form was the faster one,
# timed with eps varying at random (kappa 1: along x only)
TIMED = [(300, 100, 35.8, 64, True), (100, 50, 1.0, 1, True), (1000, 1000, 32.6, 16, True),
         (4000, 16, 56.1, 64, True), (8, 4096, 1.0, 64, True), (32, 512, 8.4, 64, True),
         (8, 512, 30.0, 64, False), (8, 2048, 29.4, 1, False), (8, 4096, 8.0, 64, False),
         (2, 2048, 1.4, 64, False), (32, 2048, 30.4, 64, False), (4, 4, 22.5, 64, False)]


@pytest.mark.parametrize("nx,ny,kappa,nrhs,lattice", TIMED)
def test_rule_takes_the_form_that_was_faster(nx, ny, kappa, nrhs, lattice):
    from qdsim_b200 import mesh as Mh, poisson as P
    m = Mh.StructuredMesh(1, nx, ny, float(nx), float(ny))
    assert P.lattice_pays(m, kappa, nrhs) == lattice


@pytest.mark.gpu
def test_a_tall_narrow_mesh_takes_the_diagonal_form(cuda):
    om, m = _mesh(4, 12000)
    eps = np.random.default_rng(1).uniform(10.0, 14.0, om.num_elements)
    prob, err = _solve(cuda, om, m, eps, 2)
    assert prob._plan is None and err <= 1e-9


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nrhs,contrast,plan", [
    (32, 1024, 64, 30.0, True),     # one right-hand side pays, 64 do not
    (8, 1024, 1, 8.0, True),
    (2, 2048, 3, 8.0, False),       # never pays: no plan
])
def test_narrow_meshes_match_the_oracle(cuda, nx, ny, nrhs, contrast, plan):
    om, m = _mesh(nx, ny, hy=2.0)
    eps = np.exp(np.random.default_rng(nx).uniform(0.0, np.log(contrast), om.num_elements))
    prob, err = _solve(cuda, om, m, eps, nrhs)
    assert (prob._plan is not None) == plan and err <= 1e-9


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,kw", [
    (1000, 300, {}),                        # large meshes at the default cap
    (300, 100, {"max_iter": 5000}),         # caps that are enough for either form
    (300, 100, {"max_iter": 1000}),
    (60, 30, {"max_iter": 60}),
])
def test_the_cap_does_not_choose_the_form(cuda, nx, ny, kw):
    """The lattice form's iterations do not grow with the mesh: at most 14 here (eps
    in 10..14), where the diagonal form takes more than 3 per column."""
    om, m = _mesh(nx, ny)
    eps = np.random.default_rng(nx).uniform(10.0, 14.0, om.num_elements)
    prob, err = _solve(cuda, om, m, eps, 1, **kw)
    assert prob.last_iters <= 14 and err <= 1e-9


@pytest.mark.gpu
def test_a_cap_that_is_enough_for_the_diagonal_form_only(cuda):
    """15 unknowns: the diagonal form ends within 15 iterations, the lattice form's
    bound is 30 at this contrast."""
    om, m = _mesh(4, 4)
    eps = np.exp(np.random.default_rng(5).uniform(0.0, np.log(8.0), om.num_elements))
    prob, err = _solve(cuda, om, m, eps, 1, max_iter=18)
    assert prob._plan is not None and err <= 1e-9
    assert prob._least_cap(1e-12) > 18


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(60, 20), (7, 90)])
@pytest.mark.parametrize("nrhs", [1, 3, 64])
def test_diagonal_form_matches_the_oracle(cuda, nx, ny, nrhs):
    """Contrast along y beyond the lattice form's bound."""
    om, m = _mesh(nx, ny)
    eps = np.where(np.repeat(np.arange(ny) % 3 == 1, 2 * nx), 300.0, 1.0)
    prob, err = _solve(cuda, om, m, eps, nrhs)
    assert prob._plan is None and prob.last_relres <= 1e-12
    # residual 1e-12 of the right-hand side, amplified by at most the square root of
    # the stiffness's condition number (< 400 sqrt(300))
    assert err <= 7e-9


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nrhs", [(60, 30, 1), (33, 64, 5), (120, 41, 64)])
@pytest.mark.parametrize("contrast", [8.0, 30.0, -40.0])
def test_lattice_form_over_its_range_of_contrasts(cuda, nx, ny, nrhs, contrast):
    """eps at random over a factor of 8 and 30 in every element, and in layers along
    y with a factor of 40; the iterations stay within the bound that the cap is
    compared with."""
    om, m = _mesh(nx, ny)
    if contrast > 0.0:
        eps = np.exp(np.random.default_rng(nx).uniform(0.0, np.log(contrast), om.num_elements))
    else:
        eps = np.repeat(np.where(np.arange(ny) < ny // 2, 1.0, -contrast), 2 * nx)
    prob, err = _solve(cuda, om, m, eps, nrhs)
    assert prob._plan is not None and 1.5 < prob._kappa <= 64.0
    assert prob.last_iters <= prob._least_cap(1e-12) and prob.last_iters < 2 * nx
    # as above, < 400 sqrt(40)
    assert err <= 3e-9


@pytest.mark.gpu
def test_long_lines_split_their_columns(cuda):
    """600 columns: a block sweeps 16 right-hand sides, and the last takes one."""
    om, m = _mesh(600, 8)
    eps = np.random.default_rng(6).uniform(10.0, 14.0, om.num_elements)
    prob, err = _solve(cuda, om, m, eps, 33)
    assert prob._plan is not None and prob.last_iters <= 14 and err <= 1e-9


@pytest.mark.gpu
def test_moved_nodes_take_the_diagonal_form(cuda):
    """The separable operator is that of equal cells: on a structured mesh whose nodes
    were moved (columns graded towards a contact) it would be the wrong operator."""
    om, m = _mesh(40, 20)
    eps = np.random.default_rng(3).uniform(10.0, 14.0, om.num_elements)
    for mesh in (om, m):
        mesh.nodes[:, 0] = mesh.Lx * (mesh.nodes[:, 0] / mesh.Lx) ** 3
    prob, err = _solve(cuda, om, m, eps, 2)
    # as above, the condition number that much larger as the smallest cell is narrower
    assert prob._plan is None and err <= 1e-9 * 40
