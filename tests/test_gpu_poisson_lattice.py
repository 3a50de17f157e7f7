"""The separably preconditioned Poisson solve (qd_poisson_lattice_solve)
against the FP64 oracle (sparse LU), at the edges of its tiles: one and two
cells, odd and even ny, row counts around the 64-mode tile and the 16-deep
stage, right-hand sides that do not divide the block.  And the rule that picks
it, on the CPU."""
import numpy as np
import pytest

from oracle import fem as O, poisson as OP

CASES = [  # nx, ny, nrhs
    (1, 1, 1), (2, 1, 2), (3, 2, 1), (5, 7, 3), (40, 31, 64), (33, 32, 5), (20, 126, 2),
    (21, 128, 7), (64, 130, 1), (17, 255, 33), (300, 12, 256), (150, 63, 100),
]


def _inputs(nx, ny, nrhs, layered, seed=0):
    rng = np.random.default_rng([seed, nx, ny, nrhs])
    om = O.structured_mesh(1, nx, ny, 2.0 * nx, 1.5 * ny)
    if layered:
        eps = np.repeat(np.tile(rng.uniform(4.0, 14.0, nx), ny), 2)
    else:
        eps = rng.uniform(10.0, 14.0, om.num_elements)
    R = 1.6e5 * rng.standard_normal((om.num_nodes, nrhs))
    return om, eps, R, rng.uniform(-0.2, 0.2, nrhs), rng.uniform(0.0, 1.0, nrhs)


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nrhs", CASES)
@pytest.mark.parametrize("layered", [False, True])
def test_lattice_solve_matches_oracle(cuda, nx, ny, nrhs, layered):
    import torch
    from qdsim_b200 import mesh as Mh, poisson as P
    om, eps, R, vp, vn = _inputs(nx, ny, nrhs, layered)
    ref = OP.solve(om, eps, R, vp, vn).reshape(om.num_nodes, nrhs)
    prob = P.PoissonProblem(Mh.StructuredMesh(1, nx, ny, om.Lx, om.Ly), eps, device=cuda)
    assert prob._plan is not None
    x0 = None
    if nrhs > 1:   # a warm start changes the work, not the answer
        x0 = torch.from_numpy(0.5 * ref + 0.01 * np.cos(np.arange(ref.size)).reshape(ref.shape))
    got = prob.solve(R, vp, vn, tol=1e-12, x0=x0).cpu().numpy().reshape(om.num_nodes, nrhs)
    # residual 1e-12 of the right-hand side, amplified by at most the condition
    # number of the discrete Laplacian in the energy sense (sqrt: < 400 here)
    assert np.abs(got - ref).max() <= 1e-9 * np.abs(ref).max()
    assert prob.last_relres <= 1e-12
    again = prob.solve(R, vp, vn, tol=1e-12, x0=x0).cpu().numpy().reshape(om.num_nodes, nrhs)
    assert np.array_equal(got, again)


def test_condition_bound_and_means():
    """gx, gy are the column sums of the oracle's stiffness entries over ny, and
    the bound covers the extreme generalised eigenvalues of (K, Kt)."""
    from qdsim_b200 import mesh as Mh, poisson as P
    nx, ny = 7, 6
    om, eps, *_ = _inputs(nx, ny, 1, False, seed=2)
    m = Mh.StructuredMesh(1, nx, ny, om.Lx, om.Ly)
    gx, gy, kappa = P.lattice_means(m, eps)
    K = _stiffness(om, eps)
    node = np.arange((nx + 1) * (ny + 1)).reshape(ny + 1, nx + 1)
    sx = [-K[node[:, i], node[:, i + 1]].sum() / ny for i in range(nx)]
    sy = [-K[node[:-1, i], node[1:, i]].sum() / ny for i in range(nx + 1)]
    assert np.allclose(gx, sx, rtol=1e-13) and np.allclose(gy, sy, rtol=1e-13)
    w = np.ones(ny + 1)
    w[0] = w[-1] = 0.5
    Kt = np.zeros_like(K)
    def edge(a, b, g):
        Kt[a, a] += g; Kt[b, b] += g; Kt[a, b] -= g; Kt[b, a] -= g   # noqa: E702
    for j in range(ny + 1):
        for i in range(nx):
            edge(node[j, i], node[j, i + 1], gx[i] * w[j])
    for j in range(ny):
        for i in range(nx + 1):
            edge(node[j, i], node[j + 1, i], gy[i])
    free = node[:, 1:-1].ravel()
    ev = np.linalg.eigvals(np.linalg.solve(Kt[np.ix_(free, free)], K[np.ix_(free, free)])).real
    assert ev.max() / ev.min() <= kappa * (1 + 1e-12)
    # layered eps: the separable operator is the operator
    om, eps, *_ = _inputs(nx, ny, 1, True, seed=3)
    assert P.lattice_means(m, eps)[2] <= 1 + 1e-12


def _stiffness(om, eps):
    """Dense P1 stiffness from the element gradients."""
    K = np.zeros((om.num_nodes, om.num_nodes))
    for e, el in enumerate(om.elems):
        p = om.nodes[el]
        J = np.array([p[1] - p[0], p[2] - p[0]])
        G = np.linalg.inv(J) @ np.array([[-1.0, 1.0, 0.0], [-1.0, 0.0, 1.0]])
        K[np.ix_(el, el)] += eps[e] * 0.5 * abs(np.linalg.det(J)) * G.T @ G
    return K


def test_rule_leaves_other_problems_to_the_diagonal_form():
    from qdsim_b200 import mesh as Mh, poisson as P
    m = Mh.StructuredMesh(1, 6, 4, 6.0, 4.0)
    eps = np.full(m.num_elements, 1.0)
    eps[m.centroids()[:, 1] > 2.0] = 200.0        # contrast along y beyond the bound
    assert P.lattice_means(m, eps)[2] > P.LATTICE_KAPPA
    eps[3] = np.nan
    assert not P.lattice_means(m, eps)[2] <= P.LATTICE_KAPPA
