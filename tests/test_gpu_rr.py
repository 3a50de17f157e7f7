"""Rayleigh-Ritz step (Cholesky congruence and tridiagonalisation in registers,
division-free bisection) through the batched solver: every block width (the
register tiles of orders 12 to 48), exactly repeated levels, decoupled blocks
(zero couplings in the tridiagonal matrix), and a start block with dependent
columns, against dense eigenvalues."""
import numpy as np
import pytest

from oracle import fem as O

pytestmark = pytest.mark.gpu


def _pencil(nx, ny, copies, seed):
    om = O.structured_mesh(1, nx, ny, float(nx), float(ny))
    rng = np.random.default_rng(seed)
    c = np.full(om.num_elements, 0.5)
    V = -0.3 * np.exp(-((om.nodes[:, 0] - nx / 2) ** 2 + (om.nodes[:, 1] - ny / 2) ** 2) / 18.0)
    V = V + (0.01 * rng.standard_normal(V.size) if seed else 0.0)
    a = O.assemble(om, c, V)
    import scipy.sparse as sp
    H, M = (sp.block_diag([x] * copies, format="csr") for x in (a.H, a.M))
    H.sort_indices(), M.sort_indices()
    return H, M


def _solve(torch, cuda, H, M, k, b, precision, x0=None):
    from qdsim_b200.eigen import lobpcg_packed
    t = lambda a, d: torch.from_numpy(np.ascontiguousarray(a.astype(d))).to(cuda)  # noqa: E731
    assert np.array_equal(H.indices, M.indices)
    E, X, R, it, info, st = lobpcg_packed(
        np.array([0, H.shape[0]], np.int32), t(H.indptr, np.int32), t(H.indices, np.int32),
        t(H.data, np.float64), t(M.data, np.float64), k, b=b, precision=precision, tol=1e-12,
        max_iter=3000, allow_not_converged=False, x0=x0)
    return E[0].cpu().numpy(), X.cpu().numpy()


def _dense(H, M, k):
    L = np.linalg.cholesky(M.toarray())
    A = np.linalg.solve(L, np.linalg.solve(L, H.toarray()).T)
    return np.linalg.eigvalsh(0.5 * (A + A.T))[:k]


@pytest.mark.parametrize("b,k", [(4, 1), (4, 2), (8, 5), (12, 8), (16, 12)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("copies", [1, 2, 3])
def test_levels_of_every_block_width(cuda, b, k, precision, copies):
    """copies > 1: the pencil is a direct sum of equal blocks, every level
    repeated exactly (an odd k or guard count may cut a group, which the
    stopping estimate cannot resolve: such cases are left out)."""
    import torch
    H, M = _pencil(16, 16, copies, 0)      # square symmetry: more repeated levels
    ref = _dense(H, M, b + 1)
    if ref[b - 1] - ref[k - 1] < 1e-6 * abs(ref[k - 1]):
        pytest.skip("the block's edge cuts a group of equal levels")
    E, X = _solve(torch, cuda, H, M, k, b, precision)
    # eigenvalue errors are quadratic in the residual: 1e-12 of |E|
    assert np.abs(E - ref[:k]).max() <= 1e-9 * np.abs(ref[:k]).max()
    G = X.T @ (M @ X)
    assert np.abs(G - np.eye(k)).max() <= 1e-8


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_dependent_start_block(cuda, precision):
    """Two equal and one zero start vector: a vanishing Cholesky pivot in X, so
    the first steps take the fallback."""
    import torch
    H, M = _pencil(20, 14, 1, 1)
    ref = _dense(H, M, 6)
    rng = np.random.default_rng(0)
    x0 = rng.standard_normal((H.shape[0], 6))
    x0[:, 3] = x0[:, 1]
    x0[:, 5] = 0.0
    E, _ = _solve(torch, cuda, H, M, 6, 12, precision, x0=torch.from_numpy(x0).to(cuda))
    assert np.abs(E - ref).max() <= 1e-9 * np.abs(ref).max()
