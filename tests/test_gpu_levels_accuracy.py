"""Accuracy of the batched solver's levels at tight tolerances, both precisions:
what is left is rounding, in proportion to the order of the projected problem."""
import numpy as np
import pytest

from test_gpu_rr import _pencil

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,k", [(4, 2), (8, 5), (12, 8), (16, 12)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny,seed", [(16, 16, 0), (20, 14, 1), (30, 20, 2), (30, 30, 3)])
@pytest.mark.parametrize("tol", [1e-12, 1e-14])
def test_levels_to_rounding(cuda, b, k, precision, nx, ny, seed, tol):
    import scipy.linalg as sl
    import torch
    from qdsim_b200.eigen import lobpcg_packed
    H, M = _pencil(nx, ny, 1, seed)
    ref = sl.eigh(H.toarray(), M.toarray(), eigvals_only=True)
    if ref[b - 1] - ref[k - 1] < 1e-6 * abs(ref[k - 1]):
        pytest.skip("the block's edge cuts a group of equal levels")
    t = lambda a, d: torch.from_numpy(np.ascontiguousarray(a.astype(d))).to(cuda)  # noqa: E731
    E, X, *_ = lobpcg_packed(
        np.array([0, H.shape[0]], np.int32), t(H.indptr, np.int32), t(H.indices, np.int32),
        t(H.data, np.float64), t(M.data, np.float64), k, b=b, precision=precision, tol=tol,
        max_iter=3000, allow_not_converged=False)
    E, X = E[0].cpu().numpy(), X.cpu().numpy()
    # tol of each level, and the rounding of a projected problem of order 3 b whose
    # norm is at most the largest level
    assert np.all(np.abs(E - ref[:k]) <= tol * np.abs(ref[:k]) + 3 * b * 2.2e-16 * ref[-1])
    assert np.abs(X.T @ (M @ X) - np.eye(k)).max() <= 3 * b * 2.2e-16
