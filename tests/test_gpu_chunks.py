"""Rows per chunk of the batched eigensolve: the default of a batch above 32,768 rows,
and chunks that end inside a sub-tile, against dense eigenvalues."""
import numpy as np
import pytest

from oracle import fem as O

pytestmark = pytest.mark.gpu


def _pencil(seed):
    om = O.structured_mesh(1, 21, 25, 21.0, 30.0)
    rng = np.random.default_rng(seed)
    a = O.assemble(om, rng.uniform(0.5, 1.0, om.num_elements), -0.3 * rng.random(om.num_nodes))
    H, M = a.H.tocsr(), a.M.tocsr()
    H.sort_indices(), M.sort_indices()
    L = np.linalg.cholesky(M.toarray())
    A = np.linalg.solve(L, np.linalg.solve(L, H.toarray()).T)
    return H, M, np.linalg.eigvalsh(0.5 * (A + A.T))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("chunk_rows,dots", [(None, 80), (128, 3), (192, 3), (320, 3)])
def test_levels(cuda, precision, chunk_rows, dots):
    import torch
    from qdsim_b200.eigen import lobpcg_packed
    kinds = [_pencil(s) for s in range(4)]
    ps = [kinds[d % 4] for d in range(dots)]
    off = np.concatenate([[0], np.cumsum([H.shape[0] for H, *_ in ps])]).astype(np.int32)
    assert (off[-1] > 32768) == (chunk_rows is None)
    nnz = np.concatenate([[0], np.cumsum([H.nnz for H, *_ in ps])])
    t = lambda a, d: torch.from_numpy(np.concatenate(a).astype(d)).to(cuda)  # noqa: E731
    E, X, *_ = lobpcg_packed(
        off, t([[0]] + [H.indptr[1:] + z for (H, *_), z in zip(ps, nnz)], np.int32),
        t([H.indices + o for (H, *_), o in zip(ps, off)], np.int32), t([H.data for H, *_ in ps], float),
        t([M.data for _, M, _ in ps], float), 8, b=12, precision=precision, tol=1e-10,
        max_iter=3000, chunk_rows=chunk_rows, allow_not_converged=False)
    E = E.cpu().numpy()
    for d, (H, M, ref) in enumerate(ps):
        # errors are quadratic in the residual (1e-10 of |E|); the scale is the
        # whole spectrum's rounding
        assert np.abs(E[d] - ref[:8]).max() <= 1e-10 * np.abs(ref[:8]).max() + 1e-13 * ref[-1]
