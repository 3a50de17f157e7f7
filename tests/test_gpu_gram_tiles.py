"""Gram partials of the batched solver (both matrices per thread, products in
pairs, sub-tiles of 64 or 80 rows): chunks that end just before, at and after a
sub-tile, row counts below the number of row groups, and every block width, in
one batch of unlike dots, against dense eigenvalues."""
import numpy as np
import pytest

from oracle import fem as O

pytestmark = pytest.mark.gpu

# interior rows of P1 meshes nx x ny: (nx - 1)(ny - 1)
SIZES = [(8, 10), (9, 9), (6, 14), (80, 2), (9, 11), (10, 10), (9, 21), (8, 24), (17, 17), (21, 25)]
ROWS = [63, 64, 65, 79, 80, 81, 160, 161, 256, 480]


def _pencils(seed):
    rng = np.random.default_rng(seed)
    out = []
    for (nx, ny), n in zip(SIZES, ROWS):
        om = O.structured_mesh(1, nx, ny, float(nx), 1.3 * ny)
        V = -0.3 * rng.random(om.num_nodes)
        a = O.assemble(om, rng.uniform(0.5, 1.0, om.num_elements), V)
        H, M = a.H.tocsr(), a.M.tocsr()
        H.sort_indices(), M.sort_indices()
        assert H.shape[0] == n and np.array_equal(H.indices, M.indices)
        out.append((H, M))
    return out


@pytest.mark.parametrize("b,k", [(4, 2), (8, 5), (12, 8), (16, 11)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("chunk_rows", [128, 192, 1024])
def test_levels_at_the_edges_of_sub_tiles(cuda, b, k, precision, chunk_rows):
    import torch
    from qdsim_b200.eigen import lobpcg_packed
    ps = _pencils(b)
    off = np.concatenate([[0], np.cumsum([H.shape[0] for H, _ in ps])]).astype(np.int32)
    nnz = np.concatenate([[0], np.cumsum([H.nnz for H, _ in ps])])
    indptr = np.concatenate([[0]] + [H.indptr[1:] + z for (H, _), z in zip(ps, nnz)])
    ind = np.concatenate([H.indices + o for (H, _), o in zip(ps, off)])
    t = lambda a, d: torch.from_numpy(np.ascontiguousarray(a.astype(d))).to(cuda)  # noqa: E731
    E, X, R, it, info, st = lobpcg_packed(
        off, t(indptr, np.int32), t(ind, np.int32), t(np.concatenate([H.data for H, _ in ps]), float),
        t(np.concatenate([M.data for _, M in ps]), float), k, b=b, precision=precision, tol=1e-10,
        max_iter=3000, chunk_rows=chunk_rows, allow_not_converged=False)
    E = E.cpu().numpy()
    for d, (H, M) in enumerate(ps):
        L = np.linalg.cholesky(M.toarray())
        A = np.linalg.solve(L, np.linalg.solve(L, H.toarray()).T)
        ref = np.linalg.eigvalsh(0.5 * (A + A.T))
        # errors are quadratic in the residual (1e-10 of |E|); the scale is the
        # whole spectrum's rounding
        assert np.abs(E[d] - ref[:k]).max() <= 1e-10 * np.abs(ref[:k]).max() + 1e-13 * ref[-1]
