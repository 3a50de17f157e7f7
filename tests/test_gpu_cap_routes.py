"""The two product kernels of the open system (rows in lattice tiles, a block per 16
rows) give equal bits on either side of the rule that chooses between them, by the
type, the columns, the rows and the nonzeros per row."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,nx,ny", [(1, 343, 352), (2, 211, 137), (3, 121, 77), (2, 40, 30)])
@pytest.mark.parametrize("b", [1, 7, 16, 20, 21, 32, 33, 48, 49, 64])
@pytest.mark.parametrize("fp32", [0, 1])
def test_both_kernels_give_equal_bits(cuda, order, nx, ny, b, fp32):
    import torch
    from qdsim_b200 import _native as N, fem as F, mesh as Mh
    from qdsim_b200.fem import stream_ptr
    m = Mh.StructuredMesh(order, nx, ny, float(nx), float(ny))
    prob = F.FEMProblem(m, device=cuda)
    g = torch.Generator(device=cuda).manual_seed(order * 100 + b)
    ct, rt = (torch.complex64, torch.float32) if fp32 else (torch.complex128, torch.float64)
    H, G, M = (torch.randn(prob.nnz, dtype=rt, device=cuda, generator=g) for _ in range(3))
    X = torch.randn(prob.n, b, dtype=ct, device=cuda, generator=g)
    got = []
    # nonzeros: of a P2 lattice (the tiles' best case), of a denser pattern, not
    # known; and no lattice
    for width, nnz in ((order * nx - 1, int(11.4 * prob.n)), (order * nx - 1, 20 * prob.n),
                       (order * nx - 1, 0), (0, 0)):
        AX, MX = (torch.full((prob.n, b + 1), 7.0, dtype=ct, device=cuda) for _ in range(2))
        N.check(N.lib().qd_cap_spmm_pattern(
            prob.n, nnz, width, b, fp32, N.ptr(prob.d_rowptr), N.ptr(prob.d_col), N.ptr(H), N.ptr(G),
            N.ptr(M), N.ptr(X), b, N.ptr(AX), N.ptr(MX), b + 1, stream_ptr()), "qd_cap_spmm_pattern")
        got.append((AX, MX))
    for ax, mx in got[1:]:
        assert torch.equal(ax, got[0][0]) and torch.equal(mx, got[0][1])
    # the rows kernel against the matrix itself
    idx = np.random.default_rng(b).integers(0, prob.n, 50)
    A = prob.to_scipy(H.double())[idx] + 1j * prob.to_scipy(G.double())[idx]
    x = X.cpu().numpy().astype(np.complex128)
    y = got[-1][0][:, :b].cpu().numpy()[idx]
    # rows of at most 37 products, in the arithmetic of the type
    tol = 37 * (1.2e-7 if fp32 else 2.3e-16)
    assert np.linalg.norm(y - A @ x) <= tol * np.linalg.norm(abs(A) @ abs(x))
