"""qd_cap_spmm_lattice, whose rows are taken in 4 x 4 tiles of the lattice,
against qd_cap_spmm and scipy: lattices that the tiles do not divide, lines
shorter than a tile, rows longer than one staging (P3 has 37 entries), and
widths that must be ignored."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,nx,ny,b", [(1, 5, 5, 1), (1, 18, 3, 16), (2, 3, 3, 17), (2, 9, 14, 48),
                                           (2, 33, 2, 33), (2, 41, 37, 5), (3, 7, 6, 31),
                                           (3, 12, 21, 64)])
@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("cap", [True, False])
def test_lattice_products(cuda, order, nx, ny, b, fp32, cap):
    import torch
    from qdsim_b200 import _native as N, fem as F, mesh as Mh
    from qdsim_b200.fem import stream_ptr
    m = Mh.StructuredMesh(order, nx, ny, float(nx), float(ny))
    prob = F.FEMProblem(m, device=cuda)
    rng = np.random.default_rng([order, nx, ny, b])
    out = prob.assemble(rng.uniform(0.3, 1.0, m.num_elements), rng.standard_normal(m.num_nodes),
                        rng.uniform(0.0, 1.0, m.num_nodes))
    ct, rt = (torch.complex64, torch.float32) if fp32 else (torch.complex128, torch.float64)
    H, M, G = (out[k].to(rt) for k in ("H", "M", "Himag"))
    X = torch.from_numpy(rng.standard_normal((prob.n, b)) + 1j * rng.standard_normal((prob.n, b))).to(cuda, ct)
    width = order * nx - 1
    got = []
    for w in (width, 0, width + 1, -3, prob.n):
        AX, MX = (torch.full((prob.n, b + 2), 7.0, dtype=ct, device=cuda) for _ in range(2))
        N.check(N.lib().qd_cap_spmm_lattice(
            prob.n, w, b, fp32, N.ptr(prob.d_rowptr), N.ptr(prob.d_col), N.ptr(H),
            N.ptr(G) if cap else None, N.ptr(M), N.ptr(X), b, N.ptr(AX), N.ptr(MX), b + 2,
            stream_ptr()), "qd_cap_spmm_lattice")
        assert (AX[:, b:] == 7.0).all() and (MX[:, b:] == 7.0).all()
        got.append((AX[:, :b].cpu().numpy(), MX[:, :b].cpu().numpy()))
    for ax, mx in got[1:]:
        assert np.array_equal(ax, got[0][0]) and np.array_equal(mx, got[0][1])
    A = prob.to_scipy(H.double()) + (1j * prob.to_scipy(G.double()) if cap else 0)
    x = X.cpu().numpy().astype(np.complex128)
    # rows of at most 37 products of order one, in the arithmetic of the type
    tol = 37 * (1.2e-7 if fp32 else 2.3e-16)
    for y, B in ((got[0][0], A), (got[0][1], prob.to_scipy(M.double()))):
        assert np.linalg.norm(y - B @ x) <= tol * np.linalg.norm(abs(B) @ abs(x))
