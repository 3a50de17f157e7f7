"""The thread-per-element adjoint pass against the FP64 oracle gradient on
random amplitudes: every order, real and complex, one state, a few and the
most, element counts around one block of 64 threads, and weights in host and
in device memory (bitwise the same)."""
import numpy as np
import pytest

from oracle import adjoint as OA, fem as O

pytestmark = pytest.mark.gpu


def _abs_gradients(om, psi, w):
    """The oracle's sums with every factor replaced by its magnitude (tables by
    their largest entry): what one rounding per operation is relative to."""
    tab = O.ref_tables(om.order)
    A, g00, g01, g11 = O.element_geometry(om.nodes, om.elems)
    P = np.abs(psi[om.elems])
    U = np.einsum("eis,ejs,s->e", P, P, np.abs(w))
    c = A * U * (np.abs(g00) * np.abs(tab.Sxx).max() + np.abs(g01) * np.abs(tab.Sxy).max()
                 + np.abs(g11) * np.abs(tab.Syy).max())
    V = np.zeros(om.num_nodes)
    np.add.at(V, om.elems.ravel(), np.repeat(A * U * np.abs(tab.T).max(), om.elems.shape[1]))
    return V, c


@pytest.mark.parametrize("order,nx,ny", [(1, 2, 2), (1, 8, 4), (1, 13, 5), (2, 2, 2), (2, 11, 3),
                                         (3, 2, 1), (3, 13, 5)])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("ns", [1, 3, 16])
def test_element_pass(cuda, order, nx, ny, cplx, ns):
    import torch
    from qdsim_b200 import _native as N, adjoint as A, fem as F, mesh as Mh
    rng = np.random.default_rng([order, nx, ny, ns])
    om = O.structured_mesh(order, nx, ny, 1.7 * nx, 0.9 * ny)
    prob = F.FEMProblem(Mh.StructuredMesh(order, nx, ny, 1.7 * nx, 0.9 * ny), device=cuda)
    dm = prob.d_dofmap.cpu().numpy()
    n = int(dm.max()) + 1
    X = rng.standard_normal((n, ns))
    w = rng.standard_normal(ns)
    if cplx:
        X = X + 1j * rng.standard_normal((n, ns))
        w = w + 1j * rng.standard_normal(ns)
    psi = np.zeros((om.num_nodes, ns), X.dtype)
    psi[dm >= 0] = X[dm[dm >= 0]]
    gV, gc = OA.gradients(om, psi, w)
    aV, ac = _abs_gradients(om, psi, w)
    Xd = torch.from_numpy(X).to(cuda)
    dV, dc = A.energy_gradients(prob, Xd, w)
    dV, dc = dV.cpu().numpy().copy(), dc.cpu().numpy().copy()
    k = om.elems.shape[1]
    # ns k^2 products in up to four operations each, 32 for the geometry, the
    # tables' own rounding and the sum over a node's elements; both sides round
    tol = 2 * (4 * ns * k * k + 32) * 2.0 ** -53
    assert np.all(np.abs(dV - gV) <= tol * aV + 1e-300)
    assert np.all(np.abs(dc - gc) <= tol * ac + 1e-300)

    m = prob.mesh
    wd = torch.as_tensor(np.stack([w.real, w.imag], 1).ravel() if cplx else w).to(cuda)
    nptr, nadj = prob.node_adjacency()
    V2 = torch.empty(m.num_nodes, dtype=torch.float64, device=cuda)
    c2 = torch.empty(m.num_elements, dtype=torch.float64, device=cuda)
    work = torch.empty(m.num_elements * k, dtype=torch.float64, device=cuda)
    N.check(N.lib().qd_adjoint(order, m.num_nodes, m.num_elements, ns, int(cplx),
                               N.ptr(prob.d_nodes), N.ptr(prob.d_elems), N.ptr(prob.d_dofmap),
                               N.ptr(Xd), N.ptr(wd), N.ptr(nptr), N.ptr(nadj), N.ptr(V2),
                               N.ptr(c2), N.ptr(work),
                               torch.cuda.current_stream().cuda_stream), "qd_adjoint")
    assert np.array_equal(V2.cpu().numpy(), dV) and np.array_equal(c2.cpu().numpy(), dc)
