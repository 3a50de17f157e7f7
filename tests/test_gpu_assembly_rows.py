"""Assembly at the edges of its row blocks: rows of high valence, whose pairs
take several passes of a block, and plan arrays that start off the word
boundaries the wide loads need."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fans(count, valence):
    """Disjoint fans of triangles, all centres numbered first (P1)."""
    ang = 2 * np.pi * np.arange(valence) / valence
    nodes = np.zeros((count * (valence + 1), 2))
    elems = []
    for f in range(count):
        c = np.array([3.0 * (f % 16), 3.0 * (f // 16)])
        nodes[f] = c
        ring = count + f * valence + np.arange(valence)
        nodes[ring] = c + np.stack([np.cos(ang), np.sin(ang)], 1)
        elems += [(f, ring[i], ring[(i + 1) % valence]) for i in range(valence)]
    return nodes, np.array(elems, np.int32)


def _dense_p1(nodes, elems, c, V):
    """H and M of the P1 weak form, element by element: linear V times two
    shape functions by the interior three-point rule."""
    n = len(nodes)
    H, M = np.zeros((n, n)), np.zeros((n, n))
    lam = np.array([[1, 1, 4], [1, 4, 1], [4, 1, 1]]) / 6.0
    for e, el in enumerate(elems):
        p = nodes[el]
        J = np.array([p[1] - p[0], p[2] - p[0]])
        A = 0.5 * abs(np.linalg.det(J))
        G = np.linalg.inv(J) @ np.array([[-1.0, 1.0, 0.0], [-1.0, 0.0, 1.0]])
        he, me = c[e] * A * G.T @ G, np.zeros((3, 3))
        for q in lam:
            me += A / 3 * np.outer(q, q)
            he += A / 3 * (q @ V[el]) * np.outer(q, q)
        H[np.ix_(el, el)] += he
        M[np.ix_(el, el)] += me
    return H, M


def _call(torch, N, plan, nodes, elems, c, V, dev, shift):
    """qd_assemble with the index arrays `shift` elements into their buffers."""
    from qdsim_b200.fem import stream_ptr

    def at(a):
        buf = torch.zeros(a.size + shift, dtype=torch.from_numpy(a[:0]).dtype, device=dev)
        buf[shift:] = torch.from_numpy(a.ravel()).to(dev)
        return buf[shift:]

    d_nodes, d_c, d_V = (torch.from_numpy(np.ascontiguousarray(a)).to(dev) for a in (nodes, c, V))
    ix = [at(a) for a in (elems, plan.rowptr, plan.adjptr, plan.adj, plan.cptr, plan.contrib,
                          plan.slotcnt)]
    H = torch.full((plan.nnz,), np.nan, dtype=torch.float64, device=dev)
    M = torch.full_like(H, np.nan)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    N.check(N.lib().qd_assemble(
        1, N.QD_ASM_FEM, len(nodes), len(elems), plan.n, N.ptr(d_nodes), N.ptr(ix[0]), N.ptr(d_c),
        N.ptr(d_V), None, *(N.ptr(t) for t in ix[1:]), N.ptr(H), N.ptr(M), None, N.ptr(status),
        stream_ptr()), "qd_assemble")
    assert int(status.item()) == 0
    return H.cpu().numpy(), M.cpu().numpy()


@pytest.mark.parametrize("count,valence", [(1, 3), (128, 16), (129, 16), (150, 9), (300, 7)])
def test_high_valence_rows(cuda, count, valence):
    import torch
    from qdsim_b200 import _native as N
    from qdsim_b200.fem import build_pattern
    nodes, elems = _fans(count, valence)
    rng = np.random.default_rng([count, valence])
    c, V = rng.uniform(0.3, 1.0, len(elems)), rng.standard_normal(len(nodes))
    n = len(nodes)
    plan = build_pattern(elems, np.arange(n, dtype=np.int32), n, n)
    H, M = _call(torch, N, plan, nodes, elems, c, V, cuda, 0)
    Hr, Mr = _dense_p1(nodes, elems, c, V)
    rows = np.repeat(np.arange(n), np.diff(plan.rowptr))
    # sums of up to 16 entries of order one
    assert np.abs(H - Hr[rows, plan.col]).max() <= 1e-13 * np.abs(Hr).max()
    assert np.abs(M - Mr[rows, plan.col]).max() <= 1e-13 * np.abs(Mr).max()


@pytest.mark.parametrize("order", [1, 2, 3])
def test_plan_off_word_boundaries(cuda, order):
    import torch
    from qdsim_b200 import _native as N, mesh as Mh
    from qdsim_b200.fem import build_pattern, dof_map_for, stream_ptr
    m = Mh.StructuredMesh(order, 23, 17, 23.0, 17.0)
    dm, n = dof_map_for(m, True)
    P = build_pattern(m.elems, dm, n, m.num_nodes)
    rng = np.random.default_rng(order)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)  # noqa: E731
    d_nodes, c = t(m.nodes), t(rng.uniform(0.3, 1.0, m.num_elements))
    V, W = t(rng.standard_normal(m.num_nodes)), t(rng.uniform(0, 1, m.num_nodes))
    got = []
    for shift in (0, 1, 2, 3):
        ix = []
        for a in (m.elems.ravel(), P.rowptr, P.adjptr, P.adj, P.cptr, P.contrib, P.slotcnt):
            buf = torch.zeros(a.size + shift, dtype=t(a[:0]).dtype, device=cuda)
            buf[shift:] = t(a)
            ix.append(buf[shift:])
        H, M, G = (torch.full((P.nnz,), np.nan, dtype=torch.float64, device=cuda) for _ in range(3))
        status = torch.zeros(1, dtype=torch.int32, device=cuda)
        N.check(N.lib().qd_assemble(
            order, N.QD_ASM_FEM, m.num_nodes, m.num_elements, n, N.ptr(d_nodes), N.ptr(ix[0]),
            N.ptr(c), N.ptr(V), N.ptr(W), *(N.ptr(x) for x in ix[1:]), N.ptr(H), N.ptr(M),
            N.ptr(G), N.ptr(status), stream_ptr()), "qd_assemble")
        got.append([x.cpu().numpy() for x in (H, M, G)])
    for g in got:
        for x, y in zip(g, got[0]):
            assert np.isfinite(x).all() and np.array_equal(x, y)
