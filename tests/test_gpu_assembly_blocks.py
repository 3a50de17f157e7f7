"""Assembly with fewer rows per block than a block takes at most (small meshes), and
at the row counts where the rows per block change: equal to the oracle, and equal
bits to the same rows assembled as part of a larger batch."""
import numpy as np
import pytest

from oracle import fem as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,sizes", [
    (1, [(3, 3), (9, 7), (40, 60), (97, 110), (300, 250)]),
    (2, [(2, 2), (7, 9), (41, 29), (120, 100)]),
    (3, [(1, 1), (2, 3), (6, 5), (13, 17), (61, 40)]),
])
@pytest.mark.parametrize("cap", [False, True])
def test_blocks_of_every_size(cuda, order, sizes, cap):
    import torch
    from qdsim_b200 import fem as F, mesh as Mh
    for nx, ny in sizes:
        rng = np.random.default_rng([order, nx, ny])
        om = O.structured_mesh(order, nx, ny, float(nx), 1.3 * ny)
        c, V = rng.uniform(0.3, 1.0, om.num_elements), rng.standard_normal(om.num_nodes)
        W = rng.uniform(0.0, 1.0, om.num_nodes) if cap else None
        m = Mh.StructuredMesh(order, nx, ny, float(nx), 1.3 * ny)
        if m.boundary.all():
            continue
        prob = F.FEMProblem(m, device=cuda)
        out = prob.assemble(c, V, W)
        ref = O.assemble(om, c, V, W) if cap else O.assemble(om, c, V)
        for key, want in (("H", ref.H), ("M", ref.M)):
            got = prob.to_scipy(out[key])
            # sums of at most 16 elements' entries of order one or the row's own scale
            assert abs(got - want).max() <= 1e-13 * abs(want).max()
        if cap:
            assert abs(prob.to_scipy(out["Himag"]) + ref.Wm).max() <= 1e-13 * abs(ref.Wm).max()
        again = prob.assemble(c, V, W)
        assert all(torch.equal(out[k], again[k]) for k in out)


def test_a_dot_alone_and_in_a_large_batch(cuda):
    """48 rows per block on its own, the most in the batch: equal bits."""
    import torch
    from qdsim_b200 import workloads as W
    from qdsim_b200.batch import DeviceBatch, HostBatch
    dots = [W.sweep_dot(i, nx=80) for i in range(24)]
    out = []
    for ds in (dots[:1], dots):
        db = DeviceBatch(HostBatch(ds), cuda)
        db.upload(non_blocking=False)
        db.assemble()
        db.check_status()
        out.append(db)
    nnz = int(out[0].H.numel())
    assert torch.equal(out[0].H, out[1].H[:nnz]) and torch.equal(out[0].M, out[1].M[:nnz])
