"""Poisson solves from several threads and streams: what one thread or stream sets
up must not reach into another's launches."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(cuda, nx, ny, seed):
    from qdsim_b200 import mesh as Mh, poisson as P
    rng = np.random.default_rng(seed)
    m = Mh.StructuredMesh(1, nx, ny, float(nx), float(ny))
    eps = np.repeat(np.tile(rng.uniform(8.0, 14.0, nx), ny), 2)
    return P.PoissonProblem(m, eps, device=cuda), 1.6e5 * rng.standard_normal(m.num_nodes)


def test_two_threads_solve_lattices_of_unlike_sizes(cuda):
    """A long line needs 170 KB of shared memory per block, a short one 1 KB; each
    thread solves on its own stream and finds what it finds alone."""
    import torch
    jobs = [_problem(cuda, 7000, 4, 0), _problem(cuda, 40, 20, 1)]
    alone = [p.solve(rho, 0.0, 0.5, max_iter=200000).clone() for p, rho in jobs]
    torch.cuda.synchronize()
    errors, start = [], threading.Barrier(len(jobs))

    def work(i):
        prob, rho = jobs[i]
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                rho = torch.from_numpy(rho).to(cuda)
                start.wait(30)
                for _ in range(150):
                    same = torch.equal(prob.solve(rho, 0.0, 0.5, max_iter=200000), alone[i])
                    if not same:
                        raise AssertionError(f"thread {i}: other values than alone")
        except Exception as exc:   # reported below, in the test's own thread
            errors.append(exc)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_a_new_problem_leaves_nothing_running(cuda):
    """Whatever the constructor computes is complete when it returns, so that the
    first solve may run on any stream.  The factors of a line of 7000 cells take
    their one thread milliseconds."""
    import torch
    _problem(cuda, 7000, 4, 2)
    assert torch.cuda.current_stream().query()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        _problem(cuda, 7000, 4, 3)
        assert side.query()
