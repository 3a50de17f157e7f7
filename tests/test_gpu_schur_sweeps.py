"""qd_complex_schur beyond 60 sweeps, where the kernel rotates Z itself instead of
logging the rotations for a second kernel: the same triangular matrix, bit for bit,
and the same Z up to rounding."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 5, 16, 41, 143, 144])
@pytest.mark.parametrize("hermitian", [False, True])
def test_both_forms_of_z(cuda, n, hermitian):
    import torch
    from qdsim_b200 import _native as N
    from qdsim_b200.fem import stream_ptr
    rng = np.random.default_rng(n)
    A = 1e-3 * (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))
    A = np.diag(np.sort(rng.uniform(0.0, 3.0, n))) + (A + A.conj().T if hermitian else A)
    Ad = torch.from_numpy(np.ascontiguousarray(A)).to(cuda)
    got = []
    for sweeps in (60, 61):
        T, Z = torch.zeros_like(Ad), torch.zeros_like(Ad)
        ran = C.c_int32()
        N.check(N.lib().qd_complex_schur(n, N.ptr(Ad), n, N.ptr(T), N.ptr(Z), n, sweeps, C.byref(ran),
                                         stream_ptr()), "qd_complex_schur")
        got.append((T.cpu().numpy(), Z.cpu().numpy(), ran.value))
    (T, Z, s), (T1, Z1, s1) = got
    assert s == s1 and np.array_equal(T, T1)
    # up to 20 sweeps of n rotations of each entry, and their rounding
    tol = 20 * n * 2.3e-16
    assert np.abs(Z - Z1).max() <= tol
    assert np.abs(A @ Z1 - Z1 @ T1).max() <= tol * np.abs(A).max() * np.sqrt(n)
    assert np.abs(Z1.conj().T @ Z1 - np.eye(n)).max() <= tol
