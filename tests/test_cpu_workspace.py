"""Workspace sizes of the batched eigensolve: a workspace for a batch serves every
smaller one, whatever rows per chunk the sizes lead to."""
import ctypes as C

import numpy as np
import pytest

from qdsim_b200 import _native as N


def _bytes(n_dots, rows, nnz, b, mode, opts=None):
    out = C.c_size_t()
    assert N.lib().qd_lobpcg_workspace_size(n_dots, rows, nnz, b, mode, None, N.ptr(opts),
                                            C.byref(out)) == N.QD_OK
    return out.value


@pytest.mark.parametrize("b", [4, 12, 16])
@pytest.mark.parametrize("mode", [N.QD_PREC_FP64, N.QD_PREC_MIXED])
@pytest.mark.parametrize("n_dots", [1, 40])
@pytest.mark.parametrize("chunk_rows", [0, 2048])
def test_size_grows_with_the_rows(b, mode, n_dots, chunk_rows):
    opts = np.zeros(1, dtype=N.LOBPCG_OPTS_DTYPE)
    opts["chunk_rows"] = chunk_rows
    rows = [1000, 20000, 32000, 32768, 32769, 33000, 40000, 60000, 120000, 299000, 300000, 300001,
            305000, 320000, 400000, 1000000]
    sizes = [_bytes(n_dots, r, 11 * r, b, mode, opts) for r in rows]
    assert sizes == sorted(sizes)
    # and with few nonzeros: the rows' own part alone
    sizes = [_bytes(n_dots, r, 2000000, b, mode, opts) for r in rows]
    assert sizes == sorted(sizes)


def test_every_multiple_of_64_from_128_is_taken():
    """Shorter chunks mean more of them: each accepted value has its own size, so the
    rows per chunk that small batches take by default can be asked for too."""
    opts = np.zeros(1, dtype=N.LOBPCG_OPTS_DTYPE)
    sizes = []
    for chunk in (128, 192, 256, 320, 512):
        opts["chunk_rows"] = chunk
        sizes.append(_bytes(4, 400000, 4000000, 12, N.QD_PREC_MIXED, opts))
    assert sizes == sorted(sizes, reverse=True) and len(set(sizes)) == len(sizes)
    opts["chunk_rows"] = 64
    other = _bytes(4, 400000, 4000000, 12, N.QD_PREC_MIXED, opts)
    opts["chunk_rows"] = 0
    assert other == _bytes(4, 400000, 4000000, 12, N.QD_PREC_MIXED, opts)


def test_the_tuner_tries_the_default_of_small_batches():
    from qdsim_b200 import autotune as AT
    assert 128 in AT.SPACE["chunk_rows"] and AT.DEFAULTS["chunk_rows"] in AT.SPACE["chunk_rows"]
