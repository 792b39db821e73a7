"""cipsi_davidson at the sizes where its products change shape: fewer rows than
a CTA's threads or than vectors in the block, remainders of the unrolled sums,
rows enough that a thread goes through all columns.  For |Hx - theta x| = r an
eigenvalue lies within r of theta; r may be tol and the rounding of the check."""
import ctypes

import numpy as np
import pytest

from cipsi_gb300 import engine

pytestmark = pytest.mark.gpu
TOL = 1e-8


@pytest.mark.parametrize("n,roots", [(1, 1), (2, 2), (5, 1), (255, 8), (257, 3), (1025, 2), (1793, 8), (160001, 2)])
def test_lowest_pairs(engine_lib, n, roots):
    rng = np.random.default_rng(n)
    d = 2.0 + 8.0 * np.sort(rng.random(n))
    d[:roots + 2] = 0.1 * np.arange(min(n, roots + 2))
    # rows couple to the next one and to one a third of the matrix away
    i, j, v = [np.arange(n)], [np.arange(n)], [0.5 * d]
    for step in {1, n // 3} - {0}:
        if step < n:
            i.append(np.arange(step, n))
            j.append(np.arange(n - step))
            v.append(0.05 * rng.standard_normal(n - step))
    i, j, v = np.concatenate(i), np.concatenate(j), np.concatenate(v)
    order = np.lexsort((j, i))
    i, j, v = i[order], j[order], np.ascontiguousarray(v[order])
    lib = engine._lib()
    P = ctypes.c_void_p
    lib.cipsi_davidson.argtypes = [ctypes.c_int32, ctypes.c_int64, P, P, P, ctypes.c_int32, ctypes.c_double,
                                   ctypes.c_int32, ctypes.c_int32, P, P, P, P, ctypes.c_char_p, ctypes.c_int32]
    ii, jj = (i + 1).astype(np.int32), (j + 1).astype(np.int32)
    w, x, it, res = np.zeros(roots), np.zeros((roots, n)), np.zeros(1, np.int32), np.zeros(roots)
    err = ctypes.create_string_buffer(256)
    rc = lib.cipsi_davidson(n, len(v), ii.ctypes.data, jj.ctypes.data, v.ctypes.data, roots, TOL, 200, 0,
                            w.ctypes.data, x.ctypes.data, it.ctypes.data, res.ctypes.data, err, 256)
    assert rc == 0, err.value
    round_ = 64 * 2.0 ** -53 * 12.0 * np.sqrt(n)  # |H| < 12; sums of 7 terms a row, of n rows in the norm
    for r in range(roots):
        y = np.zeros(n)
        np.add.at(y, i, v * x[r][j])
        np.add.at(y, j, v * x[r][i])  # the diagonal is stored as half its value
        assert np.linalg.norm(y - w[r] * x[r]) <= TOL + round_
    assert np.abs(x @ x.T - np.eye(roots)).max() <= 1e-10
    if n <= 2000:
        H = np.zeros((n, n))
        np.add.at(H, (i, j), v)
        np.add.at(H, (j, i), v)
        assert np.abs(np.linalg.eigvalsh(H)[:roots] - w).max() <= TOL + round_ * n ** 0.5
