"""Device refactorisation of factors with long columns: more than 32 updates and more than
512 products a column, which k_refactor takes in several chunks, and the smallest columns.

The device factor equals the oracle's fixed-pattern refactorisation to the last bit (the
operations and their order are the same, so there is no tolerance).
"""
from __future__ import annotations

import numpy as np
import pytest

import prispack_b200 as P
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def dense(n, seed):
    """A full symmetric positive definite matrix, rows in order, and a second one."""
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(2):
        M = rng.uniform(-1.0, 1.0, (n, n))
        M = 0.5 * (M + M.T)
        M[np.arange(n), np.arange(n)] = n + 1.0
        out.append(M.ravel())
    rowptr = np.arange(n + 1, dtype=np.uint32) * n
    col = np.tile(np.arange(n, dtype=np.uint32), n)
    return P.CSRMatrix(rowptr, col, out[0]), out[1]


@pytest.mark.parametrize("kind", [P.PRECOND_IC, P.PRECOND_ILDLT])
@pytest.mark.parametrize("precision", [P.PRISM_FP64, P.PRISM_FP32])
@pytest.mark.parametrize("n", [1, 2, 32, 33, 34, 70, 300])
def test_long_columns(n, precision, kind):
    A, val2 = dense(n, 100 + n)
    S = P.DeviceSystem(A)
    S.set_precond(kind, tol=1e-14, precision=precision)
    rp, ci, _, _ = S.precond_factor(0)
    S.update_values(val2)
    for _ in range(2):  # the second one finds the places laid out
        S.refactor()
        rc, lv, D = orc.refactor(kind, A.rowptr, A.col, val2, rp, ci, single=precision != P.PRISM_FP64)
        assert rc == 0
        _, _, dv, dd = S.precond_factor(0)
        assert np.array_equal(dv, lv)
        if kind == P.PRECOND_ILDLT:
            assert np.array_equal(dd, D)
