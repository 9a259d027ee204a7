"""Device refactorisation at the longest columns it takes: more than 512 entries (chunks of up to
1,024 products, placed beyond 512), the last accepted length, 1,024, and the first refused one.
The device factor equals the oracle's to the last bit."""
from __future__ import annotations

import numpy as np
import pytest

import prispack_b200 as P
from oracle import oracle as orc
from test_gpu_refactor_chunks import dense

pytestmark = pytest.mark.gpu


def tall(n, seed, wide=40):
    """The first `wide` rows and columns full, the rest diagonal: the factor keeps those columns
    whole and drops the fill below them (1e-5 against 1e-4 of a column of norm 1).  And second
    values."""
    import scipy.sparse as sp
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(2):
        M = rng.uniform(0.5e-3, 1e-3, (n, wide)) * rng.choice([-1.0, 1.0], (n, wide))
        top = np.tril(M[:wide], -1)
        top = top + top.T + np.eye(wide)
        A = sp.bmat([[sp.csr_matrix(top), sp.csr_matrix(M[wide:].T)], [sp.csr_matrix(M[wide:]), sp.identity(n - wide)]])
        A = A.tocsr()
        A.sort_indices()
        out.append(A)
    return P.CSRMatrix(out[0].indptr, out[0].indices, out[0].data), out[1].data


@pytest.mark.parametrize("n", [512, 513, 600, 1023, 1024])
@pytest.mark.parametrize("kind,precision", [(P.PRECOND_IC, P.PRISM_FP64), (P.PRECOND_IC, P.PRISM_FP32),
                                            (P.PRECOND_ILDLT, P.PRISM_FP64)])
def test_longest_columns(n, kind, precision):
    A, val2 = tall(n, 100 + n)
    S = P.DeviceSystem(A)
    S.set_precond(kind, tol=1e-4, precision=precision)
    rp, ci, _, _ = S.precond_factor(0)
    diag = 1 if kind == P.PRECOND_IC else 0  # entries of a column that are its diagonal
    assert np.diff(rp).max() == n - 1 + diag
    S.update_values(val2)
    for _ in range(2):
        S.refactor()
        rc, lv, D = orc.refactor(kind, A.rowptr, A.col, val2, rp, ci, single=precision != P.PRISM_FP64)
        assert rc == 0
        _, _, dv, dd = S.precond_factor(0)
        assert np.array_equal(dv, lv)
        if kind == P.PRECOND_ILDLT:
            assert np.array_equal(dd, D)


def test_full_factor_of_the_longest_columns():
    """1,024 columns that wait for one another's whole work: the refactorisation takes longer than
    a wait without progress may (1 s), and is not given up."""
    A, val2 = dense(1024, 5)
    S = P.DeviceSystem(A)
    S.set_precond(P.PRECOND_IC, tol=1e-14)
    rp, ci, _, _ = S.precond_factor(0)
    S.update_values(val2)
    S.refactor()
    rc, lv, _ = orc.refactor(P.PRECOND_IC, A.rowptr, A.col, val2, rp, ci, single=False)
    assert rc == 0 and np.array_equal(S.precond_factor(0)[2], lv)


@pytest.mark.parametrize("kind", [P.PRECOND_IC, P.PRECOND_ILDLT])
def test_longer_columns_are_refused(kind):
    A, _ = tall(1025, 7)
    S = P.DeviceSystem(A)
    S.set_precond(kind, tol=1e-4)
    v = np.random.default_rng(1).standard_normal(A.n)
    before = S.apply(v)
    with pytest.raises(P.PrismError) as e:
        S.refactor()
    assert e.value.status == 9  # PRISM_ERR_UNSUPPORTED
    assert np.array_equal(S.apply(v), before)
