"""Block sweeps on patterns where level order is faster than the dataflow slabs: few, wide
wavefronts whose rows read far and wide (a random symmetric pattern), and rows too long for the
slabs (one full row and column).  Each column equals the vector apply, before and after a
refactorisation, and more columns do not cost what the slabs would take for them."""
from __future__ import annotations

import numpy as np
import pytest

import prispack_b200 as P
from test_gpu_refactor import new_values

pytestmark = pytest.mark.gpu


def csr(A):
    A = A.tocsr()
    A.sort_indices()
    return P.CSRMatrix(A.indptr, A.indices, A.data)


def random_pattern(n=20000, per_row=2):
    import scipy.sparse as sp
    rng = np.random.default_rng(7)
    i, j = rng.integers(0, n, n * per_row), rng.integers(0, n, n * per_row)
    R = sp.coo_matrix((-rng.uniform(0.1, 1.0, n * per_row), (i, j)), shape=(n, n))
    A = (R + R.T).tocsr()
    A.setdiag(0.0)
    A.eliminate_zeros()
    return csr(A + sp.diags(np.asarray(abs(A).sum(axis=1)).ravel() + 1.0))


def arrow(n):
    """Tridiagonal, with the last row and column full."""
    import scipy.sparse as sp
    A = sp.diags([np.full(n - 1, -1.0), np.r_[np.full(n - 1, 4.0), float(n)], np.full(n - 1, -1.0)], [-1, 0, 1])
    last, rest, v = np.full(n - 2, n - 1), np.arange(n - 2), np.full(n - 2, -0.05)
    return csr(A + sp.coo_matrix((v, (last, rest)), shape=(n, n)) + sp.coo_matrix((v, (rest, last)), shape=(n, n)))


def columns_match(S, ks):
    for k in ks:
        V = np.random.default_rng(k).standard_normal((k, S.n))
        for _ in range(2):  # the first one times the layouts
            out = S.apply_batched(V)
        for c in {0, k // 2, k - 1}:
            # the same factor values in double arithmetic, summed in another order; the longest row of
            # the factor has 5,000 entries of 0.01 to 0.3 of its diagonal: within 1e-12
            one = S.apply(V[c])
            assert np.abs(out[c] - one).max() <= 1e-12 * np.abs(one).max(), (k, c)


@pytest.mark.parametrize("kind,precision", [(P.PRECOND_IC, P.PRISM_FP64), (P.PRECOND_ILDLT, P.PRISM_FP32),
                                            (P.PRECOND_ILUT, P.PRISM_FP32)])
@pytest.mark.parametrize("matrix,tol", [(random_pattern, 1e-2), (lambda: arrow(5000), 1e-9)])
def test_columns(matrix, tol, kind, precision):
    A = matrix()
    S = P.DeviceSystem(A)
    S.set_precond(kind, tol=tol, precision=precision, lfill=20)
    columns_match(S, (1, 8, 24, 25, 64))
    if kind != P.PRECOND_ILUT:
        S.update_values(new_values(A))
        S.refactor()
        columns_match(S, (8, 48, 64))


@pytest.mark.parametrize("precision", [P.PRISM_FP64, P.PRISM_FP32])
@pytest.mark.parametrize("matrix", [random_pattern, lambda: P.CSRMatrix.block_diagonal(
    [P.CSRMatrix.laplacian(5, 5, 1)] * 3000)[0]])
def test_columns_of_a_multilevel_preconditioner(matrix, precision):
    """Levels of a few wide wavefronts; no low-rank terms, so every product is in double."""
    A = matrix()
    H = P.HostAmsed(A, precision=precision, levels=3, lanczos_steps=16, low_rank=8, lowrank_type=0, reorder=0)
    assert not H.info()["ranks"].any()
    S = P.DeviceSystem(A)
    S.attach(H)
    columns_match(S, (1, 8, 40, 64, 8))


def test_many_columns_of_a_random_pattern():
    import torch
    A = random_pattern()
    S = P.DeviceSystem(A)
    S.set_stream(torch.cuda.current_stream().cuda_stream)
    S.set_precond(P.PRECOND_IC, tol=1e-2)

    def best_ms(k):
        V = torch.randn(k, A.n, device="cuda", dtype=torch.float64)
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        t = []
        for _ in range(20):
            e[0].record()
            S.apply_batched(V)
            e[1].record()
            torch.cuda.synchronize()
            t.append(e[0].elapsed_time(e[1]))
        return min(t)

    # level order takes less for 64 columns than for 4; the slabs took 2.6 times as long
    assert best_ms(64) <= 1.7 * best_ms(4)
