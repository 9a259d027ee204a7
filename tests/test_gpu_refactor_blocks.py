"""Block applies between refactorisations: the copies of the sweeps for blocks follow the new
values, whether they were uploaded before the first refactorisation or after it, for each number
of columns a CTA takes, and they are kept (a refactorisation with a block apply costs about as
much as the two alone, not a layout on the host)."""
from __future__ import annotations

import time

import numpy as np
import pytest

import prispack_b200 as P
from test_gpu_refactor import new_values

pytestmark = pytest.mark.gpu


def blocks_match(S, ks, seed):
    for k in ks:
        V = np.random.default_rng(seed + k).standard_normal((k, S.n))
        out = S.apply_batched(V)
        for c in {0, k // 2, k - 1}:
            # the same factor values in double arithmetic, summed in another order (rows of up to 40
            # entries, all within 1e-12)
            one = S.apply(V[c])
            assert np.abs(out[c] - one).max() <= 1e-12 * np.abs(one).max(), (k, c)


@pytest.mark.parametrize("kind", [P.PRECOND_IC, P.PRECOND_ILDLT])
@pytest.mark.parametrize("precision", [P.PRISM_FP64, P.PRISM_FP32])
def test_copies_follow_every_refactorisation(kind, precision):
    A = P.CSRMatrix.laplacian(24, 20, 3)
    S = P.DeviceSystem(A)
    S.set_precond(kind, tol=1e-3, precision=precision)
    blocks_match(S, (5,), 1)                 # uploaded before the first
    for step in range(3):
        S.update_values(new_values(A, seed=20 + step))
        S.refactor()
        if step > 0:
            blocks_match(S, (5, 40), 2 + step)   # 40: uploaded after a refactorisation


def test_copies_are_kept():
    import torch
    A = P.CSRMatrix.laplacian(40, 40, 40)
    S = P.DeviceSystem(A)
    S.set_precond(P.PRECOND_IC, tol=1e-3)
    V = torch.randn(8, A.n, device="cuda", dtype=torch.float64)

    def best(*calls):
        t = []
        for _ in range(5):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            for c in calls:
                c()
            torch.cuda.synchronize()
            t.append(time.perf_counter() - t0)
        return min(t)

    refactor, apply = S.refactor, lambda: S.apply_batched(V)
    apply(), refactor(), apply()
    # the two alone take about 4 ms here and the layout of both sweeps about 100 ms
    assert best(refactor, apply) <= 4 * (best(refactor) + best(apply))


@pytest.mark.parametrize("kind,precision", [(P.PRECOND_IC, P.PRISM_FP64), (P.PRECOND_ILDLT, P.PRISM_FP32)])
def test_a_failed_refactorisation_leaves_the_factor(kind, precision):
    """The vector sweeps, the factor as it is read back and copies for blocks uploaded afterwards
    all hold the last factor that was completed."""
    A = P.CSRMatrix.laplacian(24, 20, 3)
    S = P.DeviceSystem(A)
    S.set_precond(kind, tol=1e-3, precision=precision)
    S.update_values(new_values(A, seed=30))
    S.refactor()
    v = np.random.default_rng(1).standard_normal(A.n)
    before, factor = S.apply(v), S.precond_factor(0)
    rows = np.repeat(np.arange(A.n), np.diff(A.rowptr))
    bad = A.val.copy()
    # a pivot with no square root after most columns are done, or nothing to divide the first by
    at, value = (A.n - 40, -1.0) if kind == P.PRECOND_IC else (0, 0.0)
    bad[(rows == at) & (A.col == at)] = value
    S.update_values(bad)
    with pytest.raises(P.PrismError) as e:
        S.refactor()
    assert e.value.status == (4 if kind == P.PRECOND_IC else 3)
    assert np.array_equal(S.apply(v), before)
    for got, want in zip(S.precond_factor(0), factor):
        if want is not None:
            assert np.array_equal(got, want)
    blocks_match(S, (3, 30), 7)
