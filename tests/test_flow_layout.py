"""Dataflow layout of the triangular sweep kernel (k_sweep_flow) replayed on the
host (prism_selftest_flow_layout: indices, readiness, named-barrier counts, every
row once) against plain substitution: random patterns with far dependencies and
long rows, slabs from one to one a row, empty rows, wide single levels."""
from __future__ import annotations

import numpy as np
import pytest

import prispack_b200 as P
from test_stream_layout import random_triangular, substitute

# a row sums at most 80 products of size <= 0.3 |x|: in double 80 eps per level of the recursion
# stays far below 1e-12; in float 1e-4 as for the other float sweeps
TOL = {P.PRISM_FP64: 1e-12, P.PRISM_FP32: 1e-12, P.PRISM_FP32_APPLY: 1e-4}


@pytest.mark.parametrize("precision", [P.PRISM_FP64, P.PRISM_FP32, P.PRISM_FP32_APPLY])
@pytest.mark.parametrize("lower", [True, False])
@pytest.mark.parametrize("op", [0, 1, 2, 3])
def test_replay_matches_substitution(precision, lower, op):
    rng = np.random.default_rng(300 + op + 10 * lower)
    n = 901
    rp, ci, v = random_triangular(n, lower, rng, long_rows=(37, 400, 850))
    if precision != P.PRISM_FP64:
        v = v.astype(np.float32).astype(np.float64)
    d = rng.uniform(1.0, 2.0, n)
    b = rng.standard_normal(n)
    want = substitute(rp, ci, v, d, op, lower, b)
    for slabs in (1, 2, 13, 300, n):
        got = P.selftest_flow_layout(rp, ci, v, b, diag=d, op=op, lower=lower, precision=precision, num_slabs=slabs)
        assert np.abs(got - want).max() <= TOL[precision] * np.abs(want).max(), slabs


@pytest.mark.parametrize("n", [1, 8, 9, 96, 97, 1000])
def test_wide_levels_and_chains(n):
    """A diagonal sweep (one level of n rows), a chain (n levels of one row) and n rows that
    all read row 0: the edges of tasks and of barrier counts."""
    b = np.random.default_rng(n).standard_normal(n)
    got = P.selftest_flow_layout(np.zeros(n + 1, np.uint32), np.zeros(1, np.uint32), np.zeros(1), b, num_slabs=1)
    assert np.array_equal(got, b)
    rp = np.maximum(np.arange(-1, n), 0).astype(np.uint32)
    for ci in (np.arange(n - 1), np.zeros(n - 1)):
        ci = np.concatenate([ci, [0]]).astype(np.uint32)  # at least one entry for the binding
        v = np.full(n, 0.5)
        want = substitute(rp, ci, v, None, 2, True, b)
        for slabs in (1, 3):
            got = P.selftest_flow_layout(rp, ci, v, b, num_slabs=slabs)
            assert np.abs(got - want).max() <= 1e-14 * np.abs(want).max()


def test_slabs_that_need_more_slots_are_refused():
    rng = np.random.default_rng(5)
    rp, ci, v = random_triangular(200, True, rng)
    with pytest.raises(P.PrismError) as e:
        P.selftest_flow_layout(rp, ci, v, np.ones(200), num_slabs=1, max_slots=100)
    assert e.value.status == 9
