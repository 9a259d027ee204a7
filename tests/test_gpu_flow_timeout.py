"""The dataflow sweep's give-up path: a value that is never published makes the bounded wait run
out; the kernel returns with PRISM_ERR_TIMEOUT's status, all its CTAs with it, and the next sweep
on the same buffers equals the layout's host replay to the last bit."""
from __future__ import annotations

import time

import numpy as np
import pytest

import prispack_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [0, 1, 2, 4])
def test_a_wait_that_runs_out(cols):
    for wait_ns in (1_000_000, 50_000_000):
        t = time.perf_counter()
        assert P.selftest_flow_timeout(0, cols, wait_ns) == 6
        # four slabs, each giving up at most one wait after the one before it, and the second sweep
        assert time.perf_counter() - t <= 4 * wait_ns * 1e-9 + 10.0
    # other handles go on working
    A = P.CSRMatrix.laplacian(30, 30, 1)
    S = P.DeviceSystem(A)
    S.set_precond(P.PRECOND_IC, tol=1e-3)
    x, st = S.solve(np.ones(A.n), tol=1e-10)
    assert st.converged and st.true_rel_residual <= 1e-9


def test_bad_arguments():
    for cols, wait_ns in ((3, 1000), (0, 3_000_000_000)):
        with pytest.raises(P.PrismError) as e:
            P.selftest_flow_timeout(0, cols, wait_ns)
        assert e.value.status == 1
