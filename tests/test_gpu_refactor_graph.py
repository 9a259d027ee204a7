"""FGMRES before and after a refactorisation that replaces the preconditioner's device arrays
(paired sweeps are tuned again unpaired, once): the second solve captures its cycle graph anew.

The graph and plain launches run the same kernels on the same grids, so the two agree to the
last bit; an unchanged preconditioner keeps its graph."""
from __future__ import annotations

import numpy as np
import pytest

import prispack_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,precision", [(P.PRECOND_IC, P.PRISM_FP64), (P.PRECOND_ILDLT, P.PRISM_FP32_APPLY)])
def test_fgmres_after_refactor_of_paired_sweeps(monkeypatch, kind, precision):
    monkeypatch.setenv("PRISM_SWEEP_KERNEL", "stream")
    monkeypatch.setenv("PRISM_STREAM_PAIR", "2")
    A = P.CSRMatrix.laplacian(14, 12, 10)
    S = P.DeviceSystem(A)
    S.set_precond(kind, tol=1e-3, precision=precision)
    assert S.sweep_order(0).paired
    b = np.random.default_rng(3).standard_normal(A.n)

    def solve(**kw):
        return S.solve(b, solver=P.SOLVER_FGMRES, tol=1e-10, restart=20, **kw)

    x0, st0 = solve()
    assert st0.graph_nodes > 0 and st0.converged
    S.refactor()
    assert not S.sweep_order(0).paired
    for scale in (1.0, 1.5):  # the second round keeps the arrays and the graph, with new values in them
        S.update_values(scale * A.val)
        S.refactor()
        xg, sg = solve()
        xs, ss = solve(launch_mode=P.LAUNCH_STREAM)
        assert sg.graph_nodes > 0 and sg.converged
        assert np.array_equal(xg, xs) and sg.num_iter == ss.num_iter
        # both solutions have a relative residual below 1e-8 and ||A^-1|| ||A|| < 200 here
        assert np.linalg.norm(scale * xg - x0) <= 1e-5 * np.linalg.norm(x0)
