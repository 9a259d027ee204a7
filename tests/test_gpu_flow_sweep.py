"""The dataflow sweep kernel against the ordered oracle, bit for bit, at the edges of
its layout: slabs from one (the whole sweep) to more than there are SMs (a CTA takes
several), tasks and levels that do not fill, rows of one and of several chunks, the
smallest systems; and repeated sweeps on the same buffers (its exchange entries are
told apart by epoch)."""
from __future__ import annotations

import os

import numpy as np
import pytest

import prispack_b200 as P
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture
def env():
    old = dict(os.environ)
    yield os.environ
    for k in ("PRISM_FLOW_ROWS", "PRISM_SWEEP_KERNEL", "PRISM_STREAM_PAIR"):
        os.environ.pop(k, None)
        if k in old:
            os.environ[k] = old[k]


def check(S, single):
    import torch
    S.set_stream(torch.cuda.current_stream().cuda_stream)
    rng = np.random.default_rng(3)
    for sw in (0, 1):
        o = S.sweep_order(sw)
        for rep in range(3):
            v = rng.standard_normal(S.n)
            tin = torch.tensor(v, device="cuda")
            tout = torch.empty_like(tin)
            S.sweep_device(sw, tin, tout, 1)
            torch.cuda.synchronize()
            ref = orc.sweep_ordered(o, v, diag=o.diag, op=o.op, lower=o.lower, single=single)
            assert np.array_equal(tout.cpu().numpy().view(np.uint64), ref.view(np.uint64)), (sw, rep)


@pytest.mark.parametrize("grid,rows", [((1, 1, 1), 32), ((3, 2, 1), 32), ((8, 1, 1), 32), ((33, 31, 1), 32),
                                       ((64, 64, 1), 4096), ((80, 80, 1), 33), ((17, 16, 15), 64),
                                       ((24, 20, 18), 700)])
@pytest.mark.parametrize("precision", [P.PRISM_FP64, P.PRISM_FP32, P.PRISM_FP32_APPLY])
@pytest.mark.parametrize("pair", ["0", "2"])
def test_slab_sizes(env, grid, rows, precision, pair):
    env.update(PRISM_FLOW_ROWS=str(rows), PRISM_SWEEP_KERNEL="stream", PRISM_STREAM_PAIR=pair)
    S = P.DeviceSystem(P.CSRMatrix.laplacian(*grid))
    S.set_precond(P.PRECOND_IC, tol=1e-3, precision=precision)
    check(S, precision == P.PRISM_FP32_APPLY)


@pytest.mark.parametrize("kind", [P.PRECOND_ILUT, P.PRECOND_ILDLT])
def test_random_patterns(env, kind):
    """A random symmetric, diagonally dominant matrix: halos over all upstream slabs, rows of
    several chunks (ILUT with 60 entries a row)."""
    env.update(PRISM_FLOW_ROWS="100", PRISM_SWEEP_KERNEL="stream", PRISM_STREAM_PAIR="0")
    import scipy.sparse as sp
    rng = np.random.default_rng(11)
    n = 1500
    R = sp.random(n, n, density=4.0 / n, random_state=7, data_rvs=lambda k: rng.uniform(-1.0, 0.0, k))
    A = (R + R.T).tocsr()
    A = (A + sp.diags(np.asarray(abs(A).sum(axis=1)).ravel() + 1.0)).tocsr()
    A.sort_indices()
    S = P.DeviceSystem(P.CSRMatrix(A.indptr, A.indices, A.data))
    S.set_precond(kind, tol=1e-6, lfill=60)
    check(S, False)


@pytest.mark.parametrize("grid,ks,precision", [
    ((1, 1, 1), (1, 64), P.PRISM_FP64), ((9, 1, 1), (2, 25), P.PRISM_FP64),        # smaller than a task, a chain
    ((40, 33, 1), (1, 2, 3, 24, 25, 63, 64), P.PRISM_FP32),                        # both sides of each width's limits
    ((14, 13, 12), (1, 13, 27, 64), P.PRISM_FP64),                                 # rows of several chunks
    ((364, 361, 1), (25, 63), P.PRISM_FP32)])                                      # four columns a lane
@pytest.mark.parametrize("kind", [P.PRECOND_IC, P.PRECOND_ILDLT])
def test_block_columns(grid, ks, precision, kind):
    """Each column of a block against the single-vector apply: the same factor values in double
    arithmetic, summed in another order (rows of up to 30 entries, all within 1e-12)."""
    import torch
    A = P.CSRMatrix.laplacian(*grid)
    S = P.DeviceSystem(A)
    S.set_stream(torch.cuda.current_stream().cuda_stream)
    S.set_precond(kind, tol=1e-3, precision=precision)
    for k in ks:
        g = torch.Generator(device="cuda").manual_seed(k)
        V = torch.randn(k, A.n, generator=g, device="cuda", dtype=torch.float64)
        for _ in range(2):
            out = S.apply_batched(V)
        for c in {0, k // 2, k - 1}:
            one = S.apply(V[c].contiguous())
            assert float((out[c] - one).abs().max()) <= 1e-12 * float(one.abs().max()), (k, c)
