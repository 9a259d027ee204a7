"""The streamed rounds inside a handle (PRISM_SWEEP_KERNEL=rounds): the tuner takes them only for
sweeps whose dataflow slabs do not fit, so every use of them is forced here: sweeps bit for bit
against the ordered oracle, refactorisation through their value maps, the multilevel apply, and
block-diagonal factors of more blocks than there are co-resident CTAs, which go to level order."""
from __future__ import annotations

import numpy as np
import pytest

import prispack_b200 as P
from oracle import oracle as orc
from test_gpu_refactor import new_values, oracle_precond

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def rounds(monkeypatch):
    monkeypatch.setenv("PRISM_SWEEP_KERNEL", "rounds")
    monkeypatch.setenv("PRISM_STREAM_PAIR", "0")


@pytest.mark.parametrize("pair", ["0", "2"])
@pytest.mark.parametrize("precision", [P.PRISM_FP64, P.PRISM_FP32, P.PRISM_FP32_APPLY])
@pytest.mark.parametrize("kind", [P.PRECOND_IC, P.PRECOND_ILDLT, P.PRECOND_ILUT])
def test_sweeps_bitwise(monkeypatch, kind, precision, pair):
    import torch
    monkeypatch.setenv("PRISM_STREAM_PAIR", pair)
    A = (P.CSRMatrix.convection_diffusion(19, 18, 17, 10.0, 5.0, 2.5) if kind == P.PRECOND_ILUT
         else P.CSRMatrix.laplacian(19, 18, 17))
    S = P.DeviceSystem(A)
    S.set_stream(torch.cuda.current_stream().cuda_stream)
    S.set_precond(kind, tol=1e-3, lfill=20, precision=precision)
    rng = np.random.default_rng(kind)
    for sw in (0, 1):
        assert S.sweep_info(sw)["kernel"] == "rounds"
        o = S.sweep_order(sw)
        assert o.paired == (pair == "2" and precision != P.PRISM_FP32)
        for _ in range(2):
            v = rng.standard_normal(A.n)
            tin = torch.tensor(v, device="cuda")
            tout = torch.empty_like(tin)
            S.sweep_device(sw, tin, tout, 1)
            torch.cuda.synchronize()
            ref = orc.sweep_ordered(o, v, diag=o.diag, op=o.op, lower=o.lower,
                                    single=precision == P.PRISM_FP32_APPLY)
            assert np.array_equal(tout.cpu().numpy().view(np.uint64), ref.view(np.uint64)), sw


@pytest.mark.parametrize("kind,precision", [(P.PRECOND_IC, P.PRISM_FP64), (P.PRECOND_IC, P.PRISM_FP32),
                                            (P.PRECOND_IC, P.PRISM_FP32_APPLY), (P.PRECOND_ILDLT, P.PRISM_FP64),
                                            (P.PRECOND_ILDLT, P.PRISM_FP32)])
def test_refactor(kind, precision):
    A = P.CSRMatrix.laplacian(14, 12, 10)
    S = P.DeviceSystem(A)
    S.set_precond(kind, tol=1e-3, precision=precision)
    assert S.sweep_info(0)["kernel"] == S.sweep_info(1)["kernel"] == "rounds"
    v = np.random.default_rng(1).standard_normal(A.n)
    before = S.apply(v)
    S.refactor()
    assert np.array_equal(S.apply(v), before)
    rp, ci, _, _ = S.precond_factor(0)
    val2 = new_values(A)
    S.update_values(val2)
    S.refactor()
    rc, lv, D = orc.refactor(kind, A.rowptr, A.col, val2, rp, ci, single=precision != P.PRISM_FP64)
    assert rc == 0
    ref = oracle_precond(kind, A.n, rp, ci, lv, D).apply(v.copy())
    got = S.apply(v)
    # as for the other layouts: double arithmetic 1e-12, the single-precision apply 1e-5 in the 2-norm
    if precision == P.PRISM_FP32_APPLY:
        assert np.linalg.norm(got - ref) <= 1e-5 * np.linalg.norm(ref)
    else:
        assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("precision", [P.PRISM_FP64, P.PRISM_FP32])
def test_amsed_apply(precision):
    A = P.CSRMatrix.laplacian(30, 28, 26)
    H = P.HostAmsed(A, levels=3, lanczos_steps=24, low_rank=8, lowrank_type=0, reorder=0, precision=precision)
    S = P.DeviceSystem(A)
    S.attach(H)
    assert "rounds" in {S.sweep_info(sw)["kernel"] for sw in range(6) if S.sweep_info(sw)["n"]}
    b = np.random.default_rng(9).standard_normal(A.n)
    ref = orc.Amsed(H).apply(b)
    assert np.abs(S.apply(b) - ref).max() <= 1e-12 * np.abs(ref).max()


def test_more_blocks_than_ctas():
    A, _ = P.CSRMatrix.block_diagonal([P.CSRMatrix.laplacian(9, 9, 1) for _ in range(2000)])
    S = P.DeviceSystem(A)
    S.set_precond(P.PRECOND_IC, tol=1e-3)
    assert S.sweep_info(0)["kernel"] == S.sweep_info(1)["kernel"] == "level-order"
    v = np.random.default_rng(2).standard_normal(A.n)
    rp, ci, val, _ = S.precond_factor(0)
    ref = orc.Precond(P.PRECOND_IC, A.n, (rp, ci, val)).apply(v.copy())
    assert np.abs(S.apply(v) - ref).max() <= 1e-12 * np.abs(ref).max()
