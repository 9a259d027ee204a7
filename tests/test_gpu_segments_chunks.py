"""Batches of systems whose reductions run over several chunks of 4,096 rows, and of more chunks
than blocks: the partial sums, the per-system tickets (left at zero for the next kernel and the
next solve) and a block's way from chunk to chunk.  Each system against its own solve, repeated
solves bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import prispack_b200 as P

pytestmark = pytest.mark.gpu

EDGES = [(63, 65), (64, 64), (17, 241), (142, 141), (128, 96)]  # 4,095 4,096 4,097 20,022 12,288 rows
MANY = [(5, 4)] * 350 + [(110, 90)] + [(3, 3)] * 350 + [(97, 89)]  # 703 chunks, 592 blocks


def solve_all(grids, seed, check):
    import torch
    parts = [P.CSRMatrix.laplacian(*g, 1) for g in grids]
    A, seg = P.CSRMatrix.block_diagonal(parts)
    S = P.DeviceSystem(A)
    S.set_stream(torch.cuda.current_stream().cuda_stream)
    S.set_precond(P.PRECOND_IC, tol=1e-3)
    b = np.random.default_rng(seed).standard_normal(A.n)
    bd = torch.tensor(b, device="cuda")
    runs = [S.solve_segments(seg, bd, tol=1e-10, max_iter=2000) for _ in range(3)]
    x, stats = runs[0]
    for other, st in runs[1:]:
        assert torch.equal(other, x)
        assert [(s.num_iter, s.final_error) for s in st] == [(s.num_iter, s.final_error) for s in stats]
    assert all(s.converged and s.true_rel_residual < 1.5e-10 for s in stats)
    x = x.cpu().numpy()
    for s in check:
        lo, hi = seg[s], seg[s + 1]
        one = P.DeviceSystem(parts[s])
        one.set_precond(P.PRECOND_IC, tol=1e-3)
        xs, st = one.solve(b[lo:hi], tol=1e-10, max_iter=2000)
        assert abs(stats[s].num_iter - st.num_iter) <= 1, s
        if stats[s].num_iter == st.num_iter:
            # as for small systems: solutions within 1e-10 at equal iteration counts
            assert np.abs(x[lo:hi] - xs).max() <= 1e-10 * np.abs(xs).max(), s


@pytest.mark.parametrize("seed", [3, 4])
def test_systems_around_a_chunk(seed):
    solve_all(EDGES, seed, range(len(EDGES)))


def test_more_chunks_than_blocks():
    solve_all(MANY, 5, [0, 349, 350, 351, 700, 701])


@pytest.mark.parametrize("grid,count", [((1, 1), 50), ((8, 8), 60), ((13, 5), 60), ((16, 16), 40), ((19, 14), 40),
                                        ((32, 32), 12), ((41, 25), 12)])
def test_sizes_of_blocks(grid, count):
    """Systems of 1, 64, 65, 256, 266, 1,024 and 1,025 rows: each side of the sizes at which the
    kernels take larger blocks."""
    solve_all([grid] * count, 6, [0, count // 2, count - 1])
