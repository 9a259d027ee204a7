"""The FP64 low-rank block product at the edges of its split: one block, one group of blocks, several
groups, four blocks an SM with ragged last tiles; repeated runs bit for bit (the order of the two
sums is fixed), and repeated on one preconditioner (its tickets return to zero)."""
from __future__ import annotations

import numpy as np
import pytest

import prispack_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrem", [1, 8, 9, 17, 33, 371, 1184, 1185, 9473, 40001])
@pytest.mark.parametrize("rank,k", [(1, 1), (5, 13), (33, 64), (128, 2)])
def test_product(nrem, rank, k):
    rng = np.random.default_rng(nrem + rank + k)
    W, H = rng.standard_normal((nrem, rank)), rng.uniform(0.5, 2.0, rank)
    X, Y = rng.standard_normal((nrem, k)), rng.standard_normal((nrem, k))
    out = P.lowrank_block_run(W, H, X, Y, tensor=False)
    assert np.array_equal(P.lowrank_block_run(W, H, X, Y, tensor=False), out)
    ref = Y + W @ (H[:, None] * (W.T @ X))
    # a blocked sum of nrem products and one of rank: well within 1e-13 of the sum of magnitudes
    assert np.abs(out - ref).max() <= 1e-13 * (np.abs(Y) + np.abs(W) @ (H[:, None] * (np.abs(W).T @ np.abs(X)))).max()


def test_repeated_applies():
    A = P.CSRMatrix.laplacian(96, 80, 1)
    S = P.DeviceSystem(A)
    S.set_amsed(precision=P.PRISM_FP64, levels=3, lanczos_steps=32, low_rank=16, lowrank_type=0, reorder=0)
    V = np.random.default_rng(1).standard_normal((13, A.n))
    first = S.apply_batched(V)
    for k in (13, 5, 13):
        assert np.array_equal(S.apply_batched(V[:k]), first[:k])
