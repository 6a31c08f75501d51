"""CGLS on matrices whose columns (rows of A') have every kind of length the product A's
tells apart: empty, within and across a warp's 32 lanes and a block's 256 threads, just under
and over the long-row limit, with fewer rows than blocks and with several passes of all blocks.

A = [D; G]: a diagonal under random entries keeps the system well conditioned, so a few
iterations in FP64 agree to FP32 rounding of the solution (6e-8) plus the reordering of sums
of up to 5,000 terms; 2e-6 of the largest entry covers both.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths", [[0, 1, 31, 32, 33, 64], [255, 256, 257, 1, 0, 2, 3], [5000, 3, 2, 2049, 0, 1, 4, 8],
                                     [600] * 3 + [1] * 5000, [2] * 9600 + [300, 4000, 257]],
                         ids=["lanes", "block", "long", "two_passes", "three_passes"])
def test_rows_of_every_length(tomo, oracle_mod, lengths):
    rng = np.random.default_rng(len(lengths))
    M, N = len(lengths), 6000
    j = np.repeat(np.arange(M), lengths).astype(np.int32)
    i = np.concatenate([rng.choice(N, n, replace=False) for n in lengths] or [[]]).astype(np.int32)
    v = rng.uniform(0.1, 1.0, len(j)).astype(np.float32) / np.sqrt(np.maximum(np.repeat(lengths, lengths), 1))
    i = np.concatenate([i, N + np.arange(M)]).astype(np.int32)
    j = np.concatenate([j, np.arange(M)]).astype(np.int32)
    v = np.concatenate([v, np.full(M, 1.5, np.float32)]).astype(np.float32)
    o = np.lexsort((j, i))
    i, j, v = i[o], j[o], v[o]
    B = rng.standard_normal(N + M).astype(np.float32)
    x64, _ = oracle_mod.cgls_f64(N + M, M, i, j, v, B, 6)
    x = tomo.sparse_cgls_gpu(i, j, v, B, N + M, M, 6)
    assert np.max(np.abs(x - x64)) <= 2e-6 * np.max(np.abs(x64))
