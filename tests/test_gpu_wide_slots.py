"""Masked products with 8-byte accumulators at the edges of a warp row's and of
a window's mask slots, which are half as many as those of 4-byte ones. Whole
numbers: equal to the oracle's.
"""
import numpy as np
import pytest

import graphalgo_gb300 as ga
import oracle
from graphs import to_device

pytestmark = pytest.mark.gpu

MASKS = [0, 1, 127, 128, 129, 255, 256, 257, 2047, 2048, 2049, 4095, 4096, 4097, 6145]


def _rows(lengths, n, rng, dtype):
    rst = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    col = np.concatenate([np.sort(rng.choice(n, d, replace=False)) for d in lengths]).astype(np.int32)
    return oracle.Csr(len(lengths), n, rst, col, rng.integers(-3, 4, len(col)).astype(dtype))


@pytest.mark.parametrize("dtype", [np.float64, np.int64, np.float32])
@pytest.mark.parametrize("algo", ["msa", "mca", "heap", "hybrid"])
def test_slots(ctx, algo, dtype):
    rng = np.random.default_rng(4)
    k, n = 700, 9001
    M = _rows(MASKS * 2, n, rng, dtype)
    A = _rows([40] * len(MASKS) + [600] * len(MASKS), k, rng, dtype)
    B = _rows(rng.integers(0, 60, k - 2).tolist() + [300, 8000], n, rng, dtype)
    C = ga.mxm_masked(algo, to_device(ctx, A), to_device(ctx, B), to_device(ctx, M))
    rst, col, val = C.download()
    assert np.array_equal(rst, M.rst) and np.array_equal(col, M.col)
    assert np.array_equal(val, oracle.mxm_masked(A, B, M))
