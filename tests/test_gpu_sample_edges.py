"""Small masked products whose A has as many entries as the sample that their
limit is estimated from (256), one fewer and one more, and few or none. Whole
numbers: equal to the oracle's.
"""
import numpy as np
import pytest

import graphalgo_gb300 as ga
import oracle
from graphs import to_device

pytestmark = pytest.mark.gpu


def _rows(lengths, n, rng):
    rst = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    col = np.concatenate([np.sort(rng.choice(n, d, replace=False)) for d in lengths]).astype(np.int32)
    return oracle.Csr(len(lengths), n, rst, col, rng.integers(-3, 4, len(col)).astype(np.int32))


@pytest.mark.parametrize("entries", [0, 1, 2, 255, 256, 257, 511, 512, 513])
@pytest.mark.parametrize("rows", [1, 5, 300])
@pytest.mark.parametrize("algo", ["msa", "mca", "heap", "hybrid"])
def test_entries(ctx, entries, rows, algo):
    rng = np.random.default_rng(entries)
    lengths = np.bincount(rng.integers(0, rows, entries), minlength=rows)
    A, M = _rows(lengths, 1000, rng), _rows(rng.integers(0, 300, rows), 3000, rng)
    B = _rows(np.where(np.arange(1000) % 30 == 0, 700, 9), 3000, rng)
    v = ga.mxm_masked(algo, to_device(ctx, A), to_device(ctx, B), to_device(ctx, M)).download()[2]
    assert np.array_equal(v, oracle.mxm_masked(A, B, M))
