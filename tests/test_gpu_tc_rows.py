"""Per-row triangle counts whatever the hubs' indices. Whole numbers: equal to
the oracle's.
"""
import numpy as np
import pytest

import graphalgo_gb300 as ga
import oracle
from graphs import to_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flip", [False, True])
def test_tc_rows_whatever_the_hubs_indices(ctx, flip):
    """Hubs at the lowest or at the highest indices: a triangle's largest index
    is mostly the low-degree vertex's, or mostly the hub's."""
    m, rst, col = ga.gen_rmat(11, 8, seed=4)
    row = np.repeat(np.arange(m), np.diff(rst))
    if flip:
        row, col = m - 1 - row, m - 1 - col
        order = np.lexsort((col, row))
        row, col = row[order], col[order]
        rst = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=m))]).astype(np.int32)
    G = oracle.Csr(m, m, rst, col.astype(np.int32), np.ones(len(col), np.int32))
    total, rows = ga.tc("tri", to_device(ctx, G))
    ref_total, ref_rows = oracle.tc_sandia(G)
    assert total == ref_total and np.array_equal(rows, ref_rows)


@pytest.mark.parametrize("algo", ["msa", "mca", "heap"])
@pytest.mark.parametrize("n", [1, 2, 33, 300])
def test_tc_straight_from_a(ctx, algo, n):
    """The masked product of the lower parts without extracting them: a pattern
    that is not symmetric, diagonal entries, rows without a lower part, values
    that are not ones."""
    from graphs import dense_to_csr
    rng = np.random.default_rng(n)
    D = rng.random((n, n)) < 0.3
    D[n // 2] = np.arange(n) > n // 2
    for dtype in (np.int32, np.float64, np.uint8):
        G = dense_to_csr(D, rng.integers(1, 5, (n, n)), dtype)
        ref_total, ref_rows = oracle.tc_sandia(oracle.Csr(n, n, G.rst, G.col, np.ones(len(G.col), np.int32)))
        total, rows = ga.tc(algo, to_device(ctx, G))
        assert total == ref_total and np.array_equal(rows, ref_rows)
        assert ga.tc(algo, to_device(ctx, G), per_row=False)[0] == ref_total
