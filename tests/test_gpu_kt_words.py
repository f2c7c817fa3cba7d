"""The k-truss state's flags, one bit per entry in words of 32: numbers of
entries next to multiples of 32, rows that start and end inside a word, empty
rows at either end, diagonal entries, and the loops with and without the
frontier. Whole numbers: equal to the oracle's.
"""
import numpy as np
import pytest

import graphalgo_gb300 as ga
import oracle
from graphs import dense_to_csr, to_device

pytestmark = pytest.mark.gpu


def _graph(nnz, rng):
    """A symmetric graph of exactly nnz entries, its first and last rows empty."""
    n = 8
    while (n - 5) * (n - 6) < nnz:
        n += 1
    D = np.zeros((n, n), bool)
    u, v = np.triu_indices(n - 5, 1)
    pick = rng.permutation(len(u))[:nnz // 2]
    D[u[pick] + 2, v[pick] + 2] = True
    D |= D.T
    if nnz % 2:
        D[n // 2, n // 2] = True
    return dense_to_csr(D)


@pytest.mark.parametrize("nnz", [0, 1, 2, 3, 30, 31, 32, 33, 62, 63, 64, 65, 96, 512, 1023, 1024, 1025, 65536 * 2])
def test_words(ctx, nnz):
    rng = np.random.default_rng(nnz)
    G = _graph(nnz, rng)
    assert len(G.col) == nnz
    A = to_device(ctx, G)
    for k in (2, 3, 4, 6):
        R, rit = oracle.ktruss(G, k)
        for frontier in (1, 0):
            ctx.set_option(ga.OPT_KT_FRONTIER, frontier)
            try:
                C, it = ga.ktruss("tri", A, k)
            finally:
                ctx.set_option(ga.OPT_KT_FRONTIER, 1)
            r, c, v = C.download()
            assert it == rit and np.array_equal(r, R.rst) and np.array_equal(c, R.col[:R.nnz]), (k, frontier)
            assert np.all(v == 1)


def test_words_batch(ctx):
    rng = np.random.default_rng(3)
    host = [_graph(nnz, rng) for nnz in (0, 33, 64, 1, 200, 2048, 31, 999)]
    U, voff = ga.block_diag(ctx, [to_device(ctx, G) for G in host])
    for k in (3, 5):
        C, iters = ga.batch_ktruss("tri", U, voff, k)
        cr, cc, cv = C.download()
        assert np.all(cv == 1)
        for G, it, (m, r, c) in zip(host, iters, ga.split_blocks(cr, cc, voff)):
            R, rit = oracle.ktruss(G, k)
            assert it == rit and np.array_equal(r, R.rst) and np.array_equal(c, R.col[:R.nnz])
