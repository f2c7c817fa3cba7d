"""Vertex ranks of batched triangle listing. Whole numbers: equal to the
oracle's, whatever the ranks.
"""
import numpy as np
import pytest

import graphalgo_gb300 as ga
import oracle
from graphs import dense_to_csr, random_graph, to_device

pytestmark = pytest.mark.gpu


def _graphs(rng):
    full = np.ones((33, 33), bool)                      # degrees reach n (diagonal entries)
    loops = np.triu(rng.random((40, 40)) < 0.4)
    loops = loops | loops.T
    return [random_graph(1, 0.5, rng), random_graph(2, 1.1, rng), dense_to_csr(full), dense_to_csr(loops),
            random_graph(150, 0.2, rng), random_graph(64, 0.9, rng), random_graph(5, 0.0, rng)]


@pytest.mark.parametrize("k", [3, 5, 9])
@pytest.mark.parametrize("frontier", [0, 1])
def test_batch_ranks_by_graph(ctx, k, frontier):
    rng = np.random.default_rng(k)
    graphs = _graphs(rng)
    U, voff = ga.block_diag(ctx, [to_device(ctx, G) for G in graphs])
    ctx.set_option(ga.OPT_KT_FRONTIER, frontier)
    try:
        K, iters = ga.batch_ktruss("tri", U, voff, k)
    finally:
        ctx.set_option(ga.OPT_KT_FRONTIER, 1)
    rst, col, _ = K.download()
    for (m, r, c), G, it in zip(ga.split_blocks(rst, col, voff), graphs, iters):
        R, rit = oracle.ktruss(G, k)
        assert it == rit and np.array_equal(r, R.rst) and np.array_equal(c, R.col[:R.nnz])
