"""Betweenness centrality where vertices' neighbour lists are cut into pieces:
degrees around the multiples of 512, and of 2,048 in graphs of more than 256
entries per vertex, unit and weighted, symmetric and directed, one and several
blocks of 64 columns. Against the FP64 oracle, 1e-9 relative, as everywhere for BC.
"""
import numpy as np
import pytest

import graphalgo_gb300 as ga
import oracle
from graphs import to_device

pytestmark = pytest.mark.gpu


def _graph(n, degrees, per_vertex, symmetric, weighted, rng):
    """Random edges, and vertices 0, 1, ... with the given numbers of out-neighbours exactly (directed: in-neighbours
    of as many others)."""
    h = len(degrees)
    a, b = rng.integers(h, n, (2, n * per_vertex // 2))
    row, col = [a, b], [b, a]
    for v, d in enumerate(degrees):
        to = h + rng.choice(n - h, d, replace=False)
        row.append(np.full(d, v))
        col.append(to)
        if symmetric:
            row.append(to)
            col.append(np.full(d, v))
        else:
            into = h + rng.choice(n - h, d, replace=False)
            row.append(into)
            col.append(np.full(d, v))
    key = np.unique(np.concatenate(row).astype(np.int64) * n + np.concatenate(col))
    key = key[key // n != key % n]
    row, col = key // n, key % n
    rst = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))]).astype(np.int32)
    assert list(np.diff(rst)[:h]) == degrees
    val = (1 + (row + col) % 3 if weighted else np.ones(len(col))).astype(np.int32)
    return oracle.Csr(n, n, rst, col.astype(np.int32), val)


@pytest.mark.parametrize("ns", [1, 64, 65, 200])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("n,degrees,per_vertex", [
    (3000, [511, 512, 513, 1023, 1024, 1025, 2900], 4),
    (4600, [2047, 2048, 2049, 4096, 4097], 290),  # more than 256 entries per vertex
], ids=["512", "2048"])
def test_pieces(ctx, n, degrees, per_vertex, symmetric, weighted, ns):
    rng = np.random.default_rng(ns)
    G = _graph(n, degrees, per_vertex, symmetric, weighted, rng)
    assert (G.nnz > 256 * n) == (per_vertex > 256)
    src = rng.choice(n, ns, replace=False).astype(np.int32)
    got, ref = ga.bc(to_device(ctx, G), src), oracle.bc_batch(G, src)
    assert np.all(np.abs(got - ref) <= 1e-9 * np.maximum(np.abs(ref), 1.0))
