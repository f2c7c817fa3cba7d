"""Betweenness centrality at the edges of its column blocks (64 sources), of
the pieces of heavy vertices (1,024 neighbours) and of its depth, against the
FP64 oracle. Bound: 1e-9 relative, as everywhere for BC.
"""
import numpy as np
import pytest

import graphalgo_gb300 as ga
import oracle
from graphs import to_device

pytestmark = pytest.mark.gpu


def _csr(n, pairs, values=None):
    key = np.unique(pairs[:, 0].astype(np.int64) * n + pairs[:, 1])
    row, col = key // n, key % n
    keep = row != col
    row, col = row[keep], col[keep]
    rst = np.zeros(n + 1, np.int32)
    rst[1:] = np.cumsum(np.bincount(row, minlength=n))
    val = np.ones(len(col), np.int32) if values is None else values(len(col))
    return oracle.Csr(n, n, rst, col.astype(np.int32), val)


def _hubs(n, degrees, extra, rng, symmetric=True):
    """Random edges and one hub per degree (vertices 0, 1, ...)."""
    parts = [rng.integers(0, n, (extra, 2))]
    for h, d in enumerate(degrees):
        to = rng.choice(np.arange(len(degrees), n), d, replace=False)
        parts.append(np.stack([np.full(d, h), to], 1))
        if not symmetric:
            into = rng.choice(np.arange(len(degrees), n), d, replace=False)
            parts.append(np.stack([into, np.full(d, h)], 1))
    p = np.concatenate(parts)
    return np.concatenate([p, p[:, ::-1]]) if symmetric else p


def _close(got, ref):
    assert np.all(np.abs(got - ref) <= 1e-9 * np.maximum(np.abs(ref), 1.0))


@pytest.mark.parametrize("ns", [1, 31, 32, 33, 63, 64, 65, 128, 129, 300])
@pytest.mark.parametrize("loops", [0, 1])
def test_bc_column_blocks(ctx, ns, loops):
    rng = np.random.default_rng(ns)
    n = 3500
    G = _csr(n, _hubs(n, [1000, 1025, 2048, 2049, 3400], 3000, rng))
    src = rng.choice(n, ns, replace=False).astype(np.int32)
    ctx.set_option(ga.OPT_DEVICE_LOOPS, loops)
    try:
        _close(ga.bc(to_device(ctx, G), src), oracle.bc_batch(G, src))
    finally:
        ctx.set_option(ga.OPT_DEVICE_LOOPS, 1)


@pytest.mark.parametrize("ns", [7, 70])
def test_bc_directed_weighted_hubs(ctx, ns):
    rng = np.random.default_rng(5)
    n = 3000
    G = _csr(n, _hubs(n, [1030, 2900], 9000, rng, symmetric=False), lambda k: rng.integers(1, 4, k).astype(np.int32))  # the oracle's weights are int32
    src = rng.choice(n, ns, replace=False).astype(np.int32)
    _close(ga.bc(to_device(ctx, G), src), oracle.bc_batch(G, src))


@pytest.mark.parametrize("n", [2, 3, 4, 5, 400])
def test_bc_path(ctx, n):
    """One level per vertex: the level lists' ends, distances 0 and 1."""
    i = np.arange(n - 1)
    G = _csr(n, np.concatenate([np.stack([i, i + 1], 1), np.stack([i + 1, i], 1)]))
    src = np.unique([0, n // 2, n - 1]).astype(np.int32)
    _close(ga.bc(to_device(ctx, G), src), oracle.bc_batch(G, src))


def test_bc_batch_of_uneven_source_counts(ctx):
    """Graphs with 0, 1, 64 and 65 sources share the columns of one union."""
    rng = np.random.default_rng(9)
    graphs = [_csr(n, _hubs(n, [min(n - 2, 1100)], 2 * n, rng)) for n in (40, 90, 1300, 200)]
    parts = [to_device(ctx, G) for G in graphs]
    U, voff = ga.block_diag(ctx, parts)
    src = [rng.choice(G.m, k, replace=False).astype(np.int32) for G, k in zip(graphs, (0, 1, 64, 65))]
    got = ga.batch_bc(U, voff, src)
    for g, G in enumerate(graphs):
        ref = oracle.bc_batch(G, src[g]) if len(src[g]) else np.zeros(G.m)
        _close(got[voff[g]:voff[g + 1]], ref)


def test_bc_reuse_after_refusal(ctx):
    """A refused call (checked on the device) leaves the context usable."""
    rng = np.random.default_rng(3)
    G = _csr(300, _hubs(300, [250], 500, rng))
    A = to_device(ctx, G)
    ok = np.arange(5, dtype=np.int32)
    for bad in ([3, 3], [-1], [300]):
        with pytest.raises(ga.GaError):
            ga.bc(A, bad)
        _close(ga.bc(A, ok), oracle.bc_batch(G, ok))
    loop = oracle.Csr(2, 2, np.array([0, 1, 2], np.int32), np.array([0, 1], np.int32), np.ones(2, np.int32))
    with pytest.raises(ga.GaError):
        ga.bc(to_device(ctx, loop), [0])
