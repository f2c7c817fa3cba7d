"""The k-truss loop in one launch against the oracle and against the captured
loop's twin (host loops): edge sets, iteration counts and work counters, over
diagonal entries, rows cut into segments, frontiers of every size, and the
iteration bound. Whole numbers: equal.
"""
import numpy as np
import pytest

import graphalgo_gb300 as ga
import oracle
from graphs import dense_to_csr, random_graph, to_device

pytestmark = pytest.mark.gpu


def _with_loops(n, density, rng):
    D = np.triu(rng.random((n, n)) < density)
    return dense_to_csr(D | D.T)


def _clique_chain(sizes):
    """Cliques of growing size, each joined to the next by one edge."""
    n = sum(sizes)
    D = np.zeros((n, n), bool)
    at = 0
    for s in sizes:
        D[at:at + s, at:at + s] = True
        if at:
            D[at - 1, at] = D[at, at - 1] = True
        at += s
    np.fill_diagonal(D, False)
    return dense_to_csr(D)


def _ladder(n):
    """A strip of triangles that a 4-truss peels from both ends, two edges or so
    per iteration: many small frontiers."""
    D = np.zeros((n, n), bool)
    for i in range(n - 1):
        D[i, i + 1] = D[i + 1, i] = True
        if i + 2 < n:
            D[i, i + 2] = D[i + 2, i] = True
        if i + 3 < n and i % 3:
            D[i, i + 3] = D[i + 3, i] = True
    return dense_to_csr(D)


def _graphs():
    rng = np.random.default_rng(17)
    hubs = random_graph(900, 0.01, rng)
    D = np.zeros((900, 900), bool)
    D[np.repeat(np.arange(900), np.diff(hubs.rst)), hubs.col] = True
    for h in (3, 400, 401, 899):     # rows of over 128 entries, next to each other's
        D[h] = D[:, h] = rng.random(900) < 0.7
        D[h, h] = False
    D[3, 400] = D[400, 3] = D[400, 401] = D[401, 400] = True
    D |= D.T
    np.fill_diagonal(D, False)
    L = D.copy()
    L[np.arange(0, 900, 7), np.arange(0, 900, 7)] = True
    return [("one", random_graph(1, 0.0, rng)), ("two", random_graph(2, 1.5, rng)),
            ("none", random_graph(40, 0.0, rng)), ("dense", random_graph(120, 0.5, rng)),
            ("loops", _with_loops(90, 0.2, rng)), ("cliques", _clique_chain([3, 5, 8, 13, 21])),
            ("ladder", _ladder(300)), ("hubs", dense_to_csr(D)), ("hubs_loops", dense_to_csr(L))]


GRAPHS = _graphs()
KEYS = ("products", "mask_entries", "a_entries", "launches", "rows", "front_edges")


def _count(ctx, run):
    ctx.work_counters(reset=True)
    out = run()
    w = ctx.work_counters(reset=True)
    return out, {k: w[k] for k in KEYS}


@pytest.mark.parametrize("name,G", GRAPHS, ids=[g[0] for g in GRAPHS])
def test_one_launch(ctx, name, G):
    A = to_device(ctx, G)
    for k in (2, 3, 4, 5, 7, 11, 30):
        R, rit = oracle.ktruss(G, k)
        (C, it), w = _count(ctx, lambda: ga.ktruss("tri", A, k))
        r, c, v = C.download()
        assert it == rit and np.array_equal(r, R.rst) and np.array_equal(c, R.col[:R.nnz]), k
        ctx.set_option(ga.OPT_DEVICE_LOOPS, 0)
        try:
            (_, hit), hw = _count(ctx, lambda: ga.ktruss("tri", A, k))
        finally:
            ctx.set_option(ga.OPT_DEVICE_LOOPS, 1)
        assert hit == it and w == hw, k


@pytest.mark.parametrize("name,G", GRAPHS, ids=[g[0] for g in GRAPHS])
def test_sweep_one_launch(ctx, name, G):
    A = to_device(ctx, G)

    def sweep():
        out = []
        for k, C, it in ga.ktruss_sweep("tri", A, 3):
            out.append((k, it) + tuple(x.tobytes() for x in C.download()[:2]))
        return out

    one, w = _count(ctx, sweep)
    ctx.set_option(ga.OPT_DEVICE_LOOPS, 0)
    try:
        host, hw = _count(ctx, sweep)
    finally:
        ctx.set_option(ga.OPT_DEVICE_LOOPS, 1)
    assert one == host and w == hw
    cur = G
    for k, it, r, c in one:
        R, rit = oracle.ktruss(cur, k)
        assert it == rit and r == R.rst.tobytes() and c == R.col[:R.nnz].tobytes(), k
        cur = R


def test_large_frontiers(ctx):
    """Frontiers of many edges per warp and more segments than their list holds."""
    m, rst, col = ga.gen_rmat(14, 24, seed=5)
    G = oracle.Csr(m, m, rst, col, np.ones(len(col), np.int32))
    A = to_device(ctx, G)
    for k in (5, 20, 60):
        R, rit = oracle.ktruss(G, k)
        C, it = ga.ktruss("tri", A, k)
        r, c, _ = C.download()
        assert it == rit and np.array_equal(r, R.rst) and np.array_equal(c, R.col[:R.nnz]), k


def test_threads_share_the_device(built):
    """Two contexts run the loop at the same time."""
    from concurrent.futures import ThreadPoolExecutor
    m, rst, col = ga.gen_rmat(12, 16, seed=6)
    G = oracle.Csr(m, m, rst, col, np.ones(len(col), np.int32))
    want = {k: oracle.ktruss(G, k) for k in (4, 9)}

    def run(k):
        with ga.Context(0) as c:
            A = to_device(c, G)
            for _ in range(10):
                C, it = ga.ktruss("tri", A, k)
                r, cc, _ = C.download()
                R, rit = want[k]
                assert it == rit and np.array_equal(r, R.rst) and np.array_equal(cc, R.col[:R.nnz])
            A.free()
        return True

    with ThreadPoolExecutor(2) as ex:
        assert all(ex.map(run, (4, 9)))
