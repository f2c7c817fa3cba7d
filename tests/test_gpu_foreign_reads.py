"""Calls of one context on another context's matrix, which is freed and its
memory written again as soon as the call returns. Whole numbers: equal to what
the matrix gives.
"""
import ctypes

import numpy as np
import pytest

import graphalgo_gb300 as ga
import oracle
from graphs import to_device

pytestmark = pytest.mark.gpu


def _graph_and_other(scale):
    """A graph, and one of as many vertices and entries that takes its memory (the vertices in reverse)."""
    m, rst, col = ga.gen_rmat(scale, 16, seed=12)
    val = np.arange(len(col), dtype=np.int32)
    ends = np.concatenate([[0], np.cumsum(np.diff(rst)[::-1])]).astype(np.int32)
    return oracle.Csr(m, m, rst, col, val), oracle.Csr(m, m, ends, (m - 1 - col[::-1]).astype(np.int32), -val - 1)


def test_transpose_of_another_contexts_matrix(built):
    G, other_graph = _graph_and_other(15)
    row = np.repeat(np.arange(G.m, dtype=np.int32), np.diff(G.rst))
    order = np.argsort(G.col, kind="stable")
    starts = np.concatenate([[0], np.cumsum(np.bincount(G.col, minlength=G.m))])
    with ga.Context(0) as own, ga.Context(0) as other:
        for _ in range(5):
            A = to_device(own, G)
            own.sync()
            t = ctypes.c_void_p()
            rc = ga.lib().ga_transpose(other.handle, A.handle, ctypes.byref(t))
            A.free()
            junk = [to_device(own, other_graph) for _ in range(2)]
            assert rc == 0
            r, c, v = ga.Csr(other, t).download()
            assert np.array_equal(r, starts) and np.array_equal(c, row[order]) and np.array_equal(v, G.val[order])
            for x in junk:
                x.free()


@pytest.mark.parametrize("algo", [ga.MSA, ga.MCA, ga.HEAP])
def test_triangle_count_of_another_contexts_matrix(built, algo):
    G, other_graph = _graph_and_other(13)
    total, rows = oracle.tc_sandia(oracle.Csr(G.m, G.m, G.rst, G.col, np.ones(len(G.col), np.int32)))
    with ga.Context(0) as own, ga.Context(0) as other:
        # room for the counts: the total, and the rows 256 bytes behind it
        out = to_device(other, oracle.Csr(G.m, G.m, G.rst, G.col, np.zeros(len(G.col), np.int64)))
        d_total = out.device_ptrs()[2]
        for _ in range(5):
            A = to_device(own, G)
            own.sync()
            rc = ga.lib().ga_tc_device(other.handle, algo, A.handle, ctypes.c_void_p(d_total),
                                       ctypes.c_void_p(d_total + 256))
            A.free()
            junk = [to_device(own, other_graph) for _ in range(2)]
            assert rc == 0
            got = out.download()[2]
            assert got[0] == total and np.array_equal(got[32:32 + G.m], rows)
            for x in junk:
                x.free()
