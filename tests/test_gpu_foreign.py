"""k-truss and sweep calls of one context on another context's matrix, which is
freed and its memory written again as soon as the call returns; and a sweep
whose allocations fail one after the other. Whole numbers: equal to the
oracle's.
"""
import ctypes

import numpy as np
import pytest

import graphalgo_gb300 as ga
import oracle
from graphs import to_device

pytestmark = pytest.mark.gpu


def test_matrix_of_another_context(built):
    m, rst, col = ga.gen_rmat(13, 16, seed=12)
    G = oracle.Csr(m, m, rst, col, np.ones(len(col), np.int32))
    R, rit = oracle.ktruss(G, 5)
    with ga.Context(0) as own, ga.Context(0) as other:
        for _ in range(5):
            A = to_device(own, G)
            own.sync()
            c, it = ctypes.c_void_p(), ctypes.c_int()
            rc = ga.lib().ga_ktruss(other.handle, ga.TRI, A.handle, 5, ctypes.byref(c), ctypes.byref(it))
            A.free()
            junk = [to_device(own, G) for _ in range(2)]
            assert rc == 0
            C = ga.Csr(other, c)
            r, cc, _ = C.download()
            assert it.value == rit and np.array_equal(r, R.rst) and np.array_equal(cc, R.col[:R.nnz])
            for x in junk:
                x.free()


def test_sweep_out_of_memory(ctx):
    m, rst, col = ga.gen_rmat(9, 8, seed=3)
    G = oracle.Csr(m, m, rst, col, np.ones(len(col), np.int32))
    A = to_device(ctx, G)
    ga.ktruss("tri", A, 3)

    def sweep():
        return [(k, it) + tuple(x.tobytes() for x in C.download()[:2]) for k, C, it in ga.ktruss_sweep("tri", A, 3)]

    want = sweep()
    failed = 0
    for n in range(400):
        ctx.set_option(ga.OPT_FAIL_ALLOC_AFTER, n)
        try:
            got = sweep()
        except ga.GaError:
            failed += 1
            continue
        finally:
            ctx.set_option(ga.OPT_FAIL_ALLOC_AFTER, -1)
        assert got == want
        break
    assert failed and sweep() == want
