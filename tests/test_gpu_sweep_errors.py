"""A k-truss sweep whose allocations fail one after the other, asked again
after each error: it reports an error or returns what the undisturbed sweep
returns (k, iteration count and edges).
"""
import ctypes

import numpy as np
import pytest

import graphalgo_gb300 as ga
import oracle
from graphs import to_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", [ga.TRI, ga.MSA])
def test_asked_again_after_an_error(ctx, algo):
    m, rst, col = ga.gen_rmat(9, 8, seed=3)
    A = to_device(ctx, oracle.Csr(m, m, rst, col, np.ones(len(col), np.int32)))
    lib = ga.lib()

    def sweep(first_to_fail):
        """The results up to the empty one, and the errors met."""
        h, got, errors = ctypes.c_void_p(), [], 0
        assert lib.ga_ktruss_sweep_begin(ctx.handle, algo, A.handle, 3, ctypes.byref(h)) == 0
        ctx.set_option(ga.OPT_FAIL_ALLOC_AFTER, first_to_fail)
        try:
            while errors < 4:
                c, k, it = ctypes.c_void_p(), ctypes.c_int(), ctypes.c_int()
                if lib.ga_ktruss_sweep_next(h, ctypes.byref(c), ctypes.byref(k), ctypes.byref(it)) != 0:
                    assert not c
                    errors += 1
                    continue
                if not c:
                    break
                C = ga.Csr(ctx, c)
                got.append((k.value, it.value) + tuple(x.tobytes() for x in C.download()[:2]))
                C.free()
        finally:
            ctx.set_option(ga.OPT_FAIL_ALLOC_AFTER, -1)
            lib.ga_ktruss_sweep_free(h)
        return got, errors

    want, errors = sweep(-1)
    assert errors == 0
    failed = 0
    for n in range(2000):
        got, errors = sweep(n)
        assert got == want[:len(got)], n
        if errors == 0:
            assert got == want
            break
        failed += 1
    assert failed and errors == 0
