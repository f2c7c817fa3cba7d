"""C<A> = A·A of a matrix that was symmetric at its first product and whose
values were rewritten through its device addresses since: the product of the
present values. Small integers: equal to the oracle's.
"""
import numpy as np
import pytest

import graphalgo_gb300 as ga
import oracle
from graphs import to_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", ["msa", "mca", "heap"])
@pytest.mark.parametrize("asked", ["before the first product", "after it"])
def test_rewritten_in_place(ctx, algo, asked):
    m, rst, col = ga.gen_rmat(14, 20, seed=8)
    row = np.repeat(np.arange(m), np.diff(rst))
    assert len(col) >= 1 << 18
    G = oracle.Csr(m, m, rst, col, ((row + col) % 3 + 2).astype(np.int32))
    A, twin = to_device(ctx, G), to_device(ctx, G)
    if asked == "before the first product":
        A.device_ptrs()
    v = ga.mxm_masked(algo, A, A, A).download()[2]
    assert np.array_equal(v, oracle.mxm_masked(G, G, G))
    # rows scaled by 1 to 5: no longer symmetric
    scale = oracle.Csr(m, m, np.arange(m + 1, dtype=np.int32), np.arange(m, dtype=np.int32),
                       (np.arange(m) % 5 + 1).astype(np.int32))
    ga.mxm_masked_vals(algo, to_device(ctx, scale), twin, twin, A.device_ptrs()[2])
    H = oracle.Csr(m, m, rst, col, (G.val * (row % 5 + 1)).astype(np.int32))
    assert np.array_equal(A.download()[2], H.val)
    v = ga.mxm_masked(algo, A, A, A).download()[2]
    assert np.array_equal(v, oracle.mxm_masked(H, H, H))


def test_declared_symmetric(ctx):
    """Addresses asked for, symmetry declared: the product by halves, with the whole product's counters."""
    m, rst, col = ga.gen_rmat(14, 20, seed=8)
    G = oracle.Csr(m, m, rst, col, np.full(len(col), 2, np.int32))
    A = to_device(ctx, G)
    A.device_ptrs()
    A.set_symmetric(1)
    v = ga.mxm_masked("msa", A, A, A).download()[2]
    assert np.array_equal(v, oracle.mxm_masked(G, G, G))
