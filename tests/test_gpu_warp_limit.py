"""Small masked products, whose rows go to warps or CTAs by a limit estimated
from a sample of A's entries: fewer and more entries than the sample, none,
rows on both sides of the limit. Whole numbers: equal to the oracle's.
"""
import numpy as np
import pytest

import graphalgo_gb300 as ga
import oracle
from graphs import to_device

pytestmark = pytest.mark.gpu


def _rows(lengths, n, rng, dtype):
    rst = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    col = np.concatenate([np.sort(rng.choice(n, d, replace=False)) for d in lengths] or [[]]).astype(np.int32)
    return oracle.Csr(len(lengths), n, rst, col, rng.integers(-3, 4, len(col)).astype(dtype))


CASES = {"none": [0] * 5, "one": [0, 1, 0], "sample-1": [341] * 3, "sample": [512, 512], "sample+1": [5] * 205,
         "hub": [3] * 300 + [900] + [3] * 300, "all long": [700] * 40, "mixed": list(range(0, 600, 7)),
         "many": [2] * 60000}


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("algo", ["msa", "mca", "heap", "hybrid"])
def test_limit(ctx, name, algo):
    rng = np.random.default_rng(len(name))
    m, k, n = len(CASES[name]), 1000, 4000
    A = _rows(CASES[name], k, rng, np.int32)
    B = _rows(np.where(np.arange(k) % 50 == 0, 900, 8).tolist(), n, rng, np.int32)
    M = _rows(rng.integers(0, 40, m).tolist(), n, rng, np.int32)
    for option in (32768, 0, 1 << 40):
        ctx.set_option(ga.OPT_MXM_WARP_FLOPS, option)
        try:
            C = ga.mxm_masked(algo, to_device(ctx, A), to_device(ctx, B), to_device(ctx, M))
        finally:
            ctx.set_option(ga.OPT_MXM_WARP_FLOPS, 32768)
        rst, col, val = C.download()
        assert np.array_equal(rst, M.rst) and np.array_equal(col, M.col)
        assert np.array_equal(val, oracle.mxm_masked(A, B, M)), option
