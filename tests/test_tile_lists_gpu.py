"""Left operands whose tile lists have more entries than the operand itself
(columns of one entry, mostly empty columns) and are sized by a bound: beside
big columns that are bucketed through those lists, and in a batch, against the
oracle's bits."""
import numpy as np
import pytest

from combblas_gb300 import batch, local
from test_exact_visits_gpu import columns, pick

pytestmark = pytest.mark.gpu


def operands(name, rng):
    if name == "identity":
        n = 5000
        A = columns(n, [np.array([j]) for j in range(n)])
        B = columns(n, [np.arange(n), pick(rng, 0, n, 2000), np.array([], np.int64), pick(rng, 0, n, 3)])
    elif name == "mostly empty":  # 40 columns of 200 entries in a million rows, 60000 empty ones
        n, at = 60000, pick(rng, 0, 60000, 40)
        lists = [np.array([], np.int64)] * n
        for j in at:
            lists[j] = pick(rng, 0, 1 << 20, 200)
        A = columns(1 << 20, lists)
        B = columns(n, [at, np.arange(0, n, 7), at[::3]])
    else:  # 8192 entries, one more makes the count be read back
        n = 8192 + (name == "past the bound")
        A = columns(3 * n, [np.array([3 * j]) for j in range(n)])
        B = columns(n, [np.arange(n), pick(rng, 0, n, 1500)])
    for M in (A, B):
        M.values = rng.random(M.nnz) - 0.3
    return A, B


NAMES = ["identity", "mostly empty", "at the bound", "past the bound"]


@pytest.mark.parametrize("form", ["csc", "dcsc"])
@pytest.mark.parametrize("name", NAMES)
def test_short_columns_match_the_oracle(gpu_ctx, oracle_lib, name, form):
    O = oracle_lib
    A, B = operands(name, np.random.default_rng(6))
    hand = (lambda M: M) if form == "csc" else local.DCSC.from_csc
    for sr, port in (("plustimes", O.SR_PLUSTIMES_F64), ("minplus", O.SR_MINPLUS_F64)):
        exp = O.port_spgemm(A, B, port) if sr == "minplus" else O.port_spgemm(A, B, port, fold="exact")
        for kw in ({}, {"tiny_limit": 0, "small_limit": 0}):
            got = local.spgemm(hand(A), hand(B), sr=sr, **kw).to_csc()
            assert np.array_equal(got[0], exp[0]) and np.array_equal(got[1], exp[1])
            assert np.array_equal(got[2].view(np.int64), exp[2].view(np.int64))


def test_short_columns_in_a_batch(gpu_ctx, oracle_lib):
    O = oracle_lib
    pairs = [operands(name, np.random.default_rng(7)) for name in NAMES]
    b = batch.Batch([A for A, _ in pairs], [B for _, B in pairs])
    b.run()
    for p, (A, B) in enumerate(pairs):
        exp = O.port_spgemm(A, B, O.SR_PLUSTIMES_F64, fold="exact")
        cp, ir, num = b.result(p)
        assert np.array_equal(cp, exp[0]) and np.array_equal(ir, exp[1])
        assert np.array_equal(num.view(np.int64), exp[2].view(np.int64))
    b.close()
