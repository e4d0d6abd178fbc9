"""PlusTimes SpMSpV over columns that hold a row more than once, in any order:
every stored entry counts, folded in column order and within a column in stored
order, bit for bit, whether the products are pushed (rows of at most 8, at most
32 and more products) or pulled (a matrix of fewer entries, or a vector that
brings more than a quarter of them), with the plan as it was afterwards."""
import numpy as np
import pytest

from combblas_gb300 import bfs as B
from combblas_gb300 import generators as G

pytestmark = pytest.mark.gpu

PUSH = 1 << 22  # entries from which products are pushed


@pytest.mark.parametrize("dtype", [np.float64, np.float32, np.int64])
@pytest.mark.parametrize("m,n,size", [(4000, 900, PUSH), (60, 900, PUSH), (7, 300, PUSH), (4000, 900, PUSH // 8)])
def test_repeated_rows(gpu_ctx, oracle_lib, m, n, size, dtype):
    rng = np.random.default_rng(m + n)
    cols = [np.repeat(rng.integers(0, m, 3), 2) for _ in range(n)]  # some rows twice, three or four times
    for c in cols:
        rng.shuffle(c)
    fill = size - 6 * n  # a column that brings nearly all entries
    cols.append(np.arange(fill))
    cp = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int64)
    A = G.CSC(max(m, fill), n + 1, cp, np.concatenate(cols).astype(np.int64), None)
    A.values = (rng.standard_normal(A.nnz) * 100).astype(dtype)
    plan = B.SpMSpVPlan(A, dtype)
    some = np.sort(rng.choice(n, n // 2, replace=False))
    for x in (some, np.append(some, n), some[:3]):
        x = x.astype(np.int32)
        xv = (rng.standard_normal(len(x)) * 100).astype(dtype)
        er, ev = oracle_lib.port_spmspv_sr(A, oracle_lib.SX_PLUSTIMES, x, xv, dtype)
        for _ in range(2):
            r, v = plan.multiply(x, xv, "plustimes")
            assert np.array_equal(r, er) and np.array_equal(v, ev)
    plan.close()
