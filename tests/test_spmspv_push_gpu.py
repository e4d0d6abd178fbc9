"""PlusTimes SpMSpV whose products are pushed to their rows: rows of one, of at
most 8, of at most 32 and of more products (folded by a thread, a warp, or
pulled), vectors in any order, vectors long enough that all rows are pulled, and
matrices with one entry less than the push asks for, bit for bit against the oracle's fold in ascending column order."""
import numpy as np
import pytest

from combblas_gb300 import bfs as B
from combblas_gb300 import generators as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("small", [False, True])
@pytest.mark.parametrize("dtype", [np.float64, np.float32, np.int64])
@pytest.mark.parametrize("m,nx", [(20000, 700), (500, 600), (90, 31), (90, 33), (300, 1), (300, 4000), (60000, 2049)])
def test_pushed_products_match_the_oracle(gpu_ctx, oracle_lib, m, nx, dtype, small):
    rng = np.random.default_rng(m + nx)
    n = 4000
    rows = np.concatenate([rng.integers(1, m, 20 * n), np.zeros(n, np.int64)])  # every column hits row 0
    A = G.csc_from_coo(m, n, rows, np.concatenate([np.tile(np.arange(n), 20), np.arange(n)]))
    # one more column, which no vector names, makes up the entries
    fill = (1 << 22) - A.nnz - (1 if small else 0)
    m = max(m, fill)
    A = G.CSC(m, n + 1, np.append(A.colptr, A.nnz + fill), np.concatenate([A.rowidx, np.arange(fill)]), None)
    A.values = (rng.standard_normal(A.nnz) * 100).astype(dtype)
    x = rng.choice(n, nx, replace=False).astype(np.int32)  # in no order
    xv = (rng.standard_normal(nx) * 100).astype(dtype)
    plan = B.SpMSpVPlan(A, dtype)
    order = np.argsort(x)
    er, ev = oracle_lib.port_spmspv_sr(A, oracle_lib.SX_PLUSTIMES, x[order], xv[order], dtype)
    for _ in range(2):  # the plan's scratch is left as it was found
        r, v = plan.multiply(x, xv, "plustimes")
        assert np.array_equal(r, er) and np.array_equal(v, ev)
    plan.close()
