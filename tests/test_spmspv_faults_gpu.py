"""SpMSpV calls that end in an error: a vector that names a column so often that
its products pass 32 bits is refused like any other repeated index, before
anything is sized by them, and the plan multiplies on as if nothing had been."""
import numpy as np
import pytest

from combblas_gb300 import _lib as L
from combblas_gb300 import bfs as B
from combblas_gb300 import generators as G

pytestmark = pytest.mark.gpu


def matrix(rng, dtype):
    """2^22 entries and more (PlusTimes pushes its products): 64 columns of 2^16 rows and 500 of 60."""
    m, lens = 1 << 17, [1 << 16] * 64 + [60] * 500
    cp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    rows = np.concatenate([np.sort(rng.choice(m, k, replace=False)) for k in lens])
    M = G.CSC(m, len(lens), cp, rows.astype(np.int64), None)
    M.values = (rng.standard_normal(M.nnz) * 100).astype(dtype)
    return M


@pytest.mark.parametrize("dtype", [np.float64, np.int64])
def test_repeated_and_foreign_columns(gpu_ctx, oracle_lib, dtype):
    rng = np.random.default_rng(3)
    A = matrix(rng, dtype)
    plan = B.SpMSpVPlan(A, dtype)
    x = np.sort(rng.choice(np.arange(64, A.ncol), 200, replace=False)).astype(np.int32)
    xv = (rng.standard_normal(200) * 100).astype(dtype)
    good = oracle_lib.port_spmspv_sr(A, oracle_lib.SX_PLUSTIMES, x, xv, dtype)
    xi = rng.integers(0, 1 << 40, 200)
    least = oracle_lib.port_spmspv(A.with_values(None), x, xi)
    bad = [np.full(1 << 16, 5), np.array([70, 9, 70]), np.array([1, A.ncol]), np.array([-1, 3]),
           np.concatenate([np.full(1 << 16, 5), [A.ncol]])]
    for b in bad:
        for name, d in (("plustimes", dtype), ("selectmin", np.int64), ("selectmax", np.int64)):
            with pytest.raises(L.GbcError):
                plan.multiply(b.astype(np.int32), np.ones(len(b), d), name)
            r, v = plan.multiply(x, xv, "plustimes")
            assert np.array_equal(r, good[0]) and np.array_equal(v, good[1])
            r, v = plan.multiply(x, xi, "selectmin")
            assert np.array_equal(r, least[0]) and np.array_equal(v, least[1])
    plan.close()
