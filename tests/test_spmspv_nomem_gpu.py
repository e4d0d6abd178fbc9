"""SpMSpV on a device without room: wherever a call's allocations fail, it gives
the right vector (the product arrays of the pushed form can be done without) or
the error for it, and the same plan's next calls are right."""
import numpy as np
import pytest

from combblas_gb300 import _lib as L
from combblas_gb300 import bfs as B
from combblas_gb300 import generators as G
from mempool import SmallPool

pytestmark = pytest.mark.gpu

NOMEM = -2


def test_every_allocation_may_fail(gpu_ctx, oracle_lib):
    rng = np.random.default_rng(5)
    m, n = 1 << 17, 1 << 13
    A = G.csc_from_coo(m, n, rng.integers(0, m, 9 << 19), rng.integers(0, n, 9 << 19))
    assert A.nnz >= 1 << 22  # products are pushed
    A.values = rng.standard_normal(A.nnz)
    plan = B.SpMSpVPlan(A, np.float64)
    x = np.sort(rng.choice(n, n // 6, replace=False)).astype(np.int32)
    xv = rng.standard_normal(len(x))
    xi = rng.integers(0, 1 << 40, len(x))
    sums = oracle_lib.port_spmspv_sr(A, oracle_lib.SX_PLUSTIMES, x, xv)
    least = oracle_lib.port_spmspv(A.with_values(None), x, xi)
    short = oracle_lib.port_spmspv(A.with_values(None), x[:5], xi[:5])
    chunk, seen = 512 << 10, set()
    pool = SmallPool(chunk)
    for chunks in list(range(0, 12)) + [16, 20, 24, 28, 32, 48, 64, 100]:
        for name, v, want in (("plustimes", xv, sums), ("selectmin", xi, least)):
            with pool.room(chunks):
                try:
                    got = plan.multiply(x, v, name)
                    seen.add((name, True))
                except L.GbcError as e:
                    assert e.code == NOMEM
                    got = want
                    seen.add((name, False))
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
            got = plan.multiply(x[:5], xi[:5], "selectmin")
            assert np.array_equal(got[0], short[0]) and np.array_equal(got[1], short[1])
    pool.close()
    plan.close()
    assert len(seen) == 4  # both ended both ways
