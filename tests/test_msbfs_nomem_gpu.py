"""Multi-source BFS on a device without room: a call gives the right parents or
the error for it wherever an allocation fails, nothing is left allocated, and a
graph that met such a failure goes the same way as a new one afterwards."""
import numpy as np
import pytest

from combblas_gb300 import _lib as L
from combblas_gb300 import bfs as B
from mempool import SmallPool
from test_msbfs_bits_gpu import edges

pytestmark = pytest.mark.gpu

NOMEM = -2


def launches(call):
    n = L.lib().gbc_launch_count()
    got = call()
    return got, L.lib().gbc_launch_count() - n


@pytest.mark.parametrize("nroots", [1, 70])
def test_every_allocation_may_fail(gpu_ctx, oracle_lib, nroots):
    rng = np.random.default_rng(nroots)
    n = 100000 if nroots == 1 else 20000
    A = edges(n, np.concatenate([np.arange(n - 1), rng.integers(0, n, 2 * n)]),
              np.concatenate([np.arange(1, n), rng.integers(0, n, 2 * n)]))
    roots = rng.integers(0, n, nroots)
    want = oracle_lib.port_msbfs(A, roots)[0]
    fresh = B.Graph(A)
    B.msbfs(fresh, roots)
    usual = launches(lambda: B.msbfs(fresh, roots))[1]
    fresh.close()
    pool, seen = SmallPool(256 << 10, 128 << 20), set()
    for chunks in list(range(0, 30, 1 if nroots == 1 else 4)) + [40, 60, 100, 200, 300, 400]:
        g = B.Graph(A)
        with pool.room(chunks):
            try:
                assert np.array_equal(B.msbfs(g, roots)[0], want)
                seen.add(True)
            except L.GbcError as e:
                assert e.code == NOMEM
                seen.add(False)
        assert np.array_equal(B.msbfs(g, roots)[0], want)
        got, count = launches(lambda: B.msbfs(g, roots))
        assert np.array_equal(got[0], want) and count == usual
        g.close()
        assert pool.leaked() == 0
    pool.close()
    assert seen == {True, False}
