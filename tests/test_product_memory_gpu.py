"""Device memory of a product: the exact block kernel's scratch and tile lists
(at most a million segments for each of 304 blocks) are taken for the columns
that need them, and a product runs without room for them: such columns visit
every tile."""
import numpy as np
import pytest

from combblas_gb300 import _lib as L
from combblas_gb300 import batch, local
from mempool import SmallPool
from test_exact_visits_gpu import columns

pytestmark = pytest.mark.gpu

NOMEM = -2


def left(rng):
    """1.2 million entries in nearly as many (column, row tile) pairs."""
    A = columns(1 << 20, [np.unique(rng.integers(0, 1 << 20, 240)) for _ in range(5000)])
    A.values = rng.random(A.nnz) + 0.5
    return A


def right(rng, entries):
    B = columns(5000, [np.sort(rng.choice(5000, k, replace=False)) for k in entries])
    B.values = rng.random(B.nnz) + 0.5
    return B


def same(got, exp):
    for g, e in zip(got, exp):
        assert np.array_equal(np.asarray(g).view(np.int64), np.asarray(e).view(np.int64))


@pytest.mark.parametrize("sr", ["plustimes", "minplus"])
@pytest.mark.parametrize("entries", [[1] * 300 + [0] * 50, [1] * 300 + [20] * 10, [100]])
def test_scratch_is_for_the_columns_that_need_it(gpu_ctx, oracle_lib, sr, entries):
    O = oracle_lib
    rng = np.random.default_rng(len(entries))
    A, B = left(rng), right(rng, entries)
    exp = O.port_spgemm(A, B, O.SR_MINPLUS_F64) if sr == "minplus" else O.port_spgemm(A, B, 0, fold="exact")
    pool = SmallPool(1 << 20, 192 << 20)
    with pool.room(192):
        same(local.spgemm(A, B, sr=sr).to_csc(), exp)
        if sr == "plustimes":
            b = batch.Batch([A], [B])
            b.run()
            same(b.result(0), exp)
            b.close()
    assert pool.leaked() == 0
    pool.close()


@pytest.mark.parametrize("sr", ["plustimes", "minplus"])
def test_every_allocation_may_fail(gpu_ctx, oracle_lib, sr):
    O = oracle_lib
    rng = np.random.default_rng(9)
    A, B = left(rng), right(rng, [100, 2500, 20, 700, 1, 0] + [300] * 30)
    exp = O.port_spgemm(A, B, O.SR_MINPLUS_F64) if sr == "minplus" else O.port_spgemm(A, B, 0, fold="exact")
    pool, seen = SmallPool(1 << 20, 448 << 20), set()
    visits = set()
    for chunks in list(range(0, 160, 8)) + list(range(160, 448, 24)) + [448]:
        with pool.room(chunks):
            try:
                R = local.spgemm(A, B, sr=sr)
                same(R.to_csc(), exp)
                visits.add(R.stats.tile_visits_dense + R.stats.tile_visits_range)
                R.free()
                seen.add(True)
            except L.GbcError as e:
                assert e.code == NOMEM
                seen.add(False)
        assert pool.leaked() == 0
    pool.close()
    assert seen == {True, False}
    assert len(visits) > 1  # with and without room for the scratch
