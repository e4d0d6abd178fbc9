"""Which kernels take a column where A has more row tiles than the exact block
kernel buckets, told by its visits: the order-free semirings leave it there, the
oracle's values either way."""
import numpy as np
import pytest

from combblas_gb300 import local
from test_exact_visits_gpu import columns
from test_spgemm_gpu import SR_NAME

pytestmark = pytest.mark.gpu

BUCKETED = 1 << 20  # rows


def product(oracle, m, sr, deg, nb, cols=40, empty=0):
    """Visits of the default product of `cols` columns of deg x nb products over m rows, A with `empty` columns more."""
    rng = np.random.default_rng(m + deg)
    A = columns(m, [np.unique(rng.integers(0, m, deg)) for _ in range(2000)] + [np.array([], np.int64)] * empty)
    B = columns(2000 + empty, [np.sort(rng.choice(2000, nb, replace=False)) for _ in range(cols)])
    name, dt = SR_NAME[sr]
    for M in (A, B):
        M.values = (rng.random(M.nnz) * 100 + 1).astype(dt)
    R = local.spgemm(A, B, sr=name, dtype=dt)
    got = R.to_csc()
    exp = oracle.port_spgemm(A, B, sr, fold="exact") if sr == 0 else oracle.port_spgemm(A, B, sr)
    for g, e in zip(got, exp):
        assert np.array_equal(g, e)
    return R.stats.tile_visits_dense + R.stats.tile_visits_range


@pytest.mark.parametrize("sr", [2, 3, 4, 5, 6])
def test_order_free_semirings(gpu_ctx, oracle_lib, sr):
    assert product(oracle_lib, BUCKETED, sr, 60, 100) > 0
    assert product(oracle_lib, BUCKETED + 1, sr, 60, 100) == 0


@pytest.mark.parametrize("m,sr,nb,blocks", [
    (1 << 16, 3, 20, True), ((1 << 16) + 1, 3, 20, False), ((1 << 16) + 1, 3, 40, True),
    (1 << 19, 5, 40, True), ((1 << 19) + 1, 5, 40, False), ((1 << 19) + 1, 3, 40, True), ((1 << 19) + 1, 5, 100, True),
    (BUCKETED, 0, 20, True), (BUCKETED + 1, 0, 40, False), (BUCKETED + 1, 0, 100, True)])
def test_columns_of_1200_2400_and_6000_products(gpu_ctx, oracle_lib, m, sr, nb, blocks):
    assert (product(oracle_lib, m, sr, 60, nb, cols=3000) > 0) == blocks


@pytest.mark.parametrize("sr", [0, 3])
@pytest.mark.parametrize("m,nb,cols,blocks", [
    (1 << 14, 5, 40, False), (1 << 14, 15, 40, True), (1 << 14, 15, 3000, False), ((1 << 16) + 1, 15, 40, False)])
def test_few_columns_of_300_and_900_products(gpu_ctx, oracle_lib, m, nb, cols, blocks, sr):
    """On their own: to the blocks only where each has one, long enough, over few tiles."""
    assert (product(oracle_lib, m, sr, 60, nb, cols) > 0) == blocks


def test_few_columns_above_the_bucketed_rows(gpu_ctx, oracle_lib):
    assert product(oracle_lib, BUCKETED + 1, 0, 60, 15) == 0


@pytest.mark.parametrize("sr", [0, 2, 3, 4, 5, 6])
def test_hypersparse_operands(gpu_ctx, oracle_lib, sr):
    """120000 entries in 150000 columns of 2^20 rows: the order-free semirings keep their higher tiles."""
    assert (product(oracle_lib, BUCKETED, sr, 60, 100, empty=150000) > 0) == (sr == 0)
