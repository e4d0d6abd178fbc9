"""The passes that check and prepare the operands: columns at the lengths where
the whole block takes over from a warp and where the unrolled loads end, over few
and over more row tiles than one pass of mask words holds, and faults in every
part of a long column."""
import numpy as np
import pytest

from combblas_gb300 import local
from combblas_gb300._lib import GbcError
from test_exact_visits_gpu import columns, pick

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 31, 32, 33, 127, 128, 129, 255, 256, 257, 1023, 1024, 1025, 2049, 2900]


@pytest.mark.parametrize("m", [3000, 4096 * 256 + 1, 4096 * 600 + 7])
def test_product_of_columns_of_all_lengths(gpu_ctx, oracle_lib, m):
    rng = np.random.default_rng(m)
    A = columns(m, [pick(rng, 0, m, LENGTHS[k % 16] if k < 64 else k % 3) for k in range(3000)])
    B = columns(3000, [pick(rng, 0, 3000, k) for k in LENGTHS])
    for M in (A, B):
        M.values = rng.integers(-4, 5, M.nnz).astype(np.float64)
    R = local.spgemm(A, B, fold="exact")
    exp = oracle_lib.port_spgemm(A, B, 0, fold="exact")
    for g, e in zip(R.to_csc(), exp):
        assert np.array_equal(g, e)
    lens = np.diff(A.colptr)
    assert R.stats.flops == int(lens[B.rowidx].sum())


@pytest.mark.parametrize("at", [1, 31, 32, 255, 256, 700, 1024, 1025, 2899])
def test_faults_in_a_long_column_are_reported(gpu_ctx, at):
    n = 3000
    good = columns(n, [np.arange(2900), np.arange(5)])
    good.values = np.ones(good.nnz)
    eye = columns(2, [np.array([0]), np.array([1])])
    eye.values = np.ones(2)
    wide = columns(5, [np.array([0])] * n)
    wide.values = np.ones(n)
    for row, word in ((at - 1, "ascending"), (n, "out of range")):
        bad = columns(n, [np.arange(2900), np.arange(5)])
        bad.values = np.ones(bad.nnz)
        bad.rowidx[at] = row
        with pytest.raises(GbcError, match=word):
            local.spgemm(bad, eye)
        with pytest.raises(GbcError, match=word):
            local.spgemm(wide, bad)
