"""Operands of more rows than tiles of 4096 rows are kept for: a request for
higher tiles takes them under the exact fold as under the others, with the
oracle's bits, though the exact kernel's own tiles stay 4096 rows high."""
import numpy as np
import pytest

from combblas_gb300 import _lib as L
from combblas_gb300 import local
from test_exact_visits_gpu import columns

pytestmark = pytest.mark.gpu

LIMIT = 4096 * 64 * 64


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("tile_rows", [8192, 16384])
def test_more_rows_than_small_tiles_take(gpu_ctx, oracle_lib, tile_rows, special):
    O = oracle_lib
    rng = np.random.default_rng(tile_rows)
    m = 2 * LIMIT  # the most that 8192-row tiles take
    A = columns(m, [np.unique(np.concatenate([rng.integers(0, m, 700), [0, LIMIT - 1, LIMIT, m - 1]]))
                    for _ in range(20)])
    B = columns(20, [np.arange(20), np.array([3]), np.arange(0, 20, 3), np.array([], np.int64)])
    for M in (A, B):
        M.values = rng.random(M.nnz) - 0.4
    if special:  # columns that the exact kernel hands to the ordered one
        A.values[::50] = 1e-310
    got = local.spgemm(A, B, tile_rows=tile_rows).to_csc()
    exp = O.port_spgemm(A, B, O.SR_PLUSTIMES_F64, fold="exact")
    for g, e in zip(got, exp):
        assert np.array_equal(np.asarray(g).view(np.int64), np.asarray(e).view(np.int64))


@pytest.mark.parametrize("m,tile_rows", [(LIMIT + 1, 0), (LIMIT + 1, 4096), (2 * LIMIT + 1, 8192)])
def test_more_rows_still_are_refused(gpu_ctx, m, tile_rows):
    A = columns(m, [np.array([0, m - 1])])
    B = columns(1, [np.array([0])])
    for M in (A, B):
        M.values = np.ones(M.nnz)
    with pytest.raises(L.GbcError):
        local.spgemm(A, B, tile_rows=tile_rows)
