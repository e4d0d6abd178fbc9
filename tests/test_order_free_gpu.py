"""The block kernel over semirings whose add does not depend on the order: every
kind of visit (see test_exact_visits_gpu) for every such semiring, values at the
ends of their range, and fp64 min-plus columns with NaN or -0.0 among the
products, which have to keep the fold in B-entry order."""
import numpy as np
import pytest

from combblas_gb300 import local
from test_exact_visits_gpu import case
from test_spgemm_gpu import SR_NAME

pytestmark = pytest.mark.gpu

KINDS = ["direct, many segments", "direct, many rounds", "ranked, cut", "ranked, full tiles", "sorted", "many tiles"]


def same(A, B, sr, O):
    name, dt = SR_NAME[sr]
    got = local.spgemm(A, B, sr=name, dtype=dt, tiny_limit=0, small_limit=0).to_csc()
    exp = O.port_spgemm(A, B, sr)
    assert np.array_equal(got[0], exp[0]) and np.array_equal(got[1], exp[1])
    g, e = got[2], np.asarray(exp[2])
    if g.dtype == np.float64:
        assert np.array_equal(np.isnan(g), np.isnan(e))
        g, e = np.where(np.isnan(g), 0, g).view(np.int64), np.where(np.isnan(e), 0, e).view(np.int64)
    assert np.array_equal(g, e)


@pytest.mark.parametrize("sr", [2, 3, 4, 5, 6])
@pytest.mark.parametrize("kind", KINDS)
def test_visits_match_the_oracle(gpu_ctx, oracle_lib, kind, sr):
    rng = np.random.default_rng(sr)
    A, B = case(kind, rng)
    dt = SR_NAME[sr][1]
    for M in (A, B):
        if dt == np.bool_:
            M.values = rng.random(M.nnz) < 0.2  # entries whose products are all false stay, with value false
        elif dt == np.int64:
            M.values = rng.integers(-(1 << 62), 1 << 62, M.nnz)
            M.values[rng.random(M.nnz) < 0.02] = np.iinfo(np.int64).max  # min-plus: infinity
            M.values[rng.random(M.nnz) < 0.02] = np.iinfo(np.int64).min
        else:
            M.values = rng.integers(-40, 40, M.nnz) * 0.5
            M.values[rng.random(M.nnz) < 0.02] = np.inf
            M.values[rng.random(M.nnz) < 0.02] = np.finfo(np.float64).max  # the semiring's infinity
    same(A, B, sr, oracle_lib)


@pytest.mark.parametrize("special", [np.nan, -0.0])
@pytest.mark.parametrize("kind", KINDS)
def test_min_plus_keeps_the_order_where_it_matters(gpu_ctx, oracle_lib, kind, special):
    rng = np.random.default_rng(8)
    A, B = case(kind, rng)
    for M in (A, B):
        M.values = rng.integers(-2, 3, M.nnz).astype(np.float64)
        M.values[rng.random(M.nnz) < 0.3] = special
    same(A, B, 3, oracle_lib)
