"""The exact block kernel's visits at their edges: direct tiles of many
segments and of many product rounds, ranked runs that are cut because their
output does not fit, sorted ranges, more row tiles than are bucketed, each with
positive and with mixed values (zeros of both signs and cancellation among
them).  Every value is the exact sum of the rounded products, rounded once, so
the bits have to be the oracle's."""
import numpy as np
import pytest

from combblas_gb300 import generators as G
from combblas_gb300 import local

pytestmark = pytest.mark.gpu


def columns(m, lists):
    """CSC of m rows from one ascending row list per column."""
    cp = np.concatenate([[0], np.cumsum([len(r) for r in lists])]).astype(np.int64)
    return G.CSC(m, len(lists), cp, np.concatenate(lists).astype(np.int64), None)


def pick(rng, lo, hi, n):
    return np.sort(rng.choice(np.arange(lo, hi), n, replace=False))


def case(name, rng):
    if name == "direct, many segments":  # 3000 segments, three chunk tables
        A = columns(5000, [pick(rng, 0, 4096, 5) for _ in range(3000)])
        B = columns(3000, [np.arange(3000), pick(rng, 0, 3000, 1025), pick(rng, 0, 3000, 1024)])
    elif name == "direct, many rounds":  # more than 16384 products in few long segments
        A = columns(9000, [pick(rng, 0, 4096, 4000) for _ in range(12)])
        B = columns(12, [np.arange(12), np.arange(5), np.arange(4), np.arange(1)])
    elif name == "ranked, cut":  # 3000 different rows in every tile: two tiles do not fit one visit
        A = columns(40000, [np.concatenate([pick(rng, t * 4096, min(40000, t * 4096 + 4096), 1500) for t in range(9)])
                            for _ in range(6)])
        B = columns(6, [np.array([0, 1]), np.arange(6), np.array([5])])
    elif name == "ranked, full tiles":  # exactly 4096 rows of a tile, and the last, ragged one
        A = columns(20001, [np.arange(0, 20001), np.arange(4095, 8193), np.arange(1, 20000, 7)])
        B = columns(3, [np.array([0]), np.array([1]), np.array([0, 1, 2]), np.array([2])])
    elif name == "sorted":  # a few products in each of 256 tiles
        A = columns(1 << 20, [pick(rng, 0, 1 << 20, 700) for _ in range(40)])
        B = columns(40, [np.array([3, 7]), np.arange(4), np.arange(40)])
    else:  # more than 256 tiles
        A = columns((1 << 20) + 5000, [pick(rng, 0, (1 << 20) + 5000, 3000) for _ in range(30)])
        B = columns(30, [np.arange(30), np.array([29])])
    return A, B


@pytest.mark.parametrize("signs", ["positive", "mixed"])
@pytest.mark.parametrize("name", ["direct, many segments", "direct, many rounds", "ranked, cut",
                                  "ranked, full tiles", "sorted", "many tiles"])
def test_visits_match_the_oracle_bit_for_bit(gpu_ctx, oracle_lib, name, signs):
    O = oracle_lib
    rng = np.random.default_rng(len(name))
    A, B = case(name, rng)
    for M in (A, B):
        if signs == "positive":
            M.values = 1.0 - rng.random(M.nnz)
        else:  # small whole numbers cancel often; some terms are +-0.0
            M.values = rng.integers(-3, 4, M.nnz) * np.where(rng.random(M.nnz) < 0.5, 1.0, 0.125)
            M.values[rng.random(M.nnz) < 0.05] = -0.0
    cp, rows, vals = local.spgemm(A, B, fold="exact", tiny_limit=0, small_limit=0).to_csc()
    pcp, prow, pval = O.port_spgemm(A, B, O.SR_PLUSTIMES_F64, fold="exact")
    assert np.array_equal(cp, pcp) and np.array_equal(rows, prow)
    assert np.array_equal(vals.view(np.int64), pval.view(np.int64))
