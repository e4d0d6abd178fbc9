"""Exact sums over operands with stored zeros: an entry is -0.0 where all its
terms are, +0.0 where its terms cancel or one of them is +0.0, in every kind of
visit; and such operands cost about what others do."""
import numpy as np
import pytest

from combblas_gb300 import generators as G
from combblas_gb300 import local
from test_exact_visits_gpu import case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("share", [0.02, 0.6, 1.0])
@pytest.mark.parametrize("kind", ["direct, many segments", "direct, many rounds", "ranked, cut", "ranked, full tiles",
                                  "sorted", "many tiles"])
def test_signs_of_zeros(gpu_ctx, oracle_lib, kind, share):
    O = oracle_lib
    rng = np.random.default_rng(int(share * 100) + len(kind))
    A, B = case(kind, rng)
    for M in (A, B):
        M.values = rng.choice([-1.0, 1.0, 2.0], M.nnz)
        zero = rng.random(M.nnz) < share
        M.values[zero] = rng.choice([0.0, -0.0], int(zero.sum()))
    got = local.spgemm(A, B, fold="exact", tiny_limit=0, small_limit=0).to_csc()
    exp = O.port_spgemm(A, B, O.SR_PLUSTIMES_F64, fold="exact")
    assert (exp[2] == 0).any()
    for g, e in zip(got, exp):
        assert np.array_equal(np.asarray(g).view(np.int64), np.asarray(e).view(np.int64))


def test_zeros_cost_little(gpu_ctx):
    """One more bit per product: well below four times the product without zeros (looking the terms up took 14)."""
    A = G.rmat(13, 8, seed=3)
    rng = np.random.default_rng(1)
    A.values = rng.random(A.nnz) - 0.5

    def ms():
        return min(local.spgemm(A, A, fold="exact").stats.ms_total for _ in range(5))

    plain = ms()
    A.values[rng.random(A.nnz) < 0.1] = 0.0
    assert ms() < 4 * plain
