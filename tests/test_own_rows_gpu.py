"""The ordered kernel whose warps own row ranges: columns just dense enough for
it and well above, few and many row ranges, skewed rows, B columns around the
32 entries a warp takes at a time, every semiring, bit for bit against the
oracle's fold in B-entry order (plain fp32 and fp64 sums depend on that order)."""
import numpy as np
import pytest

from combblas_gb300 import generators as G
from combblas_gb300 import local
from test_exact_visits_gpu import columns, pick
from test_spgemm_gpu import SR_NAME, assert_same
from test_oracle import typed

pytestmark = pytest.mark.gpu


def case(name):
    rng = np.random.default_rng(len(name))
    if name == "few rows":  # fewer rows than ranges, 1 to 97 entries a column
        A = columns(11, [pick(rng, 0, 11, 9) for _ in range(600)])
        return A, columns(600, [pick(rng, 0, 600, n) for n in (1, 31, 32, 33, 64, 97, 600)])
    if name == "skewed":  # half of all entries in 50 of 9000 rows
        A = columns(9000, [np.union1d(pick(rng, 0, 50, 45), pick(rng, 0, 9000, 400)) for _ in range(120)])
        return A, columns(120, [pick(rng, 0, 120, n) for n in (1, 5, 32, 40, 120)])
    # many ranges: fp64 reaches 96, whole columns and sparse ones in the same product
    A = columns(33000, [np.arange(33000) if k % 3 == 0 else pick(rng, 0, 33000, 900) for k in range(36)])
    return A, columns(36, [pick(rng, 0, 36, n) for n in (2, 17, 33, 36)])


@pytest.mark.parametrize("sr", [0, 1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("name", ["few rows", "skewed", "many ranges"])
def test_owned_rows_match_the_oracle(gpu_ctx, oracle_lib, name, sr):
    O = oracle_lib
    A, B = case(name)
    A.values, B.values = np.ones(A.nnz), np.ones(B.nnz)
    A, B = typed(A, sr, 3, O), typed(B, sr, 4, O)
    if sr in (0, 1):  # a lone -0.0 stays one
        rng = np.random.default_rng(2)
        A.values[rng.random(A.nnz) < 0.1] = -0.0
        A.values[rng.random(A.nnz) < 0.3] *= -1
    srname, dt = SR_NAME[sr]
    got = local.spgemm(A, B, sr=srname, dtype=dt, fold="ordered", tiny_limit=0, small_limit=0).to_csc()
    exp = O.port_spgemm(A, B, sr)
    assert_same(*got, *exp, sr, True, name)
    if sr in (0, 1):
        assert np.array_equal(np.signbit(got[2]), np.signbit(exp[2]))
