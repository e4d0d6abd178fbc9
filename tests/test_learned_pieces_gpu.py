"""The learned products' gather into the contiguous result, which cuts the
result and not the columns into pieces: columns that span pieces, that end where
a piece ends, and long runs of empty columns, for each width of value."""
import numpy as np
import pytest

from combblas_gb300 import local
from test_exact_visits_gpu import columns, pick
from test_learned_gpu import trained_model
from combblas_gb300 import generators as G

pytestmark = pytest.mark.gpu

LENGTHS = {
    "one piece and a bit": [1024, 1, 1023, 0, 1025],
    "a long column between empty ones": [0] * 40 + [9000] + [0] * 70 + [3] * 33 + [0] * 31,
    "single entries": [1] * 2050,
    "one entry": [0] * 64 + [1],
}


@pytest.mark.parametrize("sr,dtype", [("plustimes", np.float64), ("plustimes", np.float32), ("bool", np.bool_)])
@pytest.mark.parametrize("kind", list(LENGTHS))
def test_pieces(gpu_ctx, kind, sr, dtype):
    rng = np.random.default_rng(4)
    n = len(LENGTHS[kind])
    A = columns(10000, [pick(rng, 0, 10000, k) for k in LENGTHS[kind]])
    A.values = rng.integers(1, 9, A.nnz).astype(np.float64)
    eye = columns(n, [np.array([j]) for j in range(n)])  # the product's columns are A's
    eye.values = np.ones(n)
    m = trained_model(G.rmat(10, 8, seed=42))[0]
    m.use()
    got = local.spgemm(A, eye, sr=sr, dtype=dtype, sizing="learned").to_csc()
    m.close()
    assert np.array_equal(got[0], A.colptr) and np.array_equal(got[1], A.rowidx)
    assert np.array_equal(got[2], A.values.astype(dtype))
