"""Dense-vector SpMV at the edges of its tiles (8 entries a thread, 1024 a
block): rows that end on a group, warp or tile boundary, rows across one and
several tiles, rows of single entries, empty rows between, a last ragged group."""
import numpy as np
import pytest

from combblas_gb300 import generators as G
from combblas_gb300 import local
from test_spmv_gpu import NAME, check, vectors
from test_oracle import typed

pytestmark = pytest.mark.gpu

ROWS = {
    "one entry": [1],
    "groups": [8, 8, 0, 7, 1, 0, 0, 9, 15, 16, 17, 31, 32, 256, 255, 257],
    "single": [1] * 5000,
    "tiles": [1024, 0, 1023, 1, 1025, 3, 2048, 2],
    "across": [10, 20000, 5, 0, 13000, 1024, 1],
    "one row": [9001],
}


@pytest.mark.parametrize("sr", [0, 1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("name", list(ROWS))
def test_spmv_tile_edges(gpu_ctx, oracle_lib, name, sr):
    O = oracle_lib
    rng = np.random.default_rng(sr)
    lens = np.array(ROWS[name])
    m, n = len(lens), 20003
    rows = np.repeat(np.arange(m), lens)
    cols = np.concatenate([rng.choice(n, k, replace=False) for k in lens])
    A = G.csc_from_coo(m, n, rows, cols)
    A.values = np.ones(A.nnz)
    A = typed(A.with_values(None), sr, 5, O)
    x, y0 = vectors(sr, m, n, O, 6)
    plan = local.SpMVPlan(A, O.SR_DTYPE[sr])
    y = plan.multiply(x, np.array(y0), NAME[sr])
    check(sr, y, O.port_spmv(A, x, y0, sr), O)
    assert np.array_equal(y, plan.multiply(x, np.array(y0), NAME[sr]))
    plan.close()
