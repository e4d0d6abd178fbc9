"""The warp kernels' columns at the edges of their sorts: product counts around
the register sorts' sizes (256, 512, 1024), the shared-memory sort above
them and for rows from 2^20 on, runs of equal rows across lanes, bit for bit
against the oracle."""
import numpy as np
import pytest

from combblas_gb300 import local
from test_exact_visits_gpu import columns, pick
from test_spgemm_gpu import SR_NAME, assert_same
from test_oracle import typed

pytestmark = pytest.mark.gpu

COUNTS = [1, 2, 31, 32, 33, 63, 65, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 2047, 2048, 2049, 4095, 4096]


@pytest.mark.parametrize("sr", [0, 1, 3, 5])
@pytest.mark.parametrize("m,spread", [(5000, 5000), (5000, 40), ((1 << 20) + 9, (1 << 20) + 9)])
def test_column_sizes(gpu_ctx, oracle_lib, m, spread, sr):
    """Column c of A*B has COUNTS[c] products, over few rows (long runs) or many."""
    O = oracle_lib
    rng = np.random.default_rng(sr)
    acols, bcols = [], []
    for n in COUNTS:
        mine = []
        while n > 0:
            k = int(min(n, rng.integers(1, min(spread, 300) + 1)))
            mine.append(len(acols))
            acols.append(pick(rng, m - spread, m, k))
            n -= k
        bcols.append(np.array(mine))
    A, B = columns(m, acols), columns(len(acols), bcols)
    A.values, B.values = np.ones(A.nnz), np.ones(B.nnz)
    A, B = typed(A.with_values(None), sr, 3, O), typed(B.with_values(None), sr, 4, O)
    name, dt = SR_NAME[sr]
    for fold in ("ordered", "exact") if sr == 0 else ("ordered",):
        got = local.spgemm(A, B, sr=name, dtype=dt, fold=fold, tiny_limit=256, small_limit=4096).to_csc()
        exp = O.port_spgemm(A, B, sr, fold=fold)
        assert_same(*got, *exp, sr, True, fold)
