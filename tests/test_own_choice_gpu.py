"""Which ordered columns the kernel takes whose warps own row ranges, told by the
launches that build its tables: those with long segments throughout, not those
whose products come from a few, and not where one column is most of the work.
The fold's bits are the oracle's on either side."""
import numpy as np
import pytest

from combblas_gb300 import _lib as L
from combblas_gb300 import local
from test_exact_visits_gpu import columns, pick

pytestmark = pytest.mark.gpu


def product(oracle, lens, entries, m, dtype, **kw):
    """Launches of A * B, A with columns of `lens` entries, B with columns of `entries`."""
    rng = np.random.default_rng(len(entries))
    n = len(lens)
    A = columns(m, [pick(rng, 0, m, k) for k in lens])
    B = columns(n, [pick(rng, 0, n, k) for k in entries])
    for M in (A, B):
        M.values = rng.standard_normal(M.nnz).astype(dtype)
    before = L.lib().gbc_launch_count()
    R = local.spgemm(A, B, dtype=dtype, fold="ordered", **kw)
    count = L.lib().gbc_launch_count() - before
    got, exp = R.to_csc(), oracle.port_spgemm(A, B, 1 if dtype == np.float32 else 0)
    for g, e in zip(got, exp):
        assert np.array_equal(g, e)
    return count


@pytest.mark.parametrize("dtype,long,short", [(np.float32, 1000, 100), (np.float64, 2500, 200)])
def test_segments(gpu_ctx, oracle_lib, dtype, long, short):
    kw = dict(m=20000, dtype=dtype, tiny_limit=0, small_limit=0)
    entries = [60, 1, 31, 32, 33, 50]
    base = product(oracle_lib, [short] * 60, entries, **kw)
    assert product(oracle_lib, [long] * 60, entries, **kw) >= base + 4
    # the mean is as long, from a third of the segments
    assert product(oracle_lib, [3 * long if k % 3 == 0 else 16 for k in range(60)], [60, 60, 60], **kw) < base + 4


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_one_column_among_many(gpu_ctx, oracle_lib, dtype):
    kw = dict(m=3000, dtype=dtype)
    alike = [9] * 2600
    many = product(oracle_lib, [900] * 200, alike, **kw)
    assert product(oracle_lib, [900] * 200, alike + [200], **kw) <= many - 4
