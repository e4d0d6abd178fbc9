"""Batched results written to device buffers by one kernel per product, in each
width of value, against the host copies and single products: empty products,
empty columns, an output of one entry.  And squares of one host matrix, whose
arrays are uploaded once."""
import numpy as np
import pytest

from combblas_gb300 import batch, local
from combblas_gb300 import generators as G

pytestmark = pytest.mark.gpu


def matrices():
    one = G.CSC(7, 7, np.array([0, 0, 0, 0, 1, 1, 1, 1]), np.array([3]), np.ones(1))
    none = G.CSC(5, 5, np.zeros(6, np.int64), np.zeros(0, np.int64), np.zeros(0))
    return [none, G.random_sparse(300, 300, 0.02, seed=2), one, G.rmat(9, 8, seed=3)]


@pytest.mark.parametrize("sr,dtype", [("plustimes", np.float64), ("plustimes", np.float32), ("bool", np.bool_)])
def test_device_results_are_the_host_results(gpu_ctx, sr, dtype):
    Ms = matrices()
    b = batch.Batch(Ms, Ms, sr=sr, dtype=dtype)
    b.run()
    for p, M in enumerate(Ms):
        cp, ir, num = b.result(p)
        D = b.result_device(p, M.nrow, M.ncol)
        for host, dev in ((cp, D.cp), (ir, D.ir), (num, D.num)):
            assert np.array_equal(host, dev.cpu().numpy())
        if M.nnz == 0:
            continue
        R = local.spgemm(M, M, sr=sr, dtype=dtype)
        assert R.stats.flops == b.info(p)[2]
        for host, alone in zip((cp, ir, num), R.to_csc()):
            assert np.array_equal(host, alone)
    b.close()


def test_square_and_product_of_copies_agree(gpu_ctx):
    A = G.rmat(10, 6, seed=5)
    B = G.CSC(A.nrow, A.ncol, A.colptr.copy(), A.rowidx.copy(), A.values.copy())
    for x, y in zip(local.spgemm(A, A).to_csc(), local.spgemm(A, B).to_csc()):
        assert np.array_equal(x, y)
