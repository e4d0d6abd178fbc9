"""Columns of 257 to 1024 products around the number up to which the block
kernels take them instead of the warp kernels (8 per resident block, two blocks
on each multiprocessor), alone and beside small and big columns.  And dense fp32
columns around the number from which warps own their rows (16 on each
multiprocessor)."""
import numpy as np
import pytest
import torch

from combblas_gb300 import local
from test_exact_visits_gpu import columns, pick
from test_oracle import typed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sr", [0, 3])
@pytest.mark.parametrize("others", [0, 40])
@pytest.mark.parametrize("extra", [None, 0, 1])
def test_around_the_limit(gpu_ctx, oracle_lib, extra, others, sr):
    limit = 8 * 2 * torch.cuda.get_device_properties(0).multi_processor_count
    n = 3 if extra is None else limit + extra
    rng = np.random.default_rng(n)
    A = columns(6000, [pick(rng, 0, 6000, 60) for _ in range(400)])
    B = columns(400, [pick(rng, 0, 400, 5 + j % 12) for j in range(n)] + [pick(rng, 0, 400, 1 + j * 8)
                                                                          for j in range(others)])
    for M in (A, B):
        M.values = rng.integers(-9, 10, M.nnz) * 0.25
    name = "plustimes" if sr == 0 else "minplus"
    got = local.spgemm(A, B, sr=name, fold="exact").to_csc()
    exp = oracle_lib.port_spgemm(A, B, sr, fold="exact" if sr == 0 else "ordered")
    for g, e in zip(got, exp):
        assert np.array_equal(g, e)


@pytest.mark.parametrize("extra", [-2000, 0, 1])
def test_dense_columns_around_the_limit(gpu_ctx, oracle_lib, extra):
    n = 16 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    rng = np.random.default_rng(n)
    A = columns(40, [np.arange(40) for _ in range(130)])
    B = columns(130, [pick(rng, 0, 130, 110 + j % 21) for j in range(n)] + [pick(rng, 0, 130, 20)])
    for M in (A, B):
        M.values = rng.random(M.nnz)
    A, B = typed(A, 1, 3, oracle_lib), typed(B, 1, 4, oracle_lib)
    got = local.spgemm(A, B, dtype=np.float32).to_csc()
    exp = oracle_lib.port_spgemm(A, B, 1)
    for g, e in zip(got, exp):
        assert np.array_equal(g, np.asarray(e))
