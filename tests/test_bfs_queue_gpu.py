"""BFS levels in which a block finds more vertices than its queue holds: a level
of 6 million leaves, found bottom-up and, for the pairs of a multi-source
traversal on a pattern that is not symmetric, by expansion."""
import numpy as np
import pytest

from combblas_gb300 import bfs as B
from test_msbfs_bits_gpu import edges

pytestmark = pytest.mark.gpu


def test_bottom_up_level_of_many_leaves(gpu_ctx):
    n = 6000000
    g = B.Graph(edges(n, np.zeros(n - 1, np.int64), np.arange(1, n)))
    g.set_policy("bottomup")
    par, lev, st = B.bfs(g, 0)
    assert (par[1:] == 0).all() and (lev[1:] == 1).all() and lev[0] == 0
    assert st.reached == n
    g.close()


def test_pairs_of_many_leaves(gpu_ctx):
    n = 1500000
    g = B.Graph(edges(n, np.arange(1, n), np.zeros(n - 1, np.int64), both=False))  # column 0 holds every row
    par, st = B.msbfs(g, [0, 5, 0, 0])
    assert st.reached == 3 * n + 1
    for r in (0, 2, 3):
        assert (par[r][1:] == 0).all() and par[r][0] == 0
    assert par[1][5] == 5 and (np.delete(par[1], 5) == -1).all()
    g.close()
