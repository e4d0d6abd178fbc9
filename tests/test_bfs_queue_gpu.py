"""BFS levels in which a block finds more vertices than its queue holds: a level
of 6 million leaves, found bottom-up and, for the pairs of a multi-source
traversal on a pattern that is not symmetric, by expansion; and bottom-up levels
whose vertices find their parent at any of their first neighbours."""
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


@pytest.mark.parametrize("policy", ["bottomup", "auto"])
def test_parent_at_any_neighbour(gpu_ctx, oracle_lib, policy):
    """Vertex d * 25 + j has d neighbours of which the j-th and those after it are in the frontier."""
    base, side = 25 * 25, 60
    far, near = base + np.arange(side), base + side + np.arange(side)  # near: the source's neighbours
    u, v = [np.full(side, base + 2 * side)], [near]
    for d in range(1, 25):
        for j in range(d):
            u.append(np.full(d, d * 25 + j))
            v.append(np.concatenate([far[:j], near[:d - j]]))
    A = edges(base + 2 * side + 1, np.concatenate(u), np.concatenate(v))
    g = B.Graph(A)
    g.set_policy(policy)
    par, lev, _ = B.bfs(g, base + 2 * side)
    epar, elev, _ = oracle_lib.port_bfs(A, base + 2 * side)
    assert np.array_equal(par, epar) and np.array_equal(lev, elev)
    g.close()
