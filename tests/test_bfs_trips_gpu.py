"""Traversals whose levels change direction, run level by level and as one graph
(where a bottom-up level may follow a top-down one in the same trip): vertex
counts around the words of the bitmaps, a chain, stars, a graph with loops and
isolated vertices, and more frontier tiles than one pass sums."""
import numpy as np
import pytest

from combblas_gb300 import bfs as B
from combblas_gb300 import generators as G

pytestmark = pytest.mark.gpu


def symmetric(n, edges):
    e = np.array(sorted({(a, b) for a, b in edges} | {(b, a) for a, b in edges}), np.int64).reshape(-1, 2)
    cp = np.zeros(n + 1, np.int64)
    np.add.at(cp, e[:, 0] + 1, 1)
    return G.CSC(n, n, np.cumsum(cp), e[:, 1].copy(), None)


def graph(kind, n):
    if kind == "chain":
        return symmetric(n, [(i, i + 1) for i in range(n - 1)])
    if kind == "star":
        return symmetric(n, [(n // 2, i) for i in range(n)])
    if kind == "two hubs":
        return symmetric(n, [(0, i) for i in range(1, n // 2)] + [(1, n - 1)] +
                         [(n - 1, i) for i in range(n // 2, n - 1)])
    rng = np.random.default_rng(n)  # loops, isolated vertices
    return symmetric(n, [tuple(x) for x in rng.integers(0, n, (2 * n, 2)) if x[0] % 7])


@pytest.mark.parametrize("policy", ["topdown", "bottomup", "auto"])
@pytest.mark.parametrize("n", [2, 31, 32, 33, 255, 257, 1025])
@pytest.mark.parametrize("kind", ["chain", "star", "two hubs", "random"])
def test_against_the_oracle(gpu_ctx, oracle_lib, kind, n, policy):
    A = graph(kind, n)
    g = B.Graph(A)
    g.set_policy(policy)
    for s in {0, n // 2, n - 1}:
        par, lev, st = B.bfs(g, int(s))
        epar, elev, eit = oracle_lib.port_bfs(A, int(s))
        assert np.array_equal(par, epar) and np.array_equal(lev, elev) and st.iterations == eit


def test_frontier_of_many_tiles(gpu_ctx):
    n = 2048 * 2048 + 4097  # the frontier of the second level has more tiles than are summed by every block
    ends = np.arange(1, n)
    cp = np.concatenate([[0, n - 1], n - 1 + np.arange(1, n)]).astype(np.int64)
    A = G.CSC(n, n, cp, np.concatenate([ends, np.zeros(n - 1, np.int64)]), None)
    g = B.Graph(A)
    for policy in ("topdown", "auto"):
        g.set_policy(policy)
        par, lev, st = B.bfs(g, 0)
        assert lev[0] == 0 and par[0] == 1 and (lev[1:] == 1).all() and (par[1:] == 0).all()
