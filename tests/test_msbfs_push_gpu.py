"""Levels of multi-source BFS where few edges are active: hubs whose edges all
blocks share, vertices whose edges a block flattens, frontiers wider than the
grid, and blocks that find more new vertices than they hold back, in levels of
either kind."""
import numpy as np
import pytest

from combblas_gb300 import bfs as B
from test_msbfs_bits_gpu import edges

pytestmark = pytest.mark.gpu


def graph(name, rng):
    if name == "hubs":  # three of 5000 neighbours, in a graph large enough that their level is pushed
        n = 60000
        u, v = rng.integers(0, n, 4 * n), rng.integers(0, n, 4 * n)
        hub = np.repeat([7, 8, 59999], 5000)
        return n, np.concatenate([u, hub]), np.concatenate([v, rng.integers(0, n, 15000)])
    if name == "wide":  # 1024 vertices a row, 900 rows: frontiers of any width up to a row, few neighbours
        n = 1024 * 300
        i = np.arange(n)
        right, down = i[i % 1024 != 1023], i[i < n - 1024]
        far = rng.integers(0, n, 3000)
        return n, np.concatenate([right, down, far]), np.concatenate([right + 1, down + 1024, np.sort(far)])
    if name == "stars":  # 2040 new vertices from one vertex, just no hub; 2049 from a hub
        k = np.array([2040, 2049] * 20)
        at = np.concatenate([[0], np.cumsum(k + 1)[:-1]])
        leaf = np.concatenate([a + 1 + np.arange(c) for a, c in zip(at, k)])
        return int(k.sum() + len(k)), np.concatenate([np.repeat(at, k), at[:-1]]), np.concatenate([leaf, at[1:]])
    if name == "many hubs":  # 300 of 2100 leaves in one frontier, beside a part that keeps the level thin
        hub = 1 + np.arange(300) * 2101
        leaf = (hub[:, None] + 1 + np.arange(2100)[None, :]).reshape(-1)
        n = 1 + 300 * 2101
        u = n + np.arange(1 << 20)
        return n + (1 << 20) + 3, np.concatenate([np.zeros(300, np.int64), np.repeat(hub, 2100), u, u, u]), \
            np.concatenate([hub, leaf, u + 1, u + 2, u + 3])
    n = 1300000  # "one level": more new vertices than the grid has threads, several rounds a block
    return n, np.zeros(n - 1, np.int64), np.arange(1, n)


@pytest.mark.parametrize("name,nroots", [("hubs", 1), ("hubs", 70), ("hubs", 300), ("wide", 1), ("wide", 40),
                                         ("wide", 130), ("wide", 300), ("stars", 1), ("stars", 100), ("stars", 300),
                                         ("many hubs", 1), ("many hubs", 3), ("one level", 1)])
def test_thin_levels_match_the_oracle(gpu_ctx, oracle_lib, name, nroots):
    rng = np.random.default_rng(nroots)
    n, u, v = graph(name, rng)
    A = edges(n, u, v)
    roots = rng.integers(0, n, nroots)
    if name == "many hubs":
        roots %= 600000  # not in the part beside
    roots[0] = {"hubs": 7, "one level": 0, "many hubs": 0}.get(name, roots[0])
    ref, levels = oracle_lib.port_msbfs(A, roots)
    deg = np.diff(A.colptr)
    g = B.Graph(A)
    for _ in range(2):
        par, st = B.msbfs(g, roots)
        assert np.array_equal(par, ref)
        assert st.levels == levels and st.reached == int((ref >= 0).sum())
        assert st.edges == int(((ref >= 0) * deg[None, :]).sum()) // 2
    g.close()
