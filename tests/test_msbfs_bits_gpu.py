"""Multi-source BFS at the edges of its one-bit-per-root passes: root counts
around the word sizes and the roots of one pass, vertices with more neighbours
than a chunk, graphs that stay with push levels, and patterns that are not
symmetric (which expand pairs instead)."""
import numpy as np
import pytest

from combblas_gb300 import bfs as B
from combblas_gb300 import generators as G

pytestmark = pytest.mark.gpu


def edges(n, u, v, both=True):
    u, v = np.asarray(u, np.int64), np.asarray(v, np.int64)
    return G.csc_from_coo(n, n, np.concatenate([u, v]) if both else u, np.concatenate([v, u]) if both else v)


def graph(name):
    rng = np.random.default_rng(4)
    if name == "rmat":
        return G.rmat(10, 8, seed=3, values=None)
    if name == "path":  # one or two active vertices a level: push only, many levels
        return edges(700, np.arange(699), np.arange(1, 700))
    if name == "star":  # one vertex with 3000 neighbours (chunks), loops included
        return edges(3001, np.concatenate([np.zeros(3000), [5]]), np.concatenate([np.arange(1, 3001), [5]]))
    if name == "directed":
        return edges(600, rng.integers(0, 600, 3000), rng.integers(0, 600, 3000), both=False)
    # symmetric apart from one entry, and as many entries above as below the diagonal
    M = edges(400, np.arange(399), np.arange(1, 400))
    return edges(400, np.concatenate([M.rowidx, [7, 300]]), np.concatenate([M.col_ids(), [90, 20]]), both=False)


@pytest.mark.parametrize("name,nroots", [("rmat", k) for k in (1, 2, 64, 65, 128, 129, 256, 257, 512, 513, 1100)] +
                         [("path", 3), ("path", 70), ("star", 130), ("star", 1), ("directed", 70), ("nearly", 9)])
def test_msbfs_matches_the_oracle(gpu_ctx, oracle_lib, name, nroots):
    A = graph(name)
    roots = np.random.default_rng(nroots).integers(0, A.ncol, nroots)
    g = B.Graph(A)
    ref, levels = oracle_lib.port_msbfs(A, roots)
    deg = np.diff(A.colptr)
    for _ in range(2):  # state is left as it was found
        par, st = B.msbfs(g, roots)
        assert np.array_equal(par, ref)
        assert st.levels == levels and st.reached == int((ref >= 0).sum())
        assert st.edges == int(((ref >= 0) * deg[None, :]).sum()) // 2
    g.close()


def test_msbfs_root_counts_change_between_calls(gpu_ctx, oracle_lib):
    A = graph("rmat")
    g = B.Graph(A)
    for k in (70, 3, 600, 130):
        roots = np.random.default_rng(k).integers(0, A.ncol, k)
        assert np.array_equal(B.msbfs(g, roots)[0], oracle_lib.port_msbfs(A, roots)[0])
    g.close()
