"""The rules by which the host sizes what kernels write, compiled by the host
compiler, against counts taken from matrices."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="session")
def rule(tmp_path_factory):
    """rule(expression): its value in a program that includes the rules."""
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("rules")

    def value(expr):
        src, exe = d / "r.cpp", d / "r"
        src.write_text('#include <cstdio>\n#include "size_rules.cuh"\nusing namespace gbc;\n'
                       f'int main() {{ std::printf("%lld\\n", (long long)({expr})); }}\n')
        subprocess.run([cxx, "-std=c++17", "-I", os.path.join(ROOT, "combblas_gb300", "csrc"), str(src), "-o", str(exe)],
                       check=True)
        return int(subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout)

    return value


def tile_list_entries(rows, cols, ncol, tile=4096):
    """Entries of all columns' tile lists: touched row tiles, and an end marker each."""
    return len(set(zip(cols.tolist(), (rows // tile).tolist()))) + ncol


@pytest.mark.parametrize("name", ["identity", "hypersparse", "one tile an entry", "empty", "dense columns"])
def test_tile_lists_fit_their_arrays(rule, name):
    rng = np.random.default_rng(2)
    if name == "identity":
        n = 5000
        rows = cols = np.arange(n)
    elif name == "hypersparse":
        n = 100000
        cols = np.sort(rng.choice(n, 5000, replace=False))
        rows = rng.integers(0, n, 5000)
    elif name == "one tile an entry":
        n = 30
        rows, cols = np.tile(np.arange(256) * 4096, n), np.repeat(np.arange(n), 256)
    elif name == "empty":
        n, rows, cols = 777, np.zeros(0, np.int64), np.zeros(0, np.int64)
    else:
        n = 2
        rows, cols = np.tile(np.arange(4000), n), np.repeat(np.arange(n), 4000)
    assert tile_list_entries(rows, cols, n) <= rule(f"ktl_room({len(rows)}, {n})")


@pytest.mark.parametrize("step", [4, 32, 64, 128])
def test_positions_of_an_accepted_graph_do_not_wrap(rule, step):
    """A 32-bit position that walks the last entries in steps ends past them, for the most entries accepted."""
    lo, hi = 0, (1 << 32) - 1  # most entries that a graph may have at all
    assert not rule(f"mb_positions_fit({hi})")
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (mid, hi) if rule(f"mb_positions_fit({mid})") else (lo, mid)
    nnz = lo
    for first in range(nnz - step, nnz):
        assert (first + step) & 0xFFFFFFFF >= nnz
