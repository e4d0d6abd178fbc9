"""What the framework's speed is measured on: its node-local sparse kernels,
each through the public Python entry points, on seeded synthetic matrices.

Matrices are R-MAT graphs (initiator 0.57 / 0.19 / 0.19 / 0.05, duplicates
merged, self-loops dropped, symmetrised, also cut to vertex counts that are no
power of two), planted-cluster matrices for MCL, and 27-point stencils with
their 2x2x2 aggregation.  They are made on the GPU.  A case fixes its pattern up to a
relabelling; the seed gives the relabelling of the vertices (inside blocks of
64, so that the skew of an R-MAT stays), the values, vectors and roots.  Sizes
of outputs are then the same for every seed.

``listed()`` names the cases, ``draw()`` gives more of the same ranges,
``prepare()`` makes what a program holds before the call, ``run()`` is one
pass, ``exact()`` the values in 64 bits by plain torch, ``work()`` the bytes
and operations that a pass cannot do without.
"""
import math
import random

import numpy as np
import torch

from combblas_gb300 import batch as batching
from combblas_gb300 import bfs, local, mcl, sizing

DEV = "cuda"
TORCH = {"f64": torch.float64, "f32": torch.float32, "i64": torch.int64, "bool": torch.bool}
NUMPY = {"f64": np.float64, "f32": np.float32, "i64": np.int64, "bool": np.bool_}


def listed():
    return [
        # the smallest product, host arrays in and out, as a caller with many small blocks meets it:
        # launches, copies and synchronisations
        {"name": "spgemm tiny host", "kind": "spgemm", "n": 600, "ef": 6, "sr": "plustimes", "dtype": "f64",
         "sizing": "exact", "where": "host", "form": "dcsc"},
        # an ordinary whole product, the R-MAT scale-14 configuration
        {"name": "spgemm 2^14 f64", "kind": "spgemm", "n": 1 << 14, "ef": 8, "sr": "plustimes", "dtype": "f64",
         "sizing": "exact", "where": "device", "form": "csc"},
        # a large whole product sized by the trained model instead of the symbolic pass
        {"name": "spgemm 2^16 learned", "kind": "spgemm", "n": 1 << 16, "ef": 16, "sr": "plustimes", "dtype": "f64",
         "sizing": "learned", "where": "device", "form": "csc"},
        # a shortest-path step: another semiring, DCSC operands, a vertex count that is no power of two
        {"name": "spgemm 30011 min-plus", "kind": "spgemm", "n": 30011, "ef": 12, "sr": "minplus", "dtype": "f64",
         "sizing": "exact", "where": "device", "form": "dcsc"},
        # the headline: scale 20 in column phases (the entry point itself keeps only checksums of the product)
        {"name": "phased 2^20 f64", "kind": "phased", "n": 1 << 20, "ef": 16, "budget": 3 << 30},
        # many uneven products replayed as one graph: R-MAT squares and stencil-times-aggregation products
        {"name": "batch 16", "kind": "batch", "rmat": 8, "stencil": 8, "lo": 1 << 9, "hi": 1 << 14, "side": 40},
        # one MCL expansion with prune and top-100 selection, the clustering configuration's size
        {"name": "mcl expand 2^20", "kind": "mcl_expand", "n": 1 << 20, "cluster": 1024, "select": 100,
         "sizing": "exact"},
        # the whole MCL loop to convergence
        {"name": "mcl loop 20000", "kind": "mcl_loop", "n": 20000, "cluster": 200, "select": 1100},
        # one traversal of the scale-20 graph, direction chosen per level
        {"name": "bfs 2^20", "kind": "bfs", "n": 1 << 20, "ef": 16, "policy": "auto"},
        # many traversals at once
        {"name": "msbfs 2^20 x 256", "kind": "msbfs", "n": 1 << 20, "ef": 16, "roots": 256},
        # one step of an iteration on a dense vector
        {"name": "spmv 2^20 f64", "kind": "spmv", "n": 1 << 20, "ef": 16, "sr": "plustimes", "dtype": "f64"},
        # one sparse-vector product, vectors on the host
        {"name": "spmspv 2^18 f64", "kind": "spmspv", "n": 1 << 18, "ef": 16, "entries": 2000, "sr": "plustimes",
         "dtype": "f64"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["spgemm"] * 6 + ["phased", "batch", "mcl_expand", "mcl_expand", "mcl_loop", "bfs", "bfs",
                                        "msbfs", "msbfs", "spmv", "spmv", "spmspv", "spmspv"])
    ef = rng.randint(4, 16)
    if kind == "spgemm":
        sr, dtype = rng.choice([("plustimes", "f64")] * 4 + [("plustimes", "f32"), ("plustimes", "i64"),
                                                              ("minplus", "f64"), ("minplus", "i64"),
                                                              ("select2ndmin", "i64"), ("bool", "bool")])
        host = rng.random() < 0.25
        n = _log(rng, 300, 4000) if host else _log(rng, 1000, 1 << 16)
        size = "learned" if not host and n > 8000 and rng.random() < 0.3 else "exact"
        return {"kind": kind, "n": n, "ef": ef, "sr": sr, "dtype": dtype, "sizing": size,
                "where": "host" if host else "device", "form": rng.choice(["csc", "dcsc"])}
    if kind == "phased":
        return {"kind": kind, "n": _log(rng, 1 << 16, 1 << 19), "ef": ef, "budget": _log(rng, 1 << 26, 3 << 30)}
    if kind == "batch":
        return {"kind": kind, "rmat": rng.randint(2, 10), "stencil": rng.randint(2, 10), "lo": 1 << 8,
                "hi": _log(rng, 1 << 12, 1 << 14), "side": 2 * rng.randint(10, 20)}
    if kind == "mcl_expand":
        cluster = _log(rng, 100, 1024)
        return {"kind": kind, "n": cluster * max(2, _log(rng, 1 << 14, 1 << 20) // cluster), "cluster": cluster,
                "select": rng.randint(30, 300), "sizing": rng.choice(["exact", "exact", "learned"])}
    if kind == "mcl_loop":
        cluster = _log(rng, 60, 400)
        return {"kind": kind, "n": cluster * max(2, _log(rng, 4000, 40000) // cluster), "cluster": cluster,
                "select": 1100}
    if kind == "bfs":
        return {"kind": kind, "n": _log(rng, 1 << 12, 1 << 20), "ef": ef,
                "policy": rng.choice(["auto", "auto", "topdown", "bottomup"])}
    if kind == "msbfs":
        n = _log(rng, 1 << 12, 1 << 20)
        return {"kind": kind, "n": n, "ef": ef, "roots": _log(rng, 3, min(2000, (1 << 28) // n))}
    if kind == "spmv":
        sr, dtype = rng.choice([("plustimes", "f64"), ("plustimes", "f64"), ("plustimes", "f32"), ("minplus", "f64"),
                                ("plustimes", "i64"), ("select2ndmin", "i64")])
        return {"kind": kind, "n": _log(rng, 1 << 12, 1 << 20), "ef": ef, "sr": sr, "dtype": dtype}
    sr, dtype = rng.choice([("plustimes", "f64"), ("plustimes", "f32"), ("select2ndmin", "none"),
                            ("select2nd", "none"), ("selectmax", "none")])
    n = _log(rng, 1 << 12, 1 << 18)
    return {"kind": "spmspv", "n": n, "ef": ef, "entries": _log(rng, 1, n // 8), "sr": sr, "dtype": dtype}


# ------------------------------------------------------------------ matrices
class Csc:
    """Column-compressed arrays on the GPU (int64 cp, ir; values or None)."""

    def __init__(self, nrow, ncol, cp, ir, val=None):
        self.nrow, self.ncol, self.cp, self.ir, self.val = nrow, ncol, cp, ir, val

    @property
    def nnz(self):
        return int(self.ir.numel())

    def cols(self):
        return torch.repeat_interleave(torch.arange(self.ncol, device=DEV), self.cp.diff())


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _relabel(n, seed):
    """A permutation of 0..n-1 that shuffles every block of 64."""
    at = torch.div(torch.arange(n, device=DEV), 64, rounding_mode="floor").double()
    return torch.argsort(torch.argsort(at + torch.rand(n, generator=_gen(seed + 31), device=DEV, dtype=torch.float64)))


def _from_keys(key, nrow, ncol):
    """Csc of the distinct keys col * nrow + row."""
    key = torch.unique(key)
    col = torch.div(key, nrow, rounding_mode="floor")
    cp = torch.zeros(ncol + 1, dtype=torch.int64, device=DEV)
    cp[1:] = torch.cumsum(torch.bincount(col, minlength=ncol), 0)
    return Csc(nrow, ncol, cp, key - col * nrow)


def _rmat(n, ef, seed):
    g = _gen(n * 64 + ef)
    scale = max(1, (n - 1).bit_length())
    u = torch.zeros(ef * n, dtype=torch.int64, device=DEV)
    v = torch.zeros_like(u)
    for level in range(scale):
        r = torch.rand(ef * n, generator=g, device=DEV)
        u |= (r >= 0.76).long() << level
        v |= (((r >= 0.57) & (r < 0.76)) | (r >= 0.95)).long() << level
    keep = (u != v) & (u < n) & (v < n)
    perm = _relabel(n, seed)
    u, v = perm[u[keep]], perm[v[keep]]
    return _from_keys(torch.cat([v * n + u, u * n + v]), n, n)


def _fill(M, dtype, seed):
    """Values in (0, 1], small whole numbers or ones, by type."""
    g = _gen(seed + 7919)
    if dtype in ("f64", "f32"):
        M.val = 1.0 - torch.rand(M.nnz, generator=g, device=DEV, dtype=TORCH[dtype])
    elif dtype == "i64":
        M.val = torch.randint(1, 100, (M.nnz,), generator=g, device=DEV)
    elif dtype == "bool":
        M.val = torch.ones(M.nnz, dtype=torch.bool, device=DEV)
    return M


def _planted(n, cluster, seed):
    """Column-stochastic fp32: about 24 entries of a column inside its cluster, 6 outside, and the diagonal."""
    g = _gen(n * 64 + 1)
    perm = _relabel(n, seed)
    col = torch.arange(n, device=DEV)
    cin = torch.repeat_interleave(col, torch.poisson(torch.full((n,), 24.0, device=DEV), generator=g).long())
    cout = torch.repeat_interleave(col, torch.poisson(torch.full((n,), 6.0, device=DEV), generator=g).long())
    rin = torch.div(cin, cluster, rounding_mode="floor") * cluster + torch.randint(
        0, cluster, (cin.numel(),), generator=g, device=DEV)
    rout = torch.randint(0, n, (cout.numel(),), generator=g, device=DEV)
    M = _from_keys(torch.cat([perm[cin] * n + perm[rin], perm[cout] * n + perm[rout], col * n + col]), n, n)
    v = 1.0 - torch.rand(M.nnz, generator=_gen(seed), device=DEV, dtype=torch.float64)
    c = M.cols()
    M.val = (v / torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, c, v)[c]).float()
    return M


def _stencil(side, seed):
    """27-point stencil on side^3 points: 26 on the diagonal scaled per point, -1 elsewhere."""
    n = side ** 3
    i = torch.arange(n, device=DEV)
    x, y, z = i % side, torch.div(i, side, rounding_mode="floor") % side, torch.div(i, side * side, rounding_mode="floor")
    keys = []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                a, b, c = x + dx, y + dy, z + dz
                ok = (a >= 0) & (a < side) & (b >= 0) & (b < side) & (c >= 0) & (c < side)
                keys.append((i * n + (c * side + b) * side + a)[ok])
    M = _from_keys(torch.cat(keys), n, n)
    M.val = torch.full((M.nnz,), -1.0, dtype=torch.float64, device=DEV)
    on = M.cols() == M.ir
    M.val[on] = 26.0 * (1.0 + torch.rand(n, generator=_gen(seed), device=DEV, dtype=torch.float64))
    return M


def _aggregate(side):
    """Prolongation of the 2x2x2 aggregation (side^3 by (side/2)^3, ones)."""
    n, h = side ** 3, side // 2
    i = torch.arange(n, device=DEV)
    x, y, z = i % side, torch.div(i, side, rounding_mode="floor") % side, torch.div(i, side * side, rounding_mode="floor")
    agg = (torch.div(z, 2, rounding_mode="floor") * h + torch.div(y, 2, rounding_mode="floor")) * h + torch.div(
        x, 2, rounding_mode="floor")
    M = _from_keys(agg * n + i, n, h ** 3)
    M.val = torch.ones(M.nnz, dtype=torch.float64, device=DEV)
    return M


def _handed(M, form="csc", where="device"):
    """The matrix as the caller holds it: a DeviceMatrix, or host arrays."""
    cp, jc = M.cp, None
    if form == "dcsc":
        cnt = M.cp.diff()
        jc = torch.nonzero(cnt).reshape(-1)
        cp = torch.cat([M.cp[:1], torch.cumsum(cnt[jc], 0)])
    if where == "device":
        torch.cuda.synchronize()
        return local.DeviceMatrix(M.nrow, M.ncol, cp, M.ir, M.val, jc)
    h = lambda t: t.cpu().numpy()  # noqa: E731
    if jc is None:  # host CSC as DCSC arrays over every column
        jc = torch.arange(M.ncol, device=DEV)
    return local.DCSC(M.nrow, M.ncol, h(cp), h(jc), h(M.ir), h(M.val))


class _Array:
    """A device array of a result, seen without a copy; it keeps the result alive."""

    def __init__(self, owner, ptr, n, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr or 0, False), "version": 2}


def _result(R):
    cp, jc, ir, num = R.device_ptrs()
    d = np.dtype(R.dtype)
    see = lambda p, n, t: torch.as_tensor(_Array(R, p, n, t), device=DEV)  # noqa: E731
    return {"cp": see(cp, R.nzc + 1, "<i8"), "jc": see(jc, R.nzc, "<i8"), "ir": see(ir, R.nnz, "<i8"),
            "num": see(num, R.nnz, "|b1" if d.kind == "b" else d.str)}


# -------------------------------------------------------------------- inputs
def _batch_inputs(case, seed):
    rng = random.Random(case["hi"])
    pairs = []
    for k in range(case["rmat"]):
        A = _fill(_rmat(_log(rng, case["lo"], case["hi"]), rng.randint(4, 16), seed * 64 + k), "f64", seed * 64 + k)
        pairs.append((A, A))
    for k in range(case["stencil"]):
        side = 2 * rng.randint(6, case["side"] // 2)
        pairs.append((_stencil(side, seed * 64 + k), _aggregate(side)))
    return pairs


def _inputs(case, seed):
    made = _make(case, seed)
    torch.cuda.synchronize()  # the library's stream is not the one that made them
    return made


def _make(case, seed):
    kind = case["kind"]
    if kind == "spgemm":
        return _fill(_rmat(case["n"], case["ef"], seed), case["dtype"], seed)
    if kind == "phased":
        return _fill(_rmat(case["n"], case["ef"], seed), "f64", seed)
    if kind == "batch":
        return _batch_inputs(case, seed)
    if kind in ("mcl_expand", "mcl_loop"):
        return _planted(case["n"], case["cluster"], seed)
    M = _rmat(case["n"], case["ef"], seed)
    g = _gen(seed + 104729)
    has = torch.nonzero(M.cp.diff()).reshape(-1)
    if kind in ("bfs", "msbfs"):
        at = torch.randint(0, has.numel(), (case.get("roots", 1),), generator=g, device=DEV)
        return M, has[at].cpu().numpy()
    if kind == "spmv":
        _fill(M, case["dtype"], seed)
        if case["dtype"] == "i64":
            x, y = (torch.randint(0, 1000, (M.ncol,), generator=g, device=DEV) for _ in range(2))
        else:
            x, y = (torch.rand(M.ncol, generator=g, device=DEV, dtype=TORCH[case["dtype"]]) for _ in range(2))
        return M, x, y
    if case["dtype"] != "none":
        _fill(M, case["dtype"], seed)
    at = torch.randperm(M.ncol, generator=_gen(case["n"]), device=DEV)[:case["entries"]]
    xi = torch.sort(_relabel(M.ncol, seed)[at])[0]
    if case["dtype"] == "none":
        xv = torch.randint(0, 1 << 40, (xi.numel(),), generator=g, device=DEV)
    else:
        xv = torch.rand(xi.numel(), generator=g, device=DEV, dtype=TORCH[case["dtype"]])
    return M, xi.to(torch.int32).cpu().numpy(), xv.cpu().numpy()


_CONTEXTS = []  # a context outlives every result made in it: they stay, as a program's do


def _trained(D):
    """A context of its own with a sizing model trained on this matrix's counts."""
    ctx = local.Context()
    _CONTEXTS.append(ctx)
    feat, _, nnz = sizing.features(D, D, ctx=ctx)
    keep = np.linspace(0, len(nnz) - 1, min(len(nnz), 20000)).astype(np.int64)
    model = sizing.SizingModel(ctx, seed=1)
    model.fit(feat[keep], nnz[keep], steps=200)
    model.use()
    return ctx, model


class State:
    def __init__(self, **kw):
        self.__dict__.update(kw)


def prepare(case, seed):
    kind = case["kind"]
    M = _inputs(case, seed)
    s = State(case=case, kind=kind, ctx=None, model=None)
    if kind == "spgemm":
        s.A = _handed(M, case["form"], case["where"])
        if case["sizing"] == "learned":
            s.ctx, s.model = _trained(s.A)
    elif kind == "phased":
        s.A = _handed(M)
    elif kind == "batch":
        s.pairs = [(_handed(A), _handed(B)) for A, B in M]
        s.batch = batching.Batch([a for a, _ in s.pairs], [b for _, b in s.pairs])
    elif kind in ("mcl_expand", "mcl_loop"):
        s.A = _handed(M)
        if case.get("sizing") == "learned":
            s.ctx, s.model = _trained(s.A)
        # the caller's own arrays, which hold any selection: up to `select` entries a column and a few ties
        room = case["n"] * case["select"] * 65 // 64 if kind == "mcl_expand" else M.nnz
        s.cp = torch.zeros(case["n"] + 1, dtype=torch.int64, device=DEV)
        s.ir = torch.zeros(room, dtype=torch.int64, device=DEV)
        s.num = torch.zeros(room, dtype=torch.float32, device=DEV)
    elif kind in ("bfs", "msbfs"):
        M, s.roots = M
        s.graph = bfs.Graph(_handed(M))
        if kind == "bfs":
            s.graph.set_policy(case["policy"])
            s.root = int(s.roots[0])
            s.levels = torch.empty(M.ncol, dtype=torch.int64, device=DEV)
        s.parents = torch.empty((len(s.roots), M.ncol), dtype=torch.int64, device=DEV)
    elif kind == "spmv":
        M, s.x, s.y = M
        s.plan = local.SpMVPlan(_handed(M), NUMPY[case["dtype"]])
    else:
        M, s.xi, s.xv = M
        s.plan = bfs.SpMSpVPlan(_handed(M), None if case["dtype"] == "none" else NUMPY[case["dtype"]])
    return s


def _into(s, R):
    """The selection copied into the caller's arrays."""
    R.copy_to(s.cp.data_ptr(), None, s.ir.data_ptr(), s.num.data_ptr(), local.L.GBC_DEVICE)
    return [s.cp, s.ir, s.num]


def run(s):
    c = s.case
    if s.kind == "spgemm":
        R = local.LocalHybridSpGEMM(s.A, s.A, sr=c["sr"], sizing=c["sizing"], ctx=s.ctx)
        return _result(R) if c["where"] == "device" else list(R.to_host())
    if s.kind == "phased":
        st = local.spgemm_phased(s.A, s.A, max_phase_nnz=c["budget"])
        h = st.content_hash
        return {"nnz": st.nnz, "flops": st.flops, "rows": st.row_checksum, "values": st.val_checksum,
                "hash": h - (1 << 64) if h >= 1 << 63 else h}
    if s.kind == "batch":
        s.batch.run()
        out = []
        for p, (A, B) in enumerate(s.pairs):
            C = s.batch.result_device(p, A.nrow, B.ncol)
            out.append([C.cp, C.ir, C.num])
        return out
    if s.kind == "mcl_expand":
        R, _ = mcl.mcl_expand(s.A, 1e-4, c["select"], sizing=c["sizing"], ctx=s.ctx)
        return [R.nnz] + _into(s, R)
    if s.kind == "mcl_loop":
        R, iterations, chaos = mcl.HipMCL(s.A, select=c["select"])
        return [R.nnz, iterations, chaos] + _into(s, R)
    if s.kind == "bfs":
        bfs.bfs_device(s.graph, s.root, s.parents.data_ptr(), s.levels.data_ptr())
        return [s.parents, s.levels]
    if s.kind == "msbfs":
        bfs.msbfs(s.graph, s.roots, s.parents.data_ptr())
        return [s.parents]
    if s.kind == "spmv":  # y <- y (+) A x, in place
        s.plan.multiply(s.x.data_ptr(), s.y.data_ptr(), c["sr"])
        return [s.y]
    return list(s.plan.multiply(s.xi, s.xv, c["sr"]))


# ------------------------------------------------------- values in 64 bits
def _product(A, B, sr, most=1 << 26):
    """num of A * B column by column, rows ascending, in 64 bits."""
    av, bv = A.val.double(), B.val.double()
    alen, bcol = A.cp.diff(), B.cols()
    cum = torch.cumsum(alen[B.ir], 0)
    out, e0, ne = [], 0, B.nnz
    while e0 < ne:
        done = int(cum[e0 - 1]) if e0 else 0
        e1 = int(torch.searchsorted(cum, done + most, right=True))
        if e1 < ne:  # whole columns only
            e1 = max(int(B.cp[bcol[e1]]), int(B.cp[bcol[e0] + 1]))
        k = B.ir[e0:e1]
        rep = torch.repeat_interleave(torch.arange(e1 - e0, device=DEV), alen[k])
        idx = torch.arange(rep.numel(), device=DEV) - (cum[e0:e1] - alen[k] - done)[rep] + A.cp[k][rep]
        a, b = av[idx], bv[e0:e1][rep]
        val = a * b if sr == "plustimes" else a + b if sr == "minplus" else b
        key, inv = torch.unique((bcol[e0:e1])[rep] * A.nrow + A.ir[idx], return_inverse=True)
        if sr == "plustimes":
            out.append(torch.zeros(key.numel(), dtype=torch.float64, device=DEV).index_add_(0, inv, val))
        else:
            out.append(torch.full((key.numel(),), float("inf"), dtype=torch.float64, device=DEV).scatter_reduce_(
                0, inv, val, "amin"))
        e0 = e1
    return torch.cat(out) if out else av[:0]


def exact(case, seed):
    kind = case["kind"]
    if kind == "spgemm" and case["dtype"] in ("f64", "f32"):
        A = _inputs(case, seed)
        num = _product(A, A, case["sr"])
        if case["where"] == "device":
            return {"cp": None, "jc": None, "ir": None, "num": num}
        return [None, None, None, num]
    if kind == "batch":
        return [[None, None, _product(A, B, "plustimes")] for A, B in _inputs(case, seed)]
    if kind == "spmv" and case["dtype"] in ("f64", "f32"):
        M, x, y = _inputs(case, seed)
        a, x, y = M.val.double(), x.double(), y.double()
        if case["sr"] == "plustimes":
            return [y.index_add_(0, M.ir, a * x[M.cols()])]
        return [y.scatter_reduce_(0, M.ir, a + x[M.cols()], "amin")]
    if kind == "spmspv" and case["dtype"] != "none":
        M, xi, xv = _inputs(case, seed)
        x = torch.zeros(M.ncol, dtype=torch.float64, device=DEV)
        at = torch.from_numpy(xi).to(DEV).long()
        x[at] = torch.from_numpy(xv).to(DEV).double()
        there = torch.zeros(M.ncol, dtype=torch.bool, device=DEV)
        there[at] = True
        c = M.cols()
        y = torch.zeros(M.nrow, dtype=torch.float64, device=DEV).index_add_(0, M.ir, M.val.double() * x[c])
        hit = torch.zeros(M.nrow, dtype=torch.bool, device=DEV)
        hit[M.ir[there[c]]] = True
        return [None, y[hit].cpu().numpy()]
    # phased products are too many; the MCL selections compare rounded sums with each other, so that which
    # entries stay has no value apart from the rounding; traversals and whole-number semirings are whole numbers
    return None


# ------------------------------------------------------------- bytes and flops
def _matrix_bytes(M, value):
    return M.nnz * (8 + value) + (M.ncol + 1) * 8


def _product_work(A, B, value):
    a, b = (local.DeviceMatrix(M.nrow, M.ncol, M.cp, M.ir) for M in (A, B))
    flops = int(local.estimateFLOP(a, b).sum())
    nnz = int(local.estimateNNZ_Hash(a, b).sum())
    read = _matrix_bytes(A, value) + (0 if A is B else _matrix_bytes(B, value))
    return read + nnz * (8 + value) + (B.ncol + 1) * 8, 2 * flops


def work(case):
    kind = case["kind"]
    M = _inputs(case, 1)
    size = {"f64": 8, "f32": 4, "i64": 8, "bool": 1, "none": 8}
    if kind in ("spgemm", "phased"):
        b, f = _product_work(M, M, size[case.get("dtype", "f64")])
    elif kind == "batch":
        parts = [_product_work(A, B, 8) for A, B in M]
        b, f = sum(p[0] for p in parts), sum(p[1] for p in parts)
    elif kind == "mcl_expand":
        # the matrix once and at most `select` kept entries a column; the product itself need not be stored
        _, f = _product_work(M, M, 4)
        b = _matrix_bytes(M, 4) + case["n"] * case["select"] * 12
    elif kind == "mcl_loop":
        # about the first expansion, the matrix read and its successor written
        b, f = _product_work(M, M, 4)
    elif kind == "bfs":  # row ids (4 bytes each in the handle) once, parents and levels written
        b, f = M[0].nnz * 4 + (case["n"] + 1) * 8 + case["n"] * 16, 0
    elif kind == "msbfs":
        b, f = M[0].nnz * 4 + (case["n"] + 1) * 8 + case["n"] * case["roots"] * 8, 0
    elif kind == "spmv":
        M, x, y = M
        v = size[case["dtype"]]
        b, f = M.nnz * (4 + v) + M.ncol * v + M.nrow * (2 * v + 8), 2 * M.nnz
    else:
        M, xi, xv = M
        v = size[case["dtype"]]
        touched = int(M.cp.diff()[torch.from_numpy(xi).to(DEV).long()].sum())
        b, f = xi.size * (4 + v) + touched * (4 + (0 if case["dtype"] == "none" else v)) + touched * (4 + v), 2 * touched
    return {"bytes": float(b), "flops": float(f)}
