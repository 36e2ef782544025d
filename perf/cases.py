"""The work users have this library do, as cases that can be timed.

A case names an entry point and its sizes.  The graphs are the shapes the
package's own generators make: road-shaped, grids with long-range edges,
random geometric and R-MAT.  `prepare` builds what a program has in hand
before the call (the partitioned graph, the device handle, its reserved
output, the operands of an operator), `run` makes one pass through the public
API and returns whole outputs, `work` states the bytes (each input read once,
each output written once) and `exact` the 64-bit values of floating outputs.
"""
import ctypes
import math

import numpy as np
import torch

from fastapsp_b200 import (FAP_DTYPE_F32, FAP_DTYPE_I32, Context, DeviceGraph, fapGraph)
from fastapsp_b200 import generators as G
from fastapsp_b200._lib import check, lib

INF = 1e8


def listed():
    return [
        # The drop-in class on a small graph, host matrix in hand at the end:
        # what a program written against fap::fapGraph calls.
        dict(name="dropin_grid64", kind="dropin", graph="grid", rows=64, cols=64, extra=0.0, K=8),
        # All-pairs distances left on the device, ordinary size, road-shaped.
        dict(name="solve_road20k", kind="solve", graph="road", n=20000, degree=2.1, K=24),
        # The headline configuration: road-shaped, 114,599 vertices, 128 parts.
        dict(name="solve_road114k", kind="solve", graph="road", n=114599, degree=2.1, K=128),
        # Large boundary sets: a grid with 1% long-range edges.
        dict(name="solve_grid256", kind="solve", graph="grid", rows=256, cols=256, extra=0.01, K=64),
        # Directed scale-free graph with float weights (dense part boundaries).
        dict(name="solve_rmat14_f32", kind="solve", graph="rmat", scale=14, edges=1 << 18, K=16),
        # Undirected graph with float lengths (road lengths, sensor networks).
        dict(name="solve_rgg_f32", kind="solve", graph="rgg_f32", n=20011, degree=3.0, K=20),
        # Distances and predecessors (is_path_needed).
        dict(name="paths_rgg", kind="paths", graph="rgg", n=16001, degree=2.6, K=16),
        # One sub-graph's rows without anything resident (solveSubGraph).
        dict(name="part_road50k", kind="part", graph="road", n=50001, degree=2.1, K=60),
        # A graph whose output is produced in groups of parts: refresh the
        # resident cache, then one group.
        dict(name="group_grid", kind="group", graph="grid", rows=160, cols=235, extra=0.01, K=37, groups=4),
        # Distance rows of single vertices from the resident cache.
        dict(name="rows_rgg", kind="rows", graph="rgg", n=30011, degree=3.3, K=32, count=64),
        # The stage operators on the caller's own device matrices.
        dict(name="floyd_1500", kind="floyd", s=1500, dtype="i32"),
        dict(name="minplus_f32", kind="minplus", M=900, N=20011, K=150, dtype="f32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _parts(rng, n):
    """Number of parts: blocks of 400 to 1100 rows, as the configurations have."""
    return max(2, n // rng.randint(400, 1100))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "solve", "paths", "part", "group", "rows", "dropin",
                       "floyd", "minplus"])
    if kind == "floyd":
        return dict(kind=kind, s=_log(rng, 100, 3000), dtype=rng.choice(["i32", "f32"]))
    if kind == "minplus":
        return dict(kind=kind, M=_log(rng, 60, 2000), N=_log(rng, 1000, 40000), K=_log(rng, 8, 700),
                    dtype=rng.choice(["i32", "f32"]))
    if kind == "dropin":
        rows, cols = rng.randint(24, 64), rng.randint(24, 64)
        return dict(kind=kind, graph="grid", rows=rows, cols=cols, extra=rng.choice([0.0, 0.01]),
                    K=max(2, rows * cols // rng.randint(300, 800)))
    graph = rng.choice(["road", "road", "grid", "grid", "rgg", "rgg", "rgg_f32", "rmat"])
    if graph in ("rgg_f32", "rmat") and kind != "solve":
        graph = "rgg"
    if graph == "grid":
        rows, cols = _log(rng, 40, 256), _log(rng, 40, 256)
        n = rows * cols
        case = dict(kind=kind, graph=graph, rows=rows, cols=cols, extra=rng.choice([0.0, 0.01]), K=_parts(rng, n))
    elif graph == "rmat":
        scale = rng.randint(11, 14)
        case = dict(kind=kind, graph=graph, scale=scale, edges=int((1 << scale) * rng.uniform(8, 16)),
                    K=max(2, (1 << scale) // rng.randint(700, 1100)))
    else:
        n = _log(rng, 2000, {"solve": 114599 if graph == "road" else 60000, "paths": 24000}.get(kind, 60000))
        if graph == "rgg_f32":
            n = min(n, 24000)
        degree = 2.1 if graph == "road" else round(rng.uniform(2.0, 4.0), 2)
        case = dict(kind=kind, graph=graph, n=n, degree=degree, K=_parts(rng, n))
    if kind == "paths" and graph == "grid":
        case.update(rows=min(case["rows"], 150), cols=min(case["cols"], 150))
        case["K"] = _parts(rng, case["rows"] * case["cols"])
    if kind == "group":
        case["groups"] = rng.randint(2, 5)
    if kind == "rows":
        case["count"] = _log(rng, 1, 256)
    return case


# --------------------------------------------------------------------------
# graphs
# --------------------------------------------------------------------------

def _size(case):
    if case["graph"] == "grid":
        return case["rows"] * case["cols"]
    return 1 << case["scale"] if case["graph"] == "rmat" else case["n"]


def _csr(case, seed):
    """(edge list, CSR).  A program that asks for some of a graph's parts keeps
    the graph and sees new weights: its structure does not depend on the seed."""
    kind = case["graph"]
    fixed = case["kind"] in ("part", "group")
    weights = np.random.default_rng(seed + 1)
    seed = 11 if fixed else seed
    if kind == "grid":
        wmax = 1 if case["kind"] == "dropin" else 100
        el = G.grid_graph(case["rows"], case["cols"], extra_frac=case["extra"], wmin=1, wmax=wmax,
                          drop_frac=0.02 if case["extra"] == 0.0 else 0.0, seed=seed)
    elif kind == "rmat":
        el = G.rmat_graph(case["scale"], case["edges"], seed=seed)
        _, first = np.unique(el.edges[:, 0] * el.n + el.edges[:, 1], return_index=True)  # a simple graph
        el.edges, el.weights = el.edges[first], el.weights[first]
    else:
        el = G.road_graph(case["n"], seed=seed, target_avg_degree=case["degree"])
        if kind == "rgg_f32":
            el.weights = weights.uniform(0.5, 100.0, el.weights.shape[0]).astype(np.float32)
    if fixed:
        el.weights = weights.integers(1, int(el.weights.max()) + 1, el.weights.shape[0]).astype(np.float32)
    return el, G.edges_to_csr(el)


def _host_graph(case, seed):
    el, (ro, col, w) = _csr(case, seed)
    g = fapGraph.from_csr(el.n, int(col.shape[0]), ro, col, w, case["K"], directed=el.directed)
    g.preCondition()
    return g, ro, col, w


def _chunks(rows):
    step = max(1, -(-rows // 16))
    return [(lo, min(lo + step, rows)) for lo in range(0, rows, step)]


class _DeviceRows:
    """rows x n view of a block at a device pointer, for torch."""

    def __init__(self, ptr, rows, n, ld, typestr, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"version": 3, "shape": (rows, n), "strides": (ld * 4, 4),
                                         "typestr": typestr, "data": (ptr, False)}


def _path_info(dg, part):
    ptr, rows, ld = ctypes.c_void_p(), ctypes.c_int64(), ctypes.c_int64()
    check(lib().fap_graph_path_block(dg._h, part, ctypes.byref(ptr), ctypes.byref(rows), ctypes.byref(ld)),
          "fap_graph_path_block")
    return ptr.value, rows.value, ld.value


def _blocks(dg, parts, path=False):
    """The parts' blocks (adjacent rows, in this order) as at most 16 tensors of whole rows."""
    typestr = "<i4" if path or dg.dtype == FAP_DTYPE_I32 else "<f4"
    info = [_path_info(dg, p) if path else dg.block_info(p) for p in parts]
    ptr, ld, rows = info[0][0], info[0][2], sum(x[1] for x in info)
    out = []
    for lo, hi in _chunks(rows):
        view = _DeviceRows(ptr + lo * ld * 4, hi - lo, dg.n, ld, typestr, dg)
        out.append(torch.as_tensor(view, device="cuda"))
    return out


# --------------------------------------------------------------------------
# prepare / run
# --------------------------------------------------------------------------

def _operand(case, shape, seed, device):
    """Distances with a tenth of the pairs unreachable."""
    g = torch.Generator(device=device).manual_seed(seed)
    far = torch.rand(shape, generator=g, device=device) < 0.1
    if case["dtype"] == "i32":
        return torch.randint(1, 100000, shape, generator=g, device=device, dtype=torch.int32).masked_fill_(far, int(INF))
    return (torch.rand(shape, generator=g, device=device) * 1000.0).masked_fill_(far, INF)


def _floyd_input(case, seed, device):
    """Weight matrix of a sparse directed graph of s vertices, 8 arcs each."""
    s = case["s"]
    g = torch.Generator(device=device).manual_seed(seed)
    m = torch.full((s, s), INF, dtype=torch.float32, device=device)
    at = torch.randint(0, s, (s, 8), generator=g, device=device)
    w = torch.rand((s, 8), generator=g, device=device) * 1000.0
    m.scatter_reduce_(1, at, torch.ceil(w) if case["dtype"] == "i32" else w, "amin")
    m.fill_diagonal_(0.0)
    return m.to(torch.int32) if case["dtype"] == "i32" else m


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("floyd", "minplus"):
        ctx = Context(0)
        dt = FAP_DTYPE_I32 if case["dtype"] == "i32" else FAP_DTYPE_F32
        if kind == "floyd":
            ctx.use_torch_stream()
            m = _floyd_input(case, seed, "cuda")
            return dict(case=case, ctx=ctx, dt=dt, m=m, out=torch.empty_like(m))
        a = _operand(case, (case["M"], case["K"]), seed, "cuda")
        b = _operand(case, (case["K"], case["N"]), seed + 1, "cuda")
        c = torch.empty((case["M"], case["N"]), dtype=a.dtype, device="cuda")
        torch.cuda.synchronize()
        return dict(case=case, ctx=ctx, dt=dt, a=a, b=b, c=c)
    g, ro, col, w = _host_graph(case, seed)
    if kind == "dropin":
        return dict(case=case, g=g)
    ctx = Context(0)
    dg = DeviceGraph(ctx, ro, col, w)
    vn, vo, bn = g.partInfo()
    K = case["K"]
    dg.set_parts(K, g.getGraphId(), g.getMapping(), vn, vo, bn)
    parts = list(range(1, K + 1))
    rng = np.random.default_rng(seed)
    state = dict(case=case, ctx=ctx, dg=dg, parts=parts)
    if kind == "part":
        state["parts"] = [K // 2]
        dg.reserve(int(vn.max()))
    elif kind == "group":
        state["parts"] = parts[:-(-K // case["groups"])]
        dg.cache_build()
        dg.reserve(int(vn[state["parts"]].sum()))
    elif kind == "rows":
        dg.cache_build()
        state["sources"] = rng.integers(0, _size(case), case["count"]).tolist()
    else:
        if kind == "paths":
            dg.set_param("paths", 1)
        dg.reserve()
    return state


def run(state):
    kind = state["case"]["kind"]
    if kind == "floyd":
        out = state["out"].copy_(state["m"])
        state["ctx"].floyd(out, state["dt"])
        return out
    if kind == "minplus":
        state["ctx"].minplus(state["a"], state["b"], state["c"], state["dt"])
        return state["c"]
    if kind == "dropin":
        state["g"].solve()
        return state["g"].getAllDistance()
    dg = state["dg"]
    if kind == "rows":
        return dg.rows(state["sources"])
    if kind == "group":
        dg.cache_build(rebuild=True)
    dg.solve(None if kind in ("solve", "paths") else state["parts"])
    out = dict(distance=_blocks(dg, state["parts"]))
    if kind == "paths":
        out["path"] = _blocks(dg, state["parts"], path=True)
    return out


# --------------------------------------------------------------------------
# work / exact
# --------------------------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "floyd":
        return dict(bytes=8.0 * case["s"] ** 2, flops=2.0 * case["s"] ** 3)
    if kind == "minplus":
        M, N, K = case["M"], case["N"], case["K"]
        return dict(bytes=4.0 * (M * K + K * N + M * N), flops=2.0 * M * N * K)
    n = _size(case)
    arcs = {"grid": 4.0 * n, "rmat": float(case.get("edges", 0))}.get(case["graph"], case.get("degree", 0.0) * n)
    rows = {"part": n / case["K"], "group": n / case.get("groups", 1), "rows": case.get("count", 0)}.get(kind, n)
    return dict(bytes=4.0 * n * rows * (2 if kind == "paths" else 1) + 8.0 * arcs + 4.0 * n, flops=0.0)


def _distances(case, seed, sources):
    """64-bit shortest distances (len(sources) x n) by Bellman-Ford."""
    _, (ro, col, w) = _csr(case, seed)
    n = ro.shape[0] - 1
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    u = torch.from_numpy(np.repeat(np.arange(n), np.diff(ro))).to(dev)
    v = torch.from_numpy(col.astype(np.int64)).to(dev)
    wt = torch.from_numpy(w.astype(np.float64)).to(dev)[:, None]
    s = torch.as_tensor(np.asarray(sources, dtype=np.int64), device=dev)
    d = torch.full((n, s.shape[0]), math.inf, dtype=torch.float64, device=dev)
    d[s, torch.arange(s.shape[0], device=dev)] = 0.0
    at = v[:, None].expand(-1, s.shape[0])
    while True:
        before = d.clone()
        for _ in range(8):
            d.scatter_reduce_(0, at, d[u] + wt, "amin")
        if torch.equal(before, d):
            break
    return d.masked_fill_(torch.isinf(d), INF).T


def exact(case, seed):
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "minplus" and case["dtype"] == "f32":
        a = _operand(case, (case["M"], case["K"]), seed, dev).double()
        b = _operand(case, (case["K"], case["N"]), seed + 1, dev).double()
        c = torch.full((case["M"], case["N"]), INF, dtype=torch.float64, device=dev)
        for k in range(case["K"]):
            torch.minimum(c, a[:, k:k + 1] + b[k:k + 1], out=c)
        return c
    if kind == "floyd" and case["dtype"] == "f32":
        m = _floyd_input(case, seed, dev).double()
        for k in range(case["s"]):
            torch.minimum(m, m[:, k:k + 1] + m[k:k + 1], out=m)
        return m.clamp_(max=INF)
    if kind == "rows":
        rng = np.random.default_rng(seed)
        if case["graph"] in ("road", "grid", "rgg"):
            return _distances(case, seed, rng.integers(0, _size(case), case["count"]))
    if kind == "dropin":
        g, *_ = _host_graph(case, seed)  # (the rows' order)
        return _distances(case, seed, g.getMapping())
    if kind == "solve" and case["graph"] in ("rmat", "rgg_f32"):
        g, *_ = _host_graph(case, seed)
        chunks = _chunks(_size(case))
        return dict(distance=[_distances(case, seed, g.getMapping()[:chunks[0][1]])] + [None] * (len(chunks) - 1))
    return None
