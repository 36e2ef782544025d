"""The general path (Floyd work queue, packed min-plus tiles, Floyd closure of the
boundary graph), asked for with "eliminate" 0: undirected graphs and the SSSP
form's closures take the vertex elimination by default, so the comparisons of
these forms switch it off and check that the form ran.  Also the predecessor
rows in shared memory at every number of rows a CTA holds."""
import ctypes

import numpy as np
import pytest

from fastapsp_b200 import FAP_MODE_BATCHED, FAP_MODE_PLAIN, Context, DeviceGraph, fapGraph, workloads
from fastapsp_b200 import generators as G
from fastapsp_b200._lib import check, lib

pytestmark = pytest.mark.gpu


def _workload(name):
    wl = workloads.load(name)
    ro, col, w = wl.csr()
    dg = DeviceGraph(Context(0), ro, col, w)
    dg.set_parts(wl.K, wl.graph.getGraphId(), wl.graph.getMapping(), wl.ver_num, wl.ver_offset, wl.bdy_num)
    dg.set_param("eliminate", 0)
    return wl, dg


def _device(el, K):
    ro, col, w = G.edges_to_csr(el)
    fg = fapGraph.from_csr(el.n, int(ro[-1]), ro, col, w, K, directed=el.directed)
    fg.preCondition()
    vn, vo, bn = fg.partInfo()
    dg = DeviceGraph(Context(0), ro, col, w)
    dg.set_parts(K, fg.getGraphId(), fg.getMapping(), vn, vo, bn)
    return dg, fg.getMapping(), vn, vo, bn, (ro, col, w)


def _launches(dg):
    n = ctypes.c_int64()
    check(lib().fap_graph_last_launches(dg._h, ctypes.byref(n)))
    return n.value


def _solve(dg, K, **params):
    for k, v in params.items():
        dg.set_param(k, v)
    dg.solve(None, FAP_MODE_BATCHED)
    return [dg.copy_block(p) for p in range(1, K + 1)], _launches(dg)


def _same(got, want):
    for p, (a, b) in enumerate(zip(got, want), 1):
        assert np.array_equal(a.view(np.int32), b.view(np.int32)), f"part {p}"


@pytest.mark.parametrize("name,params,stage1", [
    ("grid128", {}, "boundary graph, Floyd closure"),
    ("grid128", {"stage1": 1}, "SSSP, frontier"),
    ("grid128", {"stage1": 1, "minplus_pack16": 0}, "SSSP, frontier"),
    ("rmat14", {}, "SSSP, tiled Bellman-Ford"),
    ("road20k", {}, "boundary graph, Floyd closure"),
])
def test_queue_equals_multi_launch(cuda_ok, name, params, stage1):
    """One persistent launch against three launches a pivot block: the same
    bits, and fewer launches show that the queue ran."""
    wl, dg = _workload(name)
    want, multi = _solve(dg, wl.K, floyd_queue=0, **params)
    assert dg.stage1_name() == stage1
    got, queue = _solve(dg, wl.K, floyd_queue=1, **params)
    assert dg.stage1_name() == stage1
    blocks = -(-int(max(wl.ver_num)) // 128)
    assert multi - queue >= 3 * (blocks - 1)
    _same(got, want)


@pytest.mark.parametrize("name", ["grid128", "rmat14", "road20k"])
def test_queue_in_the_cache_build(cuda_ok, name):
    wl, dg = _workload(name)
    want, _ = _solve(dg, wl.K, floyd_queue=0)
    launches = []
    for queue in (0, 1):
        dg.set_param("floyd_queue", queue)
        dg.cache_build()
        dg.check()
        launches.append(_launches(dg))
        parts = [1, wl.K // 2, wl.K]
        dg.solve(parts, FAP_MODE_BATCHED)
        assert "elimination" not in dg.stage1_name()
        _same([dg.copy_block(p) for p in parts], [want[p - 1] for p in parts])
        dg.cache_release()
    assert launches[1] < launches[0]


@pytest.mark.parametrize("name", ["grid128", "road20k"])
def test_symmetric_queue_equals_full_queue(cuda_ok, name):
    wl, dg = _workload(name)
    want, _ = _solve(dg, wl.K, floyd_symmetric=0)
    got, _ = _solve(dg, wl.K, floyd_symmetric=1)
    assert dg.stage1_name() == "boundary graph, Floyd closure"
    _same(got, want)


def _heavy_grid(heavy_rows, seed):
    """96 x 96 grid, weights 1..100, but up to 200,000 from row heavy_rows on:
    distances there are too long for the packed tiles."""
    el = G.grid_graph(96, 96, extra_frac=0.01, wmin=1, wmax=100, seed=seed)
    rng = np.random.default_rng(seed)
    heavy = (el.edges // 96 >= heavy_rows).all(axis=1)
    el.weights = el.weights.copy()
    el.weights[heavy] = rng.integers(1, 200001, int(heavy.sum())).astype(np.float32)
    return el


@pytest.mark.parametrize("prepack", [1, 0])
@pytest.mark.parametrize("heavy_rows,expect", [(96, "all"), (48, "some"), (0, "none")])
def test_packed_tiles_equal_int32_tiles(cuda_ok, heavy_rows, expect, prepack):
    """Every tile of every part is counted in the batched, the plain and the
    cached solve, all, some or none of them packed."""
    K = 12
    dg, _, vn, _, bn, _ = _device(_heavy_grid(heavy_rows, 11), K)
    assert int(bn[1:].min()) > 16
    dg.set_param("eliminate", 0)
    dg.set_param("minplus_prepack", prepack)
    parts = list(range(1, K + 1))
    dg.set_param("minplus_pack16", 0)
    dg.solve(parts, FAP_MODE_BATCHED)
    want = [dg.copy_block(p) for p in parts]
    assert dg.pack16_tiles() == (0, 0)
    dg.set_param("minplus_pack16", 1)
    ld = -(-dg.n // 128)
    tiles = sum(-(-int(vn[p] - bn[p]) // 128) for p in parts) * ld
    seen = 0
    for mode, cached in ((FAP_MODE_BATCHED, False), (FAP_MODE_PLAIN, False), (FAP_MODE_BATCHED, True)):
        if cached:
            dg.cache_build()
        dg.solve(parts, mode)
        _same([dg.copy_block(p) for p in parts], want)
        packed, total = dg.pack16_tiles()
        seen += tiles
        assert total == seen, (mode, cached)
        if expect == "all":
            assert packed == total
        elif expect == "none":
            assert packed == 0
        else:
            assert 0 < packed < total


@pytest.mark.parametrize("n,degree,K", [(3000, 3.2, 5), (2500, 2.2, 4)])
def test_forms_without_elimination_equal_it(cuda_ok, n, degree, K):
    dg, *_ = _device(G.road_graph(n, seed=61, target_avg_degree=degree), K)
    want, _ = _solve(dg, K)
    assert "elimination" in dg.stage1_name()
    dg.set_param("eliminate", 0)
    for form in ({"floyd_queue": 0}, {"floyd_symmetric": 0}, {"stage1": 2}, {"thin_max_b": 0},
                 {"thin_max_b": 0, "minplus_pack16": 0}, {"thin_max_b": 0, "minplus_prepack": 0}):
        got, _ = _solve(dg, K, **form)
        assert dg.stage1_name() == "boundary graph, Floyd closure"
        _same(got, want)
        for k in form:
            dg.set_param(k, {"stage1": 0, "thin_max_b": 16}.get(k, 1))


def _predecessors(row, src, ro, col, w):
    """Least distance sum, then least vertex, over the in-edges; -1 where
    unreachable; the source itself."""
    u = np.repeat(np.arange(ro.shape[0] - 1), np.diff(ro))
    key = row[u].astype(np.int64) + w.astype(np.int64)
    key = np.where(row[u] < 100000000, (key << 32) | u, np.iinfo(np.int64).max)
    best = np.full(row.shape[0], np.iinfo(np.int64).max)
    np.minimum.at(best, col, key)
    pred = np.where((best == np.iinfo(np.int64).max) | (row >= 100000000), -1, best & 0xffffffff)
    pred[src] = src
    return pred


@pytest.mark.parametrize("n", [7100, 7300, 14400, 14500, 19200, 19300, 28900, 29100])
def test_predecessor_rows_at_every_width(cuda_ok, n):
    """226 KB hold 8, 4, 3 or 2 rows of this many columns, or (29,100) fewer
    than two, where the rows are gathered from global memory: the inner rows of
    a part with a wide boundary against the rule on the distances, unreachable
    columns and an odd number of rows among them."""
    el = G.grid_graph(n // 100, 100, extra_frac=0.005, drop_frac=0.05, wmin=1, wmax=30, seed=n)
    K = max(2, n // 600)
    dg, st2ed, vn, vo, bn, (ro, col, w) = _device(el, K)
    p = next(q for q in range(1, K + 1) if bn[q] > 16 and (vn[q] - bn[q]) % 2 == 1)
    dg.set_param("paths", 1)
    dg.reserve(int(vn[p]))
    dg.solve([p], FAP_MODE_BATCHED)
    D, P = dg.copy_block(p), dg.copy_path_block(p)
    inner = range(int(bn[p]), int(vn[p]))
    for r in list(inner)[::37] + list(inner)[-9:]:
        want = _predecessors(D[r], int(st2ed[vo[p] + r]), ro, col, w)
        assert np.array_equal(P[r], want), r


def test_forms_name_themselves(cuda_ok):
    """The form names say what closes the parts and the boundary graph, and the
    relaxations reported are those run."""
    def names(dg, **params):
        for k, v in params.items():
            dg.set_param(k, v)
        dg.solve(None, FAP_MODE_BATCHED)
        return dg.stage1_name()

    wl, dg = _workload("road20k")
    vn, bn = wl.ver_num[1:].astype(float), wl.bdy_num[1:].astype(float)
    assert names(dg) == "boundary graph, Floyd closure"
    assert dg.last_work() == ((vn ** 3).sum(), ((vn - bn) * bn).sum() * wl.n, 0)
    assert names(dg, eliminate=1) == "boundary graph, Floyd class closed by elimination"
    assert 0 < dg.last_work()[0] < (vn ** 3).sum() / 100 and dg.last_work()[2] == 0
    assert names(dg, stage1=1) == "SSSP, frontier, parts closed by elimination"
    assert names(dg, eliminate=0) == "SSSP, frontier"

    dg, *_ = _device(G.grid_graph(112, 111, extra_frac=0.01, wmin=1, wmax=100, seed=3), 30)
    assert names(dg) == "boundary graph, Floyd closure, parts closed by elimination"
    closures, inner, merged = dg.last_work()
    assert merged > 0
    assert names(dg, eliminate=0) == "boundary graph, Floyd closure"
    assert closures < dg.last_work()[0] and inner < dg.last_work()[1] / 2 and dg.last_work()[2] == 0
    dg.set_param("eliminate", 1)
    dg.cache_build()
    assert names(dg) == "resident cache (boundary graph, Floyd closure, parts closed by elimination)"
    assert dg.last_work()[0] == 0 and dg.last_work()[1] == inner

    dg, *_ = _device(G.rmat_graph(11, 30000, seed=62), 4)
    assert names(dg) == "SSSP, tiled Bellman-Ford, parts closed by elimination"
    assert names(dg, eliminate=0) == "SSSP, tiled Bellman-Ford"
