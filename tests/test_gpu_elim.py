"""Closures by vertex elimination ("eliminate", the default on undirected
int32 graphs) against the general path ("eliminate" 0: Floyd-Warshall and SSSP)
bit for bit, and against Dijkstra: full batches, batches of some of the parts,
the resident cache and predecessor rows; thin and wide boundaries, parts from
one vertex to more than a strip of sixteen columns holds, boundary graphs
closed by elimination and by Floyd, unreachable vertices, zero weights and
distances past the sentinel."""
import numpy as np
import pytest

from fastapsp_b200 import FAP_MODE_BATCHED, Context, DeviceGraph, fapGraph
from fastapsp_b200 import generators as G

pytestmark = pytest.mark.gpu

INF = 100000000


def _forest():
    """Road graph without a tenth of its edges: several components."""
    el = G.road_graph(1500, seed=21)
    keep = np.random.default_rng(21).random(el.edges.shape[0]) < 0.9
    el.edges, el.weights = el.edges[keep], el.weights[keep]
    return el


def _heavy():
    """Weights at the int32 path's largest: distances beyond 1e8."""
    el = G.road_graph(1200, seed=22)
    el.weights = np.random.default_rng(22).integers(900000, 1000001, el.weights.shape[0]).astype(np.float32)
    return el


def _zeros():
    el = G.random_geometric_graph(1100, 3.0, seed=23)
    el.weights[::3] = 0.0
    return el


def _grid_heavy():
    """Distances too long for the packed rows, on 2,048-vertex parts."""
    el = G.grid_graph(64, 64, wmin=1, wmax=200000, seed=30)
    return el


def _grid_forest():
    """A grid without a third of its edges: unreachable vertices beside wide boundaries."""
    return G.grid_graph(60, 61, drop_frac=0.33, wmin=1, wmax=50, seed=31)


CASES = {  # name: (graph, parts)
    "road": (lambda: G.road_graph(3001, seed=20), 5),
    "two_parts": (lambda: G.road_graph(2600, seed=32), 2),   # a strip's own columns by the hundred
    "tiny_parts": (lambda: G.road_graph(97, seed=24), 16),
    "forest": (_forest, 4),
    "heavy": (_heavy, 3),
    "zeros": (_zeros, 4),
    "rgg": (lambda: G.random_geometric_graph(5000, 3.7, seed=25), 6),
    "grid_small_parts": (lambda: G.grid_graph(40, 37, extra_frac=0.01, wmin=1, wmax=100, seed=26), 9),
    "grid_wide": (lambda: G.grid_graph(64, 64, wmin=1, wmax=100, seed=27), 2),   # 2,048-vertex parts
    "grid_heavy": (_grid_heavy, 2),
    "grid_forest": (_grid_forest, 4),
    "grid_floyd": (lambda: G.grid_graph(100, 100, extra_frac=0.01, wmin=1, wmax=100, seed=28), 40),
}


def _device(el, K):
    ro, col, w = G.edges_to_csr(el)
    fg = fapGraph.from_csr(el.n, int(ro[-1]), ro, col, w, K, directed=el.directed)
    fg.preCondition()
    dg = DeviceGraph(Context(0), ro, col, w)
    vn, vo, bn = fg.partInfo()
    dg.set_parts(K, fg.getGraphId(), fg.getMapping(), vn, vo, bn)
    return dg, fg.getMapping(), vn, vo, (ro, col, w)


def _blocks(dg, parts):
    return {p: dg.copy_block(p) for p in parts}


def _same(got, want):
    for p, b in got.items():
        assert np.array_equal(b, want[p]), f"part {p}: {int((b != want[p]).sum())} entries differ"


def _dijkstra(csr, sources):
    from scipy.sparse import csr_matrix
    from scipy.sparse.csgraph import dijkstra
    ro, col, w = csr
    # (scipy drops stored zeros: shift them to a weight too small to matter)
    data = np.where(w == 0, 1e-9, w.astype(np.float64))
    d = dijkstra(csr_matrix((data, col, ro), shape=(ro.shape[0] - 1,) * 2), indices=sources)
    return np.where(d >= INF, INF, np.round(np.where(np.isinf(d), INF, d))).astype(np.int64)


@pytest.mark.parametrize("name", CASES)
def test_elimination_equals_general_path(cuda_ok, name):
    make, K = CASES[name]
    dg, st2ed, vn, vo, csr = _device(make(), K)
    every = list(range(1, K + 1))
    dg.set_param("eliminate", 0)
    dg.solve(mode=FAP_MODE_BATCHED)
    assert "elimination" not in dg.stage1_name()
    want = _blocks(dg, every)
    dg.set_param("eliminate", 1)
    for _ in range(3):                      # direct launches, capture, replay
        dg.solve(mode=FAP_MODE_BATCHED)
        assert "elimination" in dg.stage1_name()
        _same(_blocks(dg, every), want)
    p = int(np.argmax(vn[1:])) + 1
    rows = list(range(0, int(vn[p]), max(1, int(vn[p]) // 9)))
    ref = _dijkstra(csr, st2ed[vo[p] + np.array(rows)])
    assert np.array_equal(want[p][rows].astype(np.int64), ref)
    # some of the parts, packed and in another order
    some = every[::-2]
    dg.reserve(int(max(sum(vn[q] for q in some), vn[p])))
    for batch in (some, [p]):
        dg.solve(batch, FAP_MODE_BATCHED)
        _same(_blocks(dg, batch), want)
    # the resident cache
    dg.cache_build()
    dg.solve(some, FAP_MODE_BATCHED)
    assert dg.last_stage1() == 3
    _same(_blocks(dg, some), want)
    src = st2ed[::max(1, st2ed.shape[0] // 23)].tolist()
    got = dg.rows(src)
    at = {int(v): i for i, v in enumerate(st2ed)}
    for r, v in enumerate(src):
        q = int(np.searchsorted(vo[1:K + 1], at[v], side="right"))
        assert np.array_equal(got[r], want[q][at[v] - vo[q]].astype(np.float32))  # (rows are float32)


@pytest.mark.parametrize("name", ["road", "rgg", "grid_small_parts"])
def test_elimination_gives_the_same_predecessors(cuda_ok, name):
    make, K = CASES[name]
    dg, *_ = _device(make(), K)
    dg.set_param("paths", 1)
    out = []
    for on in (0, 1):
        dg.set_param("eliminate", on)
        dg.solve(mode=FAP_MODE_BATCHED)
        out.append([dg.copy_path_block(p) for p in range(1, K + 1)])
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def _directed_int():
    el = G.rmat_graph(11, 9000, seed=33)          # duplicate arcs, hubs, unreachable pairs
    el.weights = np.ceil(el.weights)
    el.integral = True
    return el


def _float_rgg():
    el = G.random_geometric_graph(2100, 3.0, seed=34)
    el.weights = np.random.default_rng(34).uniform(0.5, 100.0, el.weights.shape[0]).astype(np.float32)
    return el


@pytest.mark.parametrize("name", ["directed_int", "float_rgg", "float_rmat"])
def test_closures_from_given_boundary_rows(cuda_ok, name):
    """The SSSP form's closures by elimination (any dtype, directed parts):
    int32 bit-identical to the Floyd-Warshall closures; float32 within 1e-5 (the
    sums associate differently) with reachability exact, and the same bits from
    batches of some of the parts and from the resident cache."""
    el, K = {"directed_int": (_directed_int(), 4), "float_rgg": (_float_rgg(), 3),
             "float_rmat": (G.rmat_graph(11, 9000, seed=35), 4)}[name]
    dg, st2ed, vn, vo, _ = _device(el, K)
    every = list(range(1, K + 1))
    dg.set_param("stage1", 1)
    dg.set_param("eliminate", 0)
    dg.solve(mode=FAP_MODE_BATCHED)
    want = _blocks(dg, every)
    dg.set_param("eliminate", 1)
    dg.solve(mode=FAP_MODE_BATCHED)
    got = _blocks(dg, every)
    for p in every:
        if name == "directed_int":
            assert np.array_equal(got[p], want[p]), p
        else:
            reach = want[p] < INF
            assert np.array_equal(got[p] < INF, reach)
            assert np.all(np.abs(got[p] - want[p])[reach] <= 1e-5 * want[p][reach])
    dg.reserve(int(vn[1:].max()))
    for p in every:
        dg.solve([p], FAP_MODE_BATCHED)
        assert np.array_equal(dg.copy_block(p).view(np.int32), got[p].view(np.int32))
    dg.cache_build()
    for p in every:
        dg.solve([p], FAP_MODE_BATCHED)
        assert dg.last_stage1() == 3
        assert np.array_equal(dg.copy_block(p).view(np.int32), got[p].view(np.int32))


def test_asymmetric_weights_keep_the_general_path(cuda_ok):
    el = G.road_graph(900, seed=29)
    both = np.concatenate([el.edges, el.edges[:, ::-1]])
    w = np.concatenate([el.weights, el.weights])
    w[3] += 1.0
    dg, *_ = _device(G.EdgeList(el.n, both, w, directed=True, weighted=True, integral=True), 3)
    dg.solve(mode=FAP_MODE_BATCHED)
    assert "elimination" not in dg.stage1_name()
