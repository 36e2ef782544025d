"""What the general path answers, elimination answers too: inputs at the limits
of the elimination's plans and kernels, with "eliminate" on (the default)
against 0."""
import numpy as np
import pytest

from fastapsp_b200 import FAP_DTYPE_F32, FAP_DTYPE_I32, FAP_MODE_BATCHED, Context, DeviceGraph, fapGraph
from fastapsp_b200 import generators as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("directed", [False, True])
def test_float_weights_beyond_the_sentinel(cuda_ok, directed):
    """Arcs of weight 1.5e8 and 3e8 (unreachable is 1e8 and more): whole small
    weights otherwise, so float32 sums are exact in any order and the blocks
    have to be the same bits."""
    el = G.rmat_graph(9, 3000, seed=41) if directed else G.road_graph(900, seed=41)
    rng = np.random.default_rng(41)
    el.weights = rng.integers(1, 50, el.weights.shape[0]).astype(np.float32)
    el.weights[::7] = 1.5e8
    el.weights[3::11] = 3e8
    ro, col, w = G.edges_to_csr(el)
    K = 3
    fg = fapGraph.from_csr(el.n, int(ro[-1]), ro, col, w, K, directed=el.directed)
    fg.preCondition()
    dg = DeviceGraph(Context(0), ro, col, w, FAP_DTYPE_F32)
    vn, vo, bn = fg.partInfo()
    dg.set_parts(K, fg.getGraphId(), fg.getMapping(), vn, vo, bn)
    out = []
    for eliminate in (0, 1):
        dg.set_param("eliminate", eliminate)
        dg.solve(mode=FAP_MODE_BATCHED)
        out.append([dg.copy_block(p) for p in range(1, K + 1)])
    assert any((b > 1e8).any() for b in out[0])
    for p, (a, b) in enumerate(zip(*out), 1):
        assert np.array_equal(a.view(np.int32), b.view(np.int32)), f"part {p}"


def test_some_of_more_parts_than_a_grid_has_rows(cuda_ok):
    """66,001 parts: a batch of a few of them (a path through four parts of two
    vertices, the other vertices alone)."""
    K, n = 66001, 66005
    gid = np.concatenate([np.repeat(np.arange(1, 5), 2), np.arange(5, K + 1)]).astype(np.int32)
    path = np.arange(8)
    edges = np.stack([path[:-1], path[1:]], 1)
    el = G.EdgeList(n, np.concatenate([edges, edges[:, ::-1]]), np.full(14, 3.0, np.float32), directed=True,
                    weighted=True, integral=True)
    ro, col, w = G.edges_to_csr(el)
    vn = np.zeros(K + 1, np.int32)
    vn[1:] = np.bincount(gid)[1:]
    bn = np.zeros(K + 1, np.int32)
    bn[1:5] = [1, 2, 2, 1]
    vo = np.concatenate([[0, 0], np.cumsum(vn[1:-1])]).astype(np.int32)
    st2ed = np.arange(n, dtype=np.int32)
    st2ed[:2] = [1, 0]                       # part 1: its boundary vertex first
    dg = DeviceGraph(Context(0), ro, col, w)
    dg.set_parts(K, gid, st2ed, vn, vo, bn)
    dg.reserve(64)
    some = [3, 1, 4, 700]
    dg.solve(some, FAP_MODE_BATCHED)
    for p in some:
        b = dg.copy_block(p)
        for r, v in enumerate(st2ed[vo[p]:vo[p] + vn[p]]):
            want = np.full(n, 100000000)
            want[v] = 0
            if v < 8:
                want[:8] = 3 * np.abs(path - v)
            assert np.array_equal(b[r], want), (p, r)


def test_no_memory_for_the_plans(cuda_ok):
    """A partition is accepted when the device has no room for the elimination's
    plans (tens of MB for this graph): the graph then takes the general path."""
    import torch
    el = G.grid_graph(224, 224, extra_frac=0.01, wmin=1, wmax=100, seed=42)
    ro, col, w = G.edges_to_csr(el)
    K = 48
    fg = fapGraph.from_csr(el.n, int(ro[-1]), ro, col, w, K, directed=el.directed)
    fg.preCondition()
    vn, vo, bn = fg.partInfo()
    parts = (K, fg.getGraphId(), fg.getMapping(), vn, vo, bn)
    dg = DeviceGraph(Context(0), ro, col, w)
    before = dg.device_bytes()
    dg.set_parts(*parts)
    plans = dg.device_bytes() - before
    assert plans > 30 << 20                  # (more than what is left below)
    del dg
    dg = DeviceGraph(Context(0), ro, col, w)
    torch.cuda.empty_cache()
    held = []

    def free():
        return torch.cuda.mem_get_info()[0]

    try:
        size = free() - (20 << 20)
        while free() > 24 << 20 and size > 10 << 20:    # all but 20 MB of the device
            try:
                held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:
                size //= 2
            size = min(size, free() - (20 << 20))
        if not 8 << 20 < free() <= 24 << 20:
            pytest.skip(f"{free()} bytes of the device left")
        dg.set_parts(*parts)
    finally:
        del held
        torch.cuda.empty_cache()
    dg.reserve(int(vn[1:4].sum()))
    some = [1, 2, 3]
    dg.solve(some, FAP_MODE_BATCHED)
    assert "elimination" not in dg.stage1_name()
    got = [dg.copy_block(p) for p in some]
    dg.set_parts(*parts)                     # now there is room
    dg.reserve(int(vn[1:4].sum()))
    dg.solve(some, FAP_MODE_BATCHED)
    for a, p in zip(got, some):
        assert np.array_equal(a, dg.copy_block(p)), p


@pytest.mark.parametrize("dtype", ["i32", "f32"])
@pytest.mark.parametrize("directed,side,closes", [
    (False, 36, True),      # whole plan in shared memory
    (False, 64, True),      # weights and heads only
    (False, 70, False),     # the parts keep Floyd-Warshall
    (True, 36, True), (True, 50, True), (True, 64, False)])
def test_numeric_elimination_by_size(cuda_ok, directed, side, closes, dtype):
    """Grid parts below and above what a CTA's shared memory holds of the numeric
    elimination: the same blocks as the general path (whole weights: float32 sums
    are exact), for all parts, one part and from the resident cache; the form's
    name says which closed them."""
    K = 2
    el = G.grid_graph(side, side, extra_frac=0.01 if side == 70 else 0.0, wmin=1, wmax=100, seed=43)
    if directed:
        rng = np.random.default_rng(43)
        el = G.EdgeList(el.n, np.concatenate([el.edges, el.edges[:, ::-1]]),
                        rng.integers(1, 100, 2 * el.edges.shape[0]).astype(np.float32), directed=True, weighted=True,
                        integral=True)
    ro, col, w = G.edges_to_csr(el)
    fg = fapGraph.from_csr(el.n, int(ro[-1]), ro, col, w, K, directed=el.directed)
    fg.preCondition()
    dg = DeviceGraph(Context(0), ro, col, w, FAP_DTYPE_I32 if dtype == "i32" else FAP_DTYPE_F32)
    vn, vo, bn = fg.partInfo()
    dg.set_parts(K, fg.getGraphId(), fg.getMapping(), vn, vo, bn)
    if directed or dtype == "f32":
        dg.set_param("stage1", 1)
    dg.set_param("eliminate", 0)
    dg.solve(mode=FAP_MODE_BATCHED)
    want = [dg.copy_block(p) for p in range(1, K + 1)]
    dg.set_param("eliminate", 1)
    for parts in (None, [2], None, None, None):          # (launched directly, then captured and replayed)
        dg.solve(parts, FAP_MODE_BATCHED)
        assert ("elimination" in dg.stage1_name()) == closes
        for p in parts or range(1, K + 1):
            assert np.array_equal(dg.copy_block(p), want[p - 1]), p
    dg.cache_build()
    assert np.array_equal(dg.rows([int(fg.getMapping()[vo[2] + 40])])[0], want[1][40].astype(np.float32))
    for parts in ([1], None):
        dg.solve(parts, FAP_MODE_BATCHED)
        assert dg.last_stage1() == 3 and ("elimination" in dg.stage1_name()) == closes
        for p in parts or range(1, K + 1):
            assert np.array_equal(dg.copy_block(p), want[p - 1]), p


def test_some_parts_merged(cuda_ok):
    """Parts whose separator rows do not fit a CTA's shared memory beside others
    that do: the batch takes the tiles for all, a batch of the others the merge."""
    el = G.grid_graph(110, 110, wmin=1, wmax=100, seed=4)
    ro, col, w = G.edges_to_csr(el)
    K = 4
    fg = fapGraph.from_csr(el.n, int(ro[-1]), ro, col, w, K, directed=el.directed)
    fg.preCondition()
    dg = DeviceGraph(Context(0), ro, col, w)
    vn, vo, bn = fg.partInfo()
    dg.set_parts(K, fg.getGraphId(), fg.getMapping(), vn, vo, bn)
    every = list(range(1, K + 1))
    dg.set_param("eliminate", 0)
    dg.solve(every, FAP_MODE_BATCHED)
    want = [dg.copy_block(p) for p in every]
    dg.set_param("eliminate", 1)
    alone = []
    for p in every:
        dg.solve([p], FAP_MODE_BATCHED)
        alone.append(dg.last_work()[2])
        assert np.array_equal(dg.copy_block(p), want[p - 1]), p
    assert 0 < sum(alone) < K
    for _ in range(3):
        dg.solve(every, FAP_MODE_BATCHED)
        assert dg.last_work()[2] == 0
        for p in every:
            assert np.array_equal(dg.copy_block(p), want[p - 1]), p
    assert dg.last_launches() < 60


def test_large_parts_with_narrow_boundaries_keep_the_tiles(cuda_ok):
    """Where one CTA of the merge fits on an SM and the boundary has few vertices,
    the tiles are faster; the blocks are the same."""
    el = G.random_geometric_graph(9600, 4.0, seed=3)
    ro, col, w = G.edges_to_csr(el)
    K = 2
    fg = fapGraph.from_csr(el.n, int(ro[-1]), ro, col, w, K, directed=el.directed)
    fg.preCondition()
    dg = DeviceGraph(Context(0), ro, col, w)
    vn, vo, bn = fg.partInfo()
    assert 16 < bn[1:].min() and bn[1:].max() < 64
    dg.set_parts(K, fg.getGraphId(), fg.getMapping(), vn, vo, bn)
    out = []
    for eliminate in (0, 1):
        dg.set_param("eliminate", eliminate)
        dg.solve(mode=FAP_MODE_BATCHED)
        assert ("elimination" in dg.stage1_name()) == bool(eliminate) and dg.last_work()[2] == 0
        out.append([dg.copy_block(p) for p in range(1, K + 1)])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
