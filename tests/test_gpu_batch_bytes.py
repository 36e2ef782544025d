"""Admission sizes: fap_graph_batch_bytes, fap_graph_rows_bytes and
fap_graph_cache_bytes bound what solves, rows and cache builds allocate, and a
server keeps within a tight budget while its batches change."""
import ctypes

import numpy as np
import pytest

from fastapsp_b200 import FAP_DTYPE_F32, FAP_MODE_BATCHED, Context, DeviceGraph, fapGraph
from fastapsp_b200 import generators as G
from fastapsp_b200._lib import check, lib, ptr
from fastapsp_b200.serve import Server

pytestmark = pytest.mark.gpu

CASES = {
    "road": (lambda: G.road_graph(3001, seed=50), 9),            # elimination, thin parts
    "rgg": (lambda: G.random_geometric_graph(4000, 3.6, seed=51), 8),
    "grid": (lambda: G.grid_graph(60, 60, extra_frac=0.01, wmin=1, wmax=100, seed=52), 6),
    "grid_parts": (lambda: G.grid_graph(100, 100, extra_frac=0.01, wmin=1, wmax=100, seed=53), 40),   # boundary closed by Floyd
    "rmat": (lambda: G.rmat_graph(10, 8000, seed=54), 4),        # float32, directed, tiled SSSP
}


def _graph(name):
    make, K = CASES[name]
    el = make()
    ro, col, w = G.edges_to_csr(el)
    fg = fapGraph.from_csr(el.n, int(ro[-1]), ro, col, w, K, directed=el.directed)
    fg.preCondition()
    vn, vo, bn = fg.partInfo()
    dg = DeviceGraph(Context(0), ro, col, w)
    dg.set_parts(K, fg.getGraphId(), fg.getMapping(), vn, vo, bn)
    return dg, K, vn, (ro, col, w, K, fg.getGraphId(), fg.getMapping(), vn, vo, bn)


def _batch_bytes(dg, parts, rows, copied):
    b = ctypes.c_int64()
    ids = None if parts is None else np.asarray(parts, np.int32)
    check(lib().fap_graph_batch_bytes(dg._h, None if ids is None else ptr(ids), 0 if ids is None else len(ids),
                                      rows, copied, ctypes.byref(b)))
    return b.value


def _rows_bytes(dg, count):
    b = ctypes.c_int64()
    check(lib().fap_graph_rows_bytes(dg._h, count, ctypes.byref(b)))
    return b.value


@pytest.mark.parametrize("params", [{}, {"eliminate": 0}, {"stage1": 1}, {"bgraph_form": 2}, {"minplus_prepack": 0}],
                         ids=lambda f: ",".join(f"{k}={v}" for k, v in f.items()) or "auto")
@pytest.mark.parametrize("name", CASES)
def test_bounds_cover_the_allocations(cuda_ok, name, params):
    dg, K, vn, _ = _graph(name)
    for k, v in params.items():
        dg.set_param(k, v)

    def batch(parts):
        every = parts or list(range(1, K + 1))
        rows, copied = int(vn[every].sum()), int(vn[every].max())
        before, bound = dg.device_bytes(), _batch_bytes(dg, parts, rows, copied)
        if rows > batch.reserved:
            dg.reserve(rows)
            batch.reserved = rows
        dg.solve(parts, FAP_MODE_BATCHED)
        dg.copy_block(every[int(np.argmax(vn[every]))], out_dtype=FAP_DTYPE_F32)
        dg.check()
        assert dg.device_bytes() - before <= bound, (parts, dg.stage1_name(), dg.device_bytes() - before, bound)
    batch.reserved = 0
    for parts in ([1], [2, 1], [K, 1, 2], list(range(1, K)), None):
        batch(parts)
    cb, built = dg.cache_bytes()
    dg.release()
    batch.reserved = 0
    before = dg.device_bytes()
    dg.cache_build()
    assert dg.device_bytes() - before <= cb, (dg.device_bytes() - before, cb)
    for count in (1, 7, 300):
        before, bound = dg.device_bytes(), _rows_bytes(dg, count)
        dg.rows((np.arange(count) * 7 % dg.n).tolist())
        # (the rows themselves are the caller's)
        assert dg.device_bytes() - before <= bound, count
    for parts in ([1], [K, 1, 2], None):
        batch(parts)


@pytest.mark.parametrize("name,slack_mb", [("grid", 1), ("grid_parts", 6), ("rgg", 0)])
def test_server_keeps_within_a_tight_budget(cuda_ok, name, slack_mb):
    """Room for every request sized exactly and some MB more: the resident
    cache does not fit, batches of every size are tried."""
    dg, K, vn, args = _graph(name)
    cache = dg.cache_bytes()[0]
    budget = dg.device_bytes() + (slack_mb << 20) + max(
        _batch_bytes(dg, [p], int(vn[p]), int(vn[p])) + int(vn[p]) * 8 for p in range(1, K + 1))
    assert dg.device_bytes() + cache > budget
    del dg
    rng = np.random.default_rng(6)
    with Server(0, budget_bytes=budget) as srv:
        gi = srv.add_csr(*args)
        reqs = [srv.submit_subgraph(gi, int(p)) for p in rng.permutation(np.repeat(np.arange(1, K + 1), 3))]
        for r in reqs:
            r.result(timeout=120)
        srv.drain()
        st = srv.stats()
        assert st.failed == 0 and st.completed == len(reqs)
        assert st.peak_bytes <= budget, st.peak_bytes - budget


def test_a_negative_count_is_refused(cuda_ok):
    dg, K, vn, _ = _graph("road")
    b = ctypes.c_int64()
    ids = np.asarray([1], np.int32)
    with pytest.raises(Exception, match="negative count"):
        check(lib().fap_graph_batch_bytes(dg._h, ptr(ids), -1, 1, 1, ctypes.byref(b)))
