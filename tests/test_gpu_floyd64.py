"""fap_op_floyd in pivot blocks of 64 at the edges of its tiles and of its
range, against the closure in 64 bits: int32 exact; float32 within s rounding
errors (a value is a sum of at most s weights), reachability exact; rows beyond
the matrix untouched."""
import numpy as np
import pytest

from fastapsp_b200 import FAP_DTYPE_F32, FAP_DTYPE_I32, Context

pytestmark = pytest.mark.gpu

INF = 1e8


@pytest.mark.parametrize("dtype", ["i32", "f32"])
@pytest.mark.parametrize("s", [1, 3, 63, 64, 65, 112, 113, 128, 129, 191, 193, 320, 700])
def test_floyd_blocks_of_64(cuda_ok, s, dtype):
    import torch
    rng = np.random.default_rng(s)
    m = np.full((s, s), INF)
    deg = min(s, 4)
    cols = rng.integers(0, s, (s, deg))
    w = rng.uniform(0.0, 100.0, (s, deg))
    w = np.floor(w) if dtype == "i32" else w.astype(np.float32)
    np.minimum.at(m, (np.repeat(np.arange(s), deg), cols.ravel()), w.ravel())
    np.fill_diagonal(m, 0.0)
    want = m.copy()
    for k in range(s):
        np.minimum(want, want[:, k:k + 1] + want[k:k + 1], out=want)
    want = np.minimum(want, INF)
    t = torch.int32 if dtype == "i32" else torch.float32
    ld = s + 5
    buf = torch.full((s + 1, ld), 7, dtype=t, device="cuda")
    buf[:s, :s] = torch.from_numpy(m).to(t)
    ctx = Context(0)
    torch.cuda.synchronize()
    ctx.floyd(buf[:s, :s], FAP_DTYPE_I32 if dtype == "i32" else FAP_DTYPE_F32)
    ctx.sync()
    got = buf[:s, :s].cpu().numpy().astype(np.float64)
    assert bool((buf[s:] == 7).all()) and bool((buf[:, s:] == 7).all())
    if dtype == "i32":
        assert np.array_equal(got, want)
    else:
        reach = want < INF
        assert np.array_equal(got < INF, reach)
        assert np.all(np.abs(got - want)[reach] <= s * 2.0 ** -24 * want[reach])


@pytest.mark.parametrize("dtype", ["i32", "f32"])
@pytest.mark.parametrize("s", [66, 255, 2240, 2369])
def test_floyd_panels_beside_the_remainder(cuda_ok, s, dtype):
    """Two pivot blocks, an even and an odd number of them, and both launch
    shapes of the remainder (35 and 38 blocks), against pivots one by one on
    the device; tolerance as above."""
    import torch
    rng = np.random.default_rng(s)
    w = rng.uniform(0.0, 1000.0, (s, 6))
    m = np.full((s, s), INF)
    np.minimum.at(m, (np.repeat(np.arange(s), 6), rng.integers(0, s, 6 * s)),
                  (np.floor(w) if dtype == "i32" else w.astype(np.float32)).ravel())
    np.fill_diagonal(m, 0.0)
    want = torch.from_numpy(m).cuda()
    for k in range(s):
        torch.minimum(want, want[:, k:k + 1] + want[k:k + 1], out=want)
    want.clamp_(max=INF)
    got = torch.from_numpy(m).to(torch.int32 if dtype == "i32" else torch.float32).cuda()
    ctx = Context(0)
    torch.cuda.synchronize()
    ctx.floyd(got, FAP_DTYPE_I32 if dtype == "i32" else FAP_DTYPE_F32)
    ctx.sync()
    got = got.double()
    if dtype == "i32":
        assert torch.equal(got, want)
    else:
        reach = want < INF
        assert torch.equal(got < INF, reach)
        assert bool(((got - want).abs()[reach] <= s * 2.0 ** -24 * want[reach]).all())


def test_symmetric_boundary_graph_panels_beside_the_remainder(cuda_ok):
    """A boundary graph of more than 2,048 vertices (symmetric tiles) after the
    elimination, bit for bit against the general path."""
    from fastapsp_b200 import DeviceGraph, fapGraph
    from fastapsp_b200 import generators as G
    el = G.grid_graph(112, 111, extra_frac=0.01, wmin=1, wmax=100, drop_frac=0.0, seed=3)
    ro, col, w = G.edges_to_csr(el)
    K = 30
    g = fapGraph.from_csr(el.n, int(col.shape[0]), ro, col, w, K, directed=el.directed)
    g.preCondition()
    vn, vo, bn = g.partInfo()
    assert 2048 < int(np.asarray(bn).sum()) <= 8192
    dg = DeviceGraph(Context(0), ro, col, w)
    dg.set_parts(K, g.getGraphId(), g.getMapping(), vn, vo, bn)
    dg.reserve()
    out = []
    for eliminate in (1, 0):
        dg.set_param("eliminate", eliminate)
        dg.solve()
        assert ("elimination" in dg.stage1_name()) == bool(eliminate)
        out.append([dg.copy_block(p) for p in range(1, K + 1)])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
