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
