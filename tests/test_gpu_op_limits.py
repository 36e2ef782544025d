"""Operators on matrices with more rows than a grid has blocks in y (65,535):
the shapes an operator takes do not depend on how its operands are staged."""
import pytest

from fastapsp_b200 import FAP_DTYPE_F32, FAP_DTYPE_I32, Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,M,N,K", [("i32", 70000, 1000, 24),      # tall
                                         ("i32", 130, 130, 66000),      # deep
                                         ("f32", 70000, 1001, 24),      # (unaligned rows)
                                         ("f32", 130, 131, 66000)])
def test_tall_and_deep_minplus(cuda_ok, dtype, M, N, K):
    """Large products: minima of exact int32 sums, or of
    float32 sums rounded once, are the same in any order."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(M)
    t = torch.int32 if dtype == "i32" else torch.float32
    a = (torch.rand((M, K), generator=g, device="cuda") * 1000).to(t)
    b = (torch.rand((K, N), generator=g, device="cuda") * 1000).to(t)
    far = torch.rand((M, K), generator=g, device="cuda") < 0.1
    a.masked_fill_(far, 100000000)
    want = torch.full((M, N), 100000000, dtype=t, device="cuda")
    step = max(1, 100000000 // (M * N))
    for k in range(0, K, step):
        torch.minimum(want, (a[:, k:k + step, None] + b[None, k:k + step]).amin(1), out=want)
    ctx = Context(0)
    for _ in range(2):                        # (the second call has packed operands)
        c = torch.full((M, N), 7, dtype=t, device="cuda")
        torch.cuda.synchronize()
        ctx.minplus(a, b, c, FAP_DTYPE_I32 if dtype == "i32" else FAP_DTYPE_F32)
        assert torch.equal(c, want)


def test_floyd_of_more_rows_than_a_grid_has(cuda_ok):
    """A 65,473 x 65,473 matrix (17 GB, and as much scratch): the ring of unit
    arcs with one chord closes to known distances."""
    import torch
    s, far = 65473, 40000
    free, _ = torch.cuda.mem_get_info()
    if free < 45 << 30:
        pytest.skip("needs 45 GB of device memory")
    m = torch.full((s, s), 100000000, dtype=torch.int32, device="cuda")
    at = torch.arange(s, device="cuda")
    m[at, at] = 0
    m[at, (at + 1) % s] = 1
    m[0, far] = 7
    ctx = Context(0)
    torch.cuda.synchronize()
    ctx.floyd(m, FAP_DTYPE_I32)
    for lo in range(0, s, 8192):
        i = at[lo:lo + 8192, None]
        ring = (at - i) % s
        chord = (-i) % s + 7 + (at - far) % s       # from i to 0, over the chord, on to j
        assert torch.equal(m[lo:lo + 8192].long(), torch.minimum(ring, chord)), lo
    del m
    torch.cuda.empty_cache()
