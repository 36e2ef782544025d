"""fap_op_minplus allocates its operands' scratch when a product needs that much
for the second time, not in the first call on a new context, and gives the same
values either way."""
import pytest

from fastapsp_b200 import FAP_DTYPE_F32, FAP_DTYPE_I32, Context

pytestmark = pytest.mark.gpu


def test_first_product_allocates_nothing(cuda_ok):
    import torch

    def product(ctx, M, N, K):
        g = torch.Generator(device="cuda").manual_seed(K)
        a = torch.randint(0, 1000, (M, K), generator=g, device="cuda", dtype=torch.int32)
        b = torch.randint(0, 1000, (K, N), generator=g, device="cuda", dtype=torch.int32)
        c = torch.empty((M, N), device="cuda", dtype=torch.int32)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        ctx.minplus(a, b, c, FAP_DTYPE_I32)
        return c, free - torch.cuda.mem_get_info()[0]

    for _ in range(2):                                    # (the kernels are loaded)
        product(ctx := Context(0), 1300, 12001, 501)
    product(ctx, 1300, 12001, 501)
    ctx = Context(0)
    first, grown = product(ctx, 1300, 12001, 501)         # 27 MB of copies
    assert grown == 0
    second, grown = product(ctx, 1300, 12001, 501)
    assert 24 << 20 <= grown <= 64 << 20
    assert torch.equal(first, second)
    third, grown = product(ctx, 1300, 12001, 501)
    assert grown == 0 and torch.equal(first, third)
    _, grown = product(ctx, 1300, 24001, 701)             # a larger one: generic again
    assert grown == 0
    _, grown = product(ctx, 1200, 12001, 501)             # (fits what is held)
    assert grown == 0


@pytest.mark.parametrize("dtype", ["i32", "f32"])
@pytest.mark.parametrize("M,N,K", [(1000, 19001, 101), (129, 60001, 200), (1025, 13501, 128), (900, 15001, 123),
                                   (128, 160001, 75), (1281, 11777, 100), (192, 40001, 170)])
def test_packed_products_of_a_context(cuda_ok, M, N, K, dtype):
    """The second and third product of a context (packed operands, held scratch
    of an earlier size and values): torch's minima, nothing written beyond."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(N)
    t = torch.int32 if dtype == "i32" else torch.float32
    ctx = Context(0)
    for step in range(3):
        a = (torch.rand((M, K), generator=g, device="cuda") * 1000).to(t)
        b = (torch.rand((K, N), generator=g, device="cuda") * 1000).to(t)
        for x in (a, b):
            x.masked_fill_(torch.rand(x.shape, generator=g, device="cuda") < 0.1, 100000000)
        want = torch.full((M, N), 100000000, dtype=t, device="cuda")
        for k in range(K):
            torch.minimum(want, a[:, k:k + 1] + b[k:k + 1], out=want)
        buf = torch.full((M + 1, N + 3), 7, dtype=t, device="cuda")
        torch.cuda.synchronize()
        ctx.minplus(a, b, buf[:M, :N], FAP_DTYPE_I32 if dtype == "i32" else FAP_DTYPE_F32)
        assert torch.equal(buf[:M, :N], want), step
        assert bool((buf[M:] == 7).all()) and bool((buf[:, N:] == 7).all())
