"""fap_op_minplus where the operands are packed first (large products) and just
below that size, with aligned and unaligned rows: the same minima as torch (one
rounding per sum in float32), nothing written beyond the result."""
import pytest

from fastapsp_b200 import FAP_DTYPE_F32, FAP_DTYPE_I32, Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["i32", "f32"])
@pytest.mark.parametrize("M,N,K", [(1000, 9999, 101), (129, 30001, 260), (1025, 8064, 128), (900, 9001, 123)])
def test_minplus_packed(cuda_ok, M, N, K, dtype):
    import torch
    g = torch.Generator(device="cuda").manual_seed(M)
    t = torch.int32 if dtype == "i32" else torch.float32

    def operand(rows, cols):
        x = torch.rand((rows, cols), generator=g, device="cuda") * 1000
        far = torch.rand((rows, cols), generator=g, device="cuda") < 0.1
        return x.to(t).masked_fill_(far, 100000000)

    a, b = operand(M, K), operand(K, N)
    want = torch.full((M, N), 100000000, dtype=t, device="cuda")
    for k in range(K):
        torch.minimum(want, a[:, k:k + 1] + b[k:k + 1], out=want)
    buf = torch.full((M + 1, N + 3), 7, dtype=t, device="cuda")
    ctx = Context(0)
    torch.cuda.synchronize()
    ctx.minplus(a, b, buf[:M, :N], FAP_DTYPE_I32 if dtype == "i32" else FAP_DTYPE_F32)
    assert torch.equal(buf[:M, :N], want)
    assert bool((buf[M:] == 7).all()) and bool((buf[:, N:] == 7).all())
