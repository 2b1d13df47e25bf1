"""RMSNorm at the edges of its forms: rows kept in registers (to 8 elements of a thread), longer ones, in place."""
import pytest
import torch

from ntransformer_b200 import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden", [1, 31, 1023, 1024, 1025, 4096, 4097, 8191, 8192, 8193, 28672])
@pytest.mark.parametrize("rows", [1, 3])
def test_rows(rows, hidden):
    g = torch.Generator().manual_seed(hidden)
    x = (torch.randn(rows, hidden, generator=g) * 3).cuda()
    w = (1 + 0.1 * torch.randn(hidden, generator=g)).cuda()
    want = x.double() * torch.rsqrt(x.double().pow(2).mean(1, keepdim=True) + 1e-5) * w.double()
    y, half = torch.full((rows, hidden), 7.0, device="cuda"), torch.full((rows, hidden), 7.0, device="cuda", dtype=torch.float16)
    K.launch_rmsnorm(y, x, w, rows, hidden, 1e-5)
    K.launch_rmsnorm_f16(half, x, w, rows, hidden, 1e-5)
    # a thread's sum has at most 28 terms, the block's 10 more additions, all of them positive: 38 roundings of 2^-24, halved by the root, and 2^-21 for the root and products
    assert ((y.double() - want).abs() <= want.abs() * (19 * 2.0**-24 + 2.0**-21)).all()
    assert torch.equal(half, y.half())
    K.launch_rmsnorm(x, x, w, rows, hidden, 1e-5)
    assert torch.equal(x, y)
