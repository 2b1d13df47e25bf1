"""Copies and cache writes at the length from which a thread takes four elements (csrc/elementwise.cu WIDE_RUN), at its remainders, and where the cache ends inside a run."""
import pytest

torch = pytest.importorskip("torch")
from ntransformer_b200 import kernels as K  # noqa: E402

pytestmark = pytest.mark.gpu
WIDE = 1 << 18


@pytest.mark.parametrize("n", [1, 255, WIDE - 1, WIDE, WIDE + 1, WIDE + 1023, 5 * WIDE + 257])
def test_copy(n):
    x, y = torch.randn(n, device="cuda"), torch.full((n + 1,), 7.0, device="cuda")
    K.launch_copy(y, x, n)
    torch.cuda.synchronize()
    assert torch.equal(y[:n], x) and y[n] == 7.0


@pytest.mark.parametrize("tokens,kv,dim", [(1, 8, 128), (255, 8, 128), (256, 8, 128), (257, 8, 128), (300, 7, 128), (4100, 1, 64)])
@pytest.mark.parametrize("start,rows", [(0, 5000), (3, 5000), (0, 200), (150, 200), (200, 200), (250, 200)])
def test_cache_write(tokens, kv, dim, start, rows):
    k, v = torch.randn(tokens, kv, dim, device="cuda"), torch.randn(tokens, kv, dim, device="cuda")
    kc, vc = (torch.full((rows + 1, kv, dim), 7.0, device="cuda", dtype=torch.float16) for _ in range(2))
    K.launch_copy_to_kv_cache(kc, vc, k, v, tokens, kv, dim, start, rows)
    torch.cuda.synchronize()
    n = max(0, min(tokens, rows - start))                          # rows behind the cache are dropped
    for c, t in ((kc, k), (vc, v)):
        want = torch.full_like(c, 7.0)
        want[start:start + n] = t[:n].half()
        assert torch.equal(c, want)
