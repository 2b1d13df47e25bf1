"""Attention of one decoded token behind the launcher boundary (csrc/attention.cu wave_splits): slices where the groups of heads fill a wave of CTAs and where they do not."""
import pytest

torch = pytest.importorskip("torch")
from ntransformer_b200 import kernels as K  # noqa: E402
from test_prefill_tc_gpu import exact, rel  # noqa: E402

pytestmark = [pytest.mark.gpu]


# 8, 24, 32 and 7 groups; more of them than half a wave has CTAs, and than a wave
@pytest.mark.parametrize("heads,kv,dim", [(32, 8, 128), (24, 8, 128), (32, 32, 128), (14, 7, 64), (160, 160, 64), (301, 301, 64)])
@pytest.mark.parametrize("keys", [64, 65, 97, 1000, 4001])
def test_slices(heads, kv, dim, keys):
    g = torch.Generator(device="cuda").manual_seed(keys)
    q = torch.randn(1, heads, dim, device="cuda", generator=g)
    kc, vc = (torch.randn(keys, kv, dim, device="cuda", generator=g).half() for _ in range(2))
    out = torch.empty_like(q)
    K.launch_attention_decode(out, q, kc, vc, keys, heads, kv, dim, keys, dim ** -0.5)
    torch.cuda.synchronize()
    # weights to 2^-22, sums of at most keys / 8 of them in a run: sqrt of that many roundings of 2^-24
    assert rel(out, exact(q, kc, vc, keys - 1, dim ** -0.5)) <= 2.0**-22 + (keys / 8) ** 0.5 * 2.0**-24


# three CTAs to an SM (narrow heads: as many slices as two of them leave room for, and one more); more groups than half a wave and than three quarters, where slices go by their cost
@pytest.mark.parametrize("heads,kv,dim", [(64, 64, 64), (40, 20, 64), (16, 8, 256), (210, 210, 128), (320, 160, 128), (256, 256, 64), (340, 340, 64)])
@pytest.mark.parametrize("keys", [65, 700, 2000])
def test_slices_by_width_and_cost(heads, kv, dim, keys):
    test_slices(heads, kv, dim, keys)
