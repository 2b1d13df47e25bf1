"""Windowed attention where lanes share a key row, at the edges of its groups, against 64 bits and against the general path (the same numbers off
16 bytes)."""
import numpy as np
import pytest
import torch

from ntransformer_b200._lib import lib
from ntransformer_b200.dtypes import DType

pytestmark = pytest.mark.gpu


def stream():
    return torch.cuda.current_stream().cuda_stream


def off_16_bytes(t):
    """the same numbers one element behind a 16-byte boundary"""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")
    buf[1:] = t.reshape(-1)
    return buf[1:].view(t.shape)


# widths: 8, 16 and 32 lanes to a row, the last lanes idle in keys or in values; keys: a group of 32 / 16 / 8 rows and one more, several groups a warp
@pytest.mark.parametrize("dim,vdim", [(8, 64), (64, 40), (72, 128), (128, 64), (136, 256), (256, 8)])
@pytest.mark.parametrize("tokens,total,window,keep,cap", [(1, 1, 0, 0, 0.0), (1, 33, 0, 0, 5.0), (1, 700, 300, 5, 30.0), (3, 129, 17, 9, 0.0), (5, 1100, 0, 0, 0.0)])
def test_attention_window_shared_rows(dim, vdim, tokens, total, window, keep, cap):
    heads, kv = 6, 2
    g = torch.Generator(device="cuda").manual_seed(dim + total)
    Q = torch.randn(tokens, heads, dim, device="cuda", generator=g)
    k = torch.randn(total, kv, dim, device="cuda", generator=g).bfloat16()
    v = torch.randn(total, kv, vdim, device="cuda", generator=g).bfloat16()
    scale = dim ** -0.5

    def run(kc, vc):
        out = torch.zeros(tokens, heads, vdim, device="cuda")
        lib().nt_b200_attention_window(out.data_ptr(), Q.data_ptr(), kc.data_ptr(), vc.data_ptr(), int(DType.BF16), tokens, total - tokens, heads, kv, dim, vdim,
                                       window, keep, scale, cap, total, stream())
        torch.cuda.synchronize()
        return out.double().cpu().numpy()

    i = torch.arange(total - tokens, total, device="cuda")[:, None]
    j = torch.arange(total, device="cuda")[None]
    seen = (j <= i) & ((i - j < window) | (j < keep) | (window == 0))
    s = torch.einsum("thd,shd->hts", Q.double(), k.double().repeat_interleave(heads // kv, 1)) * scale
    s = cap * torch.tanh(s / cap) if cap else s
    ref = torch.einsum("hts,shd->thd", torch.softmax(s.masked_fill(~seen, -np.inf), -1), v.double().repeat_interleave(heads // kv, 1)).cpu().numpy()
    # a score of magnitude below 8 carries dim additions of 2^-24 and tanh's few ulp, a weight twice that; values are below 5
    tol = 5 * 2 * (dim + 32) * 8 * 2.0 ** -24
    assert np.abs(run(k, v) - ref).max() <= tol
    assert np.abs(run(off_16_bytes(k), off_16_bytes(v)) - ref).max() <= tol
