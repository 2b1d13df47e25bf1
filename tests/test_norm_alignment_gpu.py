"""Gains of a norm at any address of a float: a borrowed tensor lies wherever its owner has it, and the fused forms read 16 bytes at a time."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from ntransformer_b200._lib import lib  # noqa: E402
from ntransformer_b200.dtypes import DType  # noqa: E402
from ntransformer_b200.engine import Model  # noqa: E402
from ntransformer_b200.model_spec import TINY  # noqa: E402
from test_block_products_gpu import activations, arrays, matrix, stream  # noqa: E402

pytestmark = [pytest.mark.gpu]


def shifted(t, floats):
    room = torch.empty(t.numel() + 4, device="cuda")
    room[floats:floats + t.numel()] = t.reshape(-1)
    return room[floats:floats + t.numel()]


@pytest.mark.parametrize("mix", ["Q4_K_M", "Q8_0", "F16"])
@pytest.mark.parametrize("tokens", [1, 5, 21, 40])
def test_model(mix, tokens):
    m = Model.synthetic(TINY, mix, seed=3)
    toks = np.random.default_rng(tokens).integers(3, TINY.vocab_size, size=tokens + 7).tolist()
    off = {n: (shifted(v[0], 2 if "attn" in n else 1), *v[1:]) if n.endswith("norm.weight") else v for n, v in m._keep.items()}
    m2 = Model.from_device_tensors(TINY, off)
    out = []
    for x in (m, m2):
        x.forward(toks[:7], 0)
        out.append(x.forward(toks[7:], 7).copy())
        x.close()
    # one step's norm and quantiser are launches of their own then: sums in another order (1e-6), which rounds cached keys and values now and then to the other side
    assert np.abs(out[0] - out[1]).max() <= 3e-4 * np.abs(out[0]).max()


@pytest.mark.parametrize("floats", [1, 2, 3])
def test_tokens_over_blocks(floats):
    tokens, rows, cols = 33, 300, 2048
    W, _ = matrix(DType.Q4_K_M, rows, cols, 1)
    x, g = activations(tokens, cols, 3), 1 + 0.1 * activations(1, cols, 4)[0]
    got = []
    for norm in (g, shifted(g, floats)):
        y = torch.zeros(tokens, rows, device="cuda")
        a, w, o, d = arrays([y], [W], [rows], [DType.Q4_K_M])
        assert lib().nt_b200_gemm_blocks(1, a, w, o, d, cols, x.data_ptr(), norm.data_ptr(), 1e-5, tokens, 0, 0, stream()) == 0
        torch.cuda.synchronize()
        got.append(y)
    assert torch.equal(*got)


def test_the_fused_gemv_refuses_what_it_cannot_read():
    W, _ = matrix(DType.Q4_K_M, 64, 512, 1)
    x, g, y = activations(1, 512, 3)[0], activations(1, 512, 4)[0], torch.zeros(64, device="cuda")
    a, w, o, d = arrays([y], [W], [64], [DType.Q4_K_M])
    for xx, gg in ((shifted(x, 2), g), (x, shifted(g, 1))):
        assert lib().nt_b200_gemv_fused_f32(1, a, w, o, d, 512, xx.data_ptr(), gg.data_ptr(), 1e-5, 0, stream()) == -2
    scratch = torch.empty(lib().nt_b200_gemv_rows_bytes(1, 512), dtype=torch.uint8, device="cuda")
    assert lib().nt_b200_gemv_rows(1, a, w, o, d, 512, x.data_ptr(), shifted(g, 1).data_ptr(), 1e-5, 1, scratch.data_ptr(), 0, stream()) == -2
