"""Tokens over F16 and BF16 matrices dealt out over all SMs (csrc/prefill_dense.cu): the edges of tiles of tokens and rows, tiles shared by several CTAs, layer scales and
residuals; and a few tokens of whole models through it against the same tokens one decode step at a time."""
import ctypes as C
import dataclasses

import numpy as np
import pytest

torch = pytest.importorskip("torch")
from ntransformer_b200 import kernels as K  # noqa: E402
from ntransformer_b200._lib import lib  # noqa: E402
from ntransformer_b200.dtypes import DType  # noqa: E402
from ntransformer_b200.engine import Model  # noqa: E402
from ntransformer_b200.model_spec import TINY  # noqa: E402
from test_block_products_gpu import activations, rel, stream  # noqa: E402
from test_short_prompt_gpu import ODD, both  # noqa: E402

pytestmark = [pytest.mark.gpu]


def product(ys, Ws, x, dtype, fine, add=False, norm_w=None, col_scale=None, alpha=1.0):
    n = len(ys)
    y, w, o = (C.c_void_p * n)(*[t.data_ptr() for t in ys]), (C.c_void_p * n)(*[t.data_ptr() for t in Ws]), (C.c_int * n)(*[t.shape[0] for t in Ws])
    ptr = lambda t: None if t is None else t.data_ptr()   # noqa: E731
    rc = lib().nt_b200_gemm_dense_tc(n, y, w, o, int(dtype), x.shape[1], x.data_ptr(), ptr(norm_w), 1e-5, x.shape[0], int(fine), int(add), ptr(col_scale), alpha, stream())
    torch.cuda.synchronize()
    return rc


def bound(dtype, fine):
    """What the parts of an activation leave of it (11 bits each of F16, 8 of BF16); an addition to an accumulator, one for 16 columns, cuts off at most 2^-23 of what it holds
    (5 results of one token: nothing averages); F32 sums."""
    parts = {(DType.F16, False): 2.0 ** -22, (DType.F16, True): 2.0 ** -24, (DType.BF16, False): 2.0 ** -16, (DType.BF16, True): 2.0 ** -24}[dtype, bool(fine)]
    return parts + (64 if fine else 256) / 16 * 2.0 ** -23 + 2.0 ** -22


@pytest.mark.parametrize("dtype,torch_type", [(DType.F16, torch.float16), (DType.BF16, torch.bfloat16)], ids=["F16", "BF16"])
@pytest.mark.parametrize("fine", [False, True])
@pytest.mark.parametrize("tokens", [1, 16, 17, 80, 81, 128, 129, 300])
@pytest.mark.parametrize("rows,cols", [((5,), 256), ((128, 300, 33), 768), ((2000,), 512), ((257, 130), 4096)])
def test_products(dtype, torch_type, fine, tokens, rows, cols):
    g = torch.Generator(device="cuda").manual_seed(tokens + cols)
    Ws = [(torch.randn(r, cols, generator=g, device="cuda") * cols ** -0.5).to(torch_type) for r in rows]
    x, gains = activations(tokens, cols, cols + tokens), 1 + 0.1 * activations(1, cols, 4)[0]
    u = x.double() / (x.double().pow(2).mean(1, keepdim=True) + 1e-5).sqrt() * gains.double()
    ys = [torch.full((tokens + 1, r), 7.0, device="cuda") for r in rows]
    assert product(ys, Ws, x, dtype, fine, norm_w=gains) == 0
    for y, W in zip(ys, Ws):
        # (the norm itself is F32: a few roundings more)
        assert rel(y[:tokens], u @ W.double().T) <= bound(dtype, fine) + 2.0 ** -22 and (y[tokens] == 7.0).all()
    scale = 1 + activations(1, rows[0], 9)[0].abs()
    y, again = (torch.full((tokens + 1, rows[0]), 3.0, device="cuda") for _ in range(2))
    for t in (y, again):
        assert product([t], Ws[:1], x, dtype, fine, add=True, col_scale=scale, alpha=-0.5) == 0
    ref = 3.0 - 0.5 * (x.double() @ Ws[0].double().T) * scale.double()
    assert rel(y[:tokens], ref) <= bound(dtype, fine) and (y[tokens] == 3.0).all()
    assert torch.equal(y, again)                                   # the shares of a tile are added in one order


def test_what_is_refused():
    W, x, y = torch.zeros(64, 320, device="cuda").half(), torch.zeros(4, 320, device="cuda"), torch.full((4, 64), 7.0, device="cuda")
    assert product([y], [W], x, DType.F16, True) < 0 and (y == 7.0).all()                       # columns that are no multiple of 256
    W, x = torch.zeros(64 * 256 + 8, device="cuda").half()[4:4 + 64 * 256].view(64, 256), torch.zeros(4, 256, device="cuda")
    assert product([y], [W], x, DType.F16, True) < 0 and (y == 7.0).all()                       # rows off 16 bytes
    assert product([y], [W], x, DType.F32, True) < 0 and (y == 7.0).all()


def one_by_one(W, x, dtype):
    y = torch.zeros(x.shape[0], W.shape[0], device="cuda")
    for t in range(x.shape[0]):
        lib().nt_b200_gemv_dense(y[t].data_ptr(), None, None, W.data_ptr(), None, None, W.shape[0], 0, 0, 1, W.shape[1], x[t].data_ptr(), int(dtype), 0, None, 1.0, stream())
    torch.cuda.synchronize()
    return y


# against the same tokens a GEMV at a time, F32 sums: the form that the fine one took the place of (the plain one is at 2 to 20 times its error).
# Where one product is most of a short row's sum the order of additions decides: 1024 columns, one number in a thousand 3000 times the others, 1.20e-7 here and 1.05e-7 there.
@pytest.mark.parametrize("dtype,torch_type", [(DType.F16, torch.float16), (DType.BF16, torch.bfloat16)], ids=["F16", "BF16"])
@pytest.mark.parametrize("cols,wild,by", [(c, w, b) for c in (512, 1024, 4096, 14336) for w, b in ((0.0, 1.0), (0.01, 10.0))] + [(4096, 0.001, 3000.0), (14336, 0.001, 3000.0)])
def test_fine_is_as_exact_as_one_by_one(dtype, torch_type, cols, wild, by):
    g = torch.Generator(device="cuda").manual_seed(cols)
    W, x = (torch.randn(700, cols, generator=g, device="cuda") * cols ** -0.5).to(torch_type), activations(21, cols, 6, wild, by)
    y, ref = torch.zeros(21, 700, device="cuda"), x.double() @ W.double().T
    assert product([y], [W], x, dtype, True) == 0
    assert rel(y, ref) <= 1.05 * rel(one_by_one(W, x, dtype), ref)


# rows with a single weight of 1 give a token's numbers back: all 24 bits of them, but for what lies below 2^-24 of F16 once a token's largest is at 2^13 to 2^14
@pytest.mark.parametrize("dtype,torch_type", [(DType.F16, torch.float16), (DType.BF16, torch.bfloat16)], ids=["F16", "BF16"])
def test_fine_keeps_every_bit(dtype, torch_type):
    x = activations(9, 1024, 8, 0.01, 1000.0)
    x[1] *= 1e-12
    x[2] *= 1e12
    at = torch.randperm(1024, generator=torch.Generator().manual_seed(1))[:300].cuda()
    W = torch.zeros(300, 1024, device="cuda").to(torch_type)
    W[torch.arange(300, device="cuda"), at] = 1
    y = torch.zeros(9, 300, device="cuda")
    assert product([y], [W], x, dtype, True) == 0
    left = (y.double() - x[:, at].double()).abs()
    assert (left <= x.abs().amax(1, keepdim=True).double() * (2.0 ** -37 if dtype == DType.F16 else 0.0)).all()


@pytest.mark.parametrize("n,before", [(2, 0), (17, 5), (31, 40)])
def test_f16_tokens_together_equal_one_by_one(n, before):
    toks = np.random.default_rng(n).integers(0, ODD.vocab_size, size=n + before).tolist()
    both(ODD, "F16", toks[:before], toks[before:], sorted({0, n // 2, n - 1}))


@pytest.mark.parametrize("hidden,inter", [(640, 1280), (512, 1056)])
def test_f16_shapes_that_are_not_taken_run_one_by_one(hidden, inter):
    cfg = dataclasses.replace(TINY, hidden_size=hidden, intermediate_size=inter, n_heads=hidden // 64, n_kv_heads=hidden // 128, head_dim=64, vocab_size=520)
    m = Model.synthetic(cfg, "F16", seed=5)
    a = m.forward_logits([5, 6, 7], 0, [2]).copy()
    m.set_prefill_min_tokens(0)
    b = m.forward_logits([5, 6, 7], 0, [2])
    assert np.array_equal(a, b)
    m.close()


@pytest.mark.parametrize("n,before", [(3, 4), (15, 30)])
def test_bf16_family_tokens_together_equal_one_by_one(n, before):
    g = torch.Generator(device="cuda").manual_seed(3)
    W, ff, heads, kv = 512, 768, 4, 2
    mixer = {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 30.0, "mask": {"size": 16, "keep_first": 4}}
    cfg = {"architecture": "Zelunex", "vocab": 300, "width": W, "norm": {"eps": 1e-5}, "residual_mult": 0.5,
           "layers": [{"type": "attention", "mixer": mixer, "mlp": {"kind": "dense", "ff": ff}} for _ in range(2)]}
    mat = lambda r, c, std: (torch.randn(r, c, generator=g, device="cuda") * std).bfloat16()   # noqa: E731
    vec = lambda k: 1 + 0.1 * torch.randn(k, generator=g, device="cuda")   # noqa: E731
    t = {"embed": mat(300, W, 1.0), "final.norm": vec(W), "head": mat(300, W, W ** -0.5)}
    for i in range(2):
        p = "l%d." % i
        t.update({p + "norm1": vec(W), p + "mix.q": mat(512, W, W ** -0.5), p + "mix.k": mat(256, W, W ** -0.5), p + "mix.v": mat(256, W, W ** -0.5), p + "mix.q.norm": vec(512),
                  p + "mix.k.norm": vec(256), p + "mix.o": mat(W, 512, 512 ** -0.5), p + "ls1": vec(W), p + "mlp.gate": mat(ff, W, W ** -0.5), p + "mlp.up": mat(ff, W, W ** -0.5),
                  p + "mlp.down": mat(W, ff, ff ** -0.5), p + "ls2": vec(W)})
    toks = np.random.default_rng(n).integers(0, 300, size=n + before).tolist()
    out = []
    for together in (True, False):
        m = Model.from_config_json(cfg, dict(t), max_context=128)
        m.set_prefill_min_tokens(16 if together else 0)
        m.forward_logits(toks[:before], 0, [])
        n0 = K.launch_count()
        out.append((m.forward_logits(toks[before:], before, [0, n - 1]).copy(), K.launch_count() - n0))
        m.close()
    (a, na), (b, nb) = out
    assert na < nb, "the tokens ran one at a time"
    # products of 24 bits either way; sums in another order may round a cached key or value to its other BF16 neighbour (2^-8 of it)
    assert np.abs(a - b).max() <= 2e-3 * np.abs(b).max(), np.abs(a - b).max() / np.abs(b).max()
