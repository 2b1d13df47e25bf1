"""Tokens over GGUF blocks on the tensor cores (csrc/prefill_blocks.cu) through nt_b200_gemm_blocks: the dealing out of tiles, formats side by side, wide ranges of
activations, and the precision of the form that takes a few tokens' place (csrc/gemv_rows.cu, 24-bit integers)."""
import ctypes as C
import dataclasses

import numpy as np
import pytest

torch = pytest.importorskip("torch")
from ntransformer_b200._lib import lib  # noqa: E402
from ntransformer_b200.dtypes import DType  # noqa: E402
from ntransformer_b200.engine import Model  # noqa: E402
from ntransformer_b200.model_spec import TINY  # noqa: E402
from oracle import oracle as O  # noqa: E402
from test_block_products_gpu import FORMATS, activations, arrays, blocks_product, matrix, rel, rows_product, stream  # noqa: E402

pytestmark = [pytest.mark.gpu]


def product(ys, Ws, outs, dts, x, fine=False, add=False, norm_w=None):
    y, w, o, d = arrays(ys, Ws, outs, dts)
    assert lib().nt_b200_gemm_blocks(len(Ws), y, w, o, d, x.shape[1], x.data_ptr(), norm_w.data_ptr() if norm_w is not None else None, 1e-5, x.shape[0], int(fine),
                                     int(add), stream()) == 0
    torch.cuda.synchronize()


def bound(dt, columns):
    """An addition to an accumulator leaves 2/3 of 2^-24 of it: one for 16 columns, twice (two halves of the tokens; a third product's are small), of sums that may
    be twice the result's size where minima are taken off (codes are not centred); pairs of halves and F32 additions leave 2^-22."""
    return 2 * columns // 16 * 2.0 ** -24 * 2 / 3 * (2 if dt in (DType.Q4_K_M, DType.Q5_K) else 1) + 2.0 ** -22


# one tile shared by as many CTAs as it has super-blocks; tiles that start and end inside a CTA's run; more tiles than CTAs; several tiles of tokens; ragged Q6_K
@pytest.mark.parametrize("dt", FORMATS, ids=lambda d: d.name)
@pytest.mark.parametrize("tokens,rows,cols", [(2, 5, 256), (16, 128, 4096), (33, 300, 2816), (129, 257, 4096), (257, 20000, 512), (21, 4096, 14336), (384, 640, 1280)])
@pytest.mark.parametrize("fine", [False, True])
def test_products(dt, tokens, rows, cols, fine):
    W, W64 = matrix(dt, rows, cols, rows)
    x = activations(tokens, cols, cols)
    ref = x.double() @ W64.T
    y = torch.full((tokens + 1, rows), 7.0, device="cuda")
    product([y], [W], [rows], [dt], x, fine)
    assert rel(y[:tokens], ref) <= bound(dt, 64 if fine else 256) and (y[tokens] == 7.0).all()
    again = torch.zeros_like(y)
    product([again], [W], [rows], [dt], x, fine)
    assert torch.equal(again[:tokens], y[:tokens])                 # the shares of a tile are added in one order
    product([y], [W], [rows], [dt], x, fine, add=True)
    assert rel(y[:tokens], 2 * ref) <= bound(dt, 64 if fine else 256) and (y[tokens] == 7.0).all()


@pytest.mark.parametrize("dts", [(DType.Q4_K_M, DType.Q4_K_M, DType.Q6_K), (DType.Q5_K, DType.Q8_0, DType.Q6_K), (DType.Q4_0, DType.Q6_K), (DType.Q6_K, DType.Q5_K)])
@pytest.mark.parametrize("cols", [2048, 1280])
def test_formats_side_by_side_and_norm(dts, cols):
    tokens, outs = 70, [300, 33, 128][: len(dts)]
    mats = [matrix(d, o, cols, o) for d, o in zip(dts, outs)]
    x, g = activations(tokens, cols, 3), 1 + 0.1 * activations(1, cols, 4)[0]
    u = x.double() / (x.double().pow(2).mean(1, keepdim=True) + 1e-5).sqrt() * g.double()
    ys = [torch.zeros(tokens, o, device="cuda") for o in outs]
    product(ys, [m[0] for m in mats], outs, dts, x, norm_w=g)
    for y, d, (_, W64) in zip(ys, dts, mats):
        assert rel(y, u @ W64.T) <= bound(d, 256)


@pytest.mark.parametrize("dt", FORMATS, ids=lambda d: d.name)
def test_activations_of_any_size_and_what_a_nan_reaches(dt):
    tokens, rows, cols = 9, 130, 1024
    W, W64 = matrix(dt, rows, cols, 1)
    x = activations(tokens, cols, 5)
    for t, by in enumerate((1e-20, 1e-6, 0.01, 1.0, 3e4, 1e6, 1e12)):
        x[t] *= by
    x[7] = 0
    x[8, 500] = float("nan")
    y = torch.zeros(tokens, rows, device="cuda")
    product([y], [W], [rows], [dt], x)
    ref = x.double() @ W64.T
    for t in range(7):
        assert rel(y[t], ref[t]) <= bound(dt, 256), t
    assert (y[7] == 0).all() and torch.isnan(y[8]).all()


@pytest.mark.parametrize("dt", [DType.Q4_K_M, DType.Q5_K, DType.Q6_K], ids=lambda d: d.name)      # (Q8_0 and Q4_0 stay with the integers)
@pytest.mark.parametrize("cols", [1024, 4096, 14336])
@pytest.mark.parametrize("wild,by", [(0.0, 1.0), (0.01, 10.0), (0.001, 3000.0)])
def test_a_few_tokens_are_no_further_from_64_bits_than_24_bit_integers(dt, cols, wild, by):
    tokens, rows = 21, 1024
    W, W64 = matrix(dt, rows, cols, 9)
    x = activations(tokens, cols, 10, wild, by) * 0.3
    ref = x.double() @ W64.T
    y, old = torch.zeros(tokens, rows, device="cuda"), torch.zeros(tokens, rows, device="cuda")
    product([y], [W], [rows], [dt], x, fine=True)
    rows_product([old], [W], [rows], [dt], x)
    print("%s %d, %g of them x %g: %.2e here, %.2e integers" % (dt.name, cols, wild, by, rel(y, ref), rel(old, ref)))
    assert rel(y, ref) <= rel(old, ref)


@pytest.mark.parametrize("dt", [DType.Q4_K_M, DType.Q6_K], ids=lambda d: d.name)
@pytest.mark.parametrize("tokens", [9, 21, 70])
def test_a_few_tokens_hold_what_24_bit_integers_hold(dt, tokens):
    """One weight of 1 to a row: the result is a column of the tokens, as the product has it."""
    cols = 512
    rows = cols
    raw = np.zeros((rows, cols // 256, 144 if dt == DType.Q4_K_M else 210), np.uint8)
    one = np.array([1.0], np.float16).view(np.uint8)
    for c in range(cols):
        b, i = raw[c, c // 256], c % 256
        if dt == DType.Q4_K_M:                                     # d = 1, dmin = 0, scales of 1
            b[0:2], b[4:8], b[12:16] = one, 1, 1
            b[16 + i // 64 * 32 + i % 32] = 1 << (4 if i % 64 >= 32 else 0)
        else:                                                      # d = 1, a scale of 1 for these 16 weights and none elsewhere; 33 - 32, 32 - 32
            b[208:210], b[192 + i // 16] = one, 1
            b[128:192] = 0xAA
            h, q = i // 128, i % 128 // 32
            b[64 * h + 32 * (q & 1) + i % 32] = 1 << (4 if q >= 2 else 0)
    raw = raw.reshape(rows, -1)
    assert np.array_equal(O.dequant_rows(int(dt), raw, rows, cols), np.eye(cols, dtype=np.float32))
    x = activations(tokens, cols, 3)
    y = torch.zeros(tokens, rows, device="cuda")
    product([y], [torch.from_numpy(raw).cuda()], [rows], [dt], x, fine=True)
    held = x.abs().reshape(tokens, -1, 32).amax(2, keepdim=True).expand(-1, -1, 32).reshape(tokens, cols) * 2.0 ** -24      # of the 32 columns' largest
    assert ((y - x).abs() <= held).all()


@pytest.mark.parametrize("dt", [DType.Q4_K_M, DType.Q5_K, DType.Q6_K], ids=lambda d: d.name)
def test_a_token_s_product_is_the_same_however_many_share_the_call(dt):
    rows, cols = 1300, 2816
    W, _ = matrix(dt, rows, cols, 7)
    x = activations(64, cols, 8)
    got = []
    for tokens in (9, 16, 31, 64):
        y = torch.zeros(tokens, rows, device="cuda")
        product([y], [W], [rows], [dt], x[:tokens].contiguous(), fine=True)
        got.append(y)
    assert all(torch.equal(y[:9], got[0]) for y in got) and torch.equal(got[3][:31], got[2])


@pytest.mark.parametrize("dt", [DType.Q4_K_M, DType.Q6_K], ids=lambda d: d.name)
@pytest.mark.parametrize("tokens", [700, 1025])
def test_long_runs_go_through_the_kept_memory_in_portions(dt, tokens):
    """14336 columns: 700 tokens are the most that the memory a device keeps between calls takes, or two portions with the third halves."""
    rows, cols = 130, 14336
    W, W64 = matrix(dt, rows, cols, 11)
    x = activations(tokens, cols, 12)
    ref = x.double() @ W64.T
    for fine in (False, True):
        y = torch.full((tokens + 1, rows), 7.0, device="cuda")
        product([y], [W], [rows], [dt], x, fine)
        assert rel(y[:tokens], ref) <= bound(dt, 64 if fine else 256) and (y[tokens] == 7.0).all()
    y = torch.full((tokens + 1, rows), 7.0, device="cuda")
    blocks_product([y], [W], [rows], [dt], x)
    blocks_product([y], [W], [rows], [dt], x, add=True)
    assert rel(y[:tokens], 2 * ref) <= bound(dt, 256) and (y[tokens] == 7.0).all()


@pytest.mark.parametrize("dt", [DType.Q4_K_M, DType.Q6_K], ids=lambda d: d.name)
def test_captured(dt):
    tokens, rows, cols = 40, 300, 2048
    W, _ = matrix(dt, rows, cols, 1)
    x = activations(tokens, cols, 2)
    ws = torch.empty(lib().nt_b200_gemm_f16_tc_workspace_bytes(tokens, cols), dtype=torch.uint8, device="cuda")
    lib().nt_b200_split_activations(ws.data_ptr(), x.data_ptr(), tokens, cols, stream())
    ys = [torch.zeros(tokens, rows, device="cuda") for _ in range(4)]
    want = [torch.zeros(tokens, rows, device="cuda") for _ in range(2)]

    def calls(a, b):
        for y, of_ws in ((a, False), (b, True)):
            c, w, o, d = arrays([y], [W], [rows], [dt])
            if of_ws:
                assert lib().nt_b200_gemm_blocks_ws(1, c, w, o, d, cols, ws.data_ptr(), tokens, 0, stream()) == 0
            else:
                assert lib().nt_b200_gemm_blocks(1, c, w, o, d, cols, x.data_ptr(), None, 0.0, tokens, 1, 0, stream()) == 0

    calls(*want)
    torch.cuda.synchronize()
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=side):
        calls(ys[0], ys[1])
        calls(ys[2], ys[3])
    for _ in range(3):
        for y in ys:
            y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(y, want[i & 1]) for i, y in enumerate(ys))


@pytest.mark.parametrize("mix", ["Q4_K_M", "Q8_0"])
def test_prompts_of_other_lengths_before_leave_nothing_behind(mix):
    """The counts of a product's shared tiles lie in the tokens' workspace, where other lengths have other numbers: each split clears them."""
    cfg = dataclasses.replace(TINY, max_seq_len=1024)
    toks = np.random.default_rng(4).integers(3, cfg.vocab_size, size=700).tolist()
    m = Model.synthetic(cfg, mix, seed=6)
    want = {}
    for n in (130, 40, 11, 300, 33, 130, 20, 11, 700, 40, 300, 20, 33, 700):
        got = m.forward(toks[:n], 0).copy()
        assert np.array_equal(want.setdefault(n, got), got), n
    m.close()
