"""The two matrix kernels for several tokens over GGUF blocks, called directly, against 64 bits: csrc/gemv_rows.cu (a few tokens, 24-bit integers) and
csrc/prefill_blocks.cu (prompts, pairs of F16 on the tensor cores); and the precision of what took an earlier form's place against that form."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
from ntransformer_b200 import kernels as K  # noqa: E402
from ntransformer_b200._lib import lib  # noqa: E402
from ntransformer_b200.dtypes import DType  # noqa: E402
from ntransformer_b200.synth import random_blocks_np  # noqa: E402
from oracle import oracle as O  # noqa: E402

pytestmark = [pytest.mark.gpu]
FORMATS = [DType.Q4_K_M, DType.Q5_K, DType.Q6_K, DType.Q8_0, DType.Q4_0]


def stream():
    return torch.cuda.current_stream().cuda_stream


def matrix(dt, rows, cols, seed):
    raw = random_blocks_np(dt, rows, cols, np.random.default_rng(seed))
    return torch.from_numpy(raw).cuda(), torch.from_numpy(O.dequant_rows(int(dt), raw, rows, cols)).cuda().double()


def activations(tokens, cols, seed, wild=0.02, by=10.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(tokens, cols, device="cuda", generator=g)
    return x * torch.where(torch.rand(tokens, cols, device="cuda", generator=g) < wild, by, 1.0)


def arrays(ys, Ws, outs, dts):
    n = len(Ws)
    return (C.c_void_p * n)(*[y.data_ptr() for y in ys]), (C.c_void_p * n)(*[w.data_ptr() for w in Ws]), (C.c_int * n)(*outs), (C.c_int * n)(*map(int, dts))


def rows_product(ys, Ws, outs, dts, x, epilogue=0, norm_w=None):
    tokens, cols = x.shape
    scratch = torch.empty(lib().nt_b200_gemv_rows_bytes(tokens, cols), dtype=torch.uint8, device="cuda")
    y, w, o, d = arrays(ys, Ws, outs, dts)
    assert lib().nt_b200_gemv_rows(len(Ws), y, w, o, d, cols, x.data_ptr(), norm_w.data_ptr() if norm_w is not None else None, 1e-5, tokens, scratch.data_ptr(), epilogue,
                                   stream()) == 0
    torch.cuda.synchronize()


def blocks_product(Cs, Ws, outs, dts, x, add=False):
    tokens, cols = x.shape
    ws = torch.empty(lib().nt_b200_gemm_f16_tc_workspace_bytes(tokens, cols), dtype=torch.uint8, device="cuda")
    lib().nt_b200_split_activations(ws.data_ptr(), x.data_ptr(), tokens, cols, stream())
    c, w, o, d = arrays(Cs, Ws, outs, dts)
    assert lib().nt_b200_gemm_blocks_ws(len(Ws), c, w, o, d, cols, ws.data_ptr(), tokens, int(add), stream()) == 0
    torch.cuda.synchronize()


def rel(got, ref):
    return float(((got.double() - ref).norm() / ref.norm()).item())


# tokens: one pass of 8, its remainders, several; rows around tiles of 16 and 32; one, a stage's 8 and more super-blocks, an odd number (Q6_K at any even address)
@pytest.mark.parametrize("dt", FORMATS, ids=lambda d: d.name)
@pytest.mark.parametrize("tokens,rows,cols", [(2, 33, 256), (8, 16, 2048), (9, 100, 2304), (31, 4743, 768), (64, 40, 11008)])
def test_few_tokens(dt, tokens, rows, cols):
    W, W64 = matrix(dt, rows, cols, rows)
    x = activations(tokens, cols, cols)
    ref = x.double() @ W64.T
    # 24-bit integers (2^-24 of a 32-block's largest), exact products, F32 sums over super-blocks: the bound of the single token's test
    bound = 4e-6 * x.abs().max().item() * cols ** 0.5 * 0.02
    y = torch.full((tokens + 1, rows), 7.0, device="cuda")
    rows_product([y], [W], [rows], [dt], x)
    assert (y[:tokens].double() - ref).abs().max().item() <= bound and (y[tokens] == 7.0).all()
    rows_product([y], [W], [rows], [dt], x, epilogue=1)
    assert (y[:tokens].double() - 2 * ref).abs().max().item() <= 2 * bound and (y[tokens] == 7.0).all()


@pytest.mark.parametrize("dts", [(DType.Q4_K_M, DType.Q4_K_M, DType.Q6_K), (DType.Q4_K_M, DType.Q5_K), (DType.Q4_0, DType.Q6_K)])
def test_few_tokens_several_matrices_and_norm(dts):
    tokens, cols, outs = 21, 1536, [64, 33, 100][: len(dts)]
    mats = [matrix(d, o, cols, o) for d, o in zip(dts, outs)]
    x, g = activations(tokens, cols, 3), 1 + 0.1 * activations(1, cols, 4)[0]
    u = x.double() / (x.double().pow(2).mean(1, keepdim=True) + 1e-5).sqrt() * g.double()
    ys = [torch.zeros(tokens, o, device="cuda") for o in outs]
    rows_product(ys, [m[0] for m in mats], outs, dts, x, norm_w=g)
    for y, (_, W64) in zip(ys, mats):
        assert rel(y, u @ W64.T) <= 2e-6


@pytest.mark.parametrize("dt", FORMATS, ids=lambda d: d.name)
def test_few_tokens_swiglu_and_what_a_nan_reaches(dt):
    tokens, rows, cols = 11, 70, 1024
    (G, G64), (U, U64) = matrix(dt, rows, cols, 1), matrix(dt, rows, cols, 2)
    x = activations(tokens, cols, 5)
    y = torch.zeros(tokens, rows, device="cuda")
    rows_product([y, y], [G, U], [rows, rows], [dt, dt], x, epilogue=2)
    assert rel(y, torch.nn.functional.silu(x.double() @ G64.T) * (x.double() @ U64.T)) <= 4e-6       # two products, and the fast-math sigmoid
    x[3, 500] = float("nan")
    rows_product([y], [G], [rows], [dt], x)
    assert torch.isnan(y[3]).all() and torch.isfinite(y[:3]).all() and torch.isfinite(y[4:]).all()


def cut(cols):
    """Three products for 16 columns of half the row, at most 2048: each addition to an accumulator is cut by half a unit (2^-24 of the sum so far) on average and
    always to one side, over sums that grow to the accumulator's: 2/3 of 2^-24 each; F32 additions of the partial sums and pairs of halves add 2^-21."""
    return 3 * -(-min(2048, cols / 2) // 16) * 2.0 ** -24 * 2 / 3 + 2.0 ** -21


# tokens around the tile widths (multiples of 16 up to 128, several column tiles), rows around 128, K of one and of several super-blocks
@pytest.mark.parametrize("dt", FORMATS, ids=lambda d: d.name)
@pytest.mark.parametrize("tokens,rows,cols", [(17, 100, 256), (113, 129, 2304), (256, 128, 4096), (300, 1000, 768), (500, 384, 11008)])
def test_prompt(dt, tokens, rows, cols):
    W, W64 = matrix(dt, rows, cols, rows)
    x = activations(tokens, cols, cols)
    ref = x.double() @ W64.T
    y = torch.full((tokens + 1, rows), 7.0, device="cuda")
    blocks_product([y], [W], [rows], [dt], x)
    assert rel(y[:tokens], ref) <= cut(cols) and (y[tokens] == 7.0).all()
    blocks_product([y], [W], [rows], [dt], x, add=True)
    assert rel(y[:tokens], 2 * ref) <= cut(cols) and (y[tokens] == 7.0).all()


def test_prompt_several_matrices():
    tokens, cols, outs, dts = 77, 2048, [256, 64, 130], [DType.Q4_K_M, DType.Q4_K_M, DType.Q6_K]
    mats = [matrix(d, o, cols, o) for d, o in zip(dts, outs)]
    x = activations(tokens, cols, 8)
    ys = [torch.zeros(tokens, o, device="cuda") for o in outs]
    blocks_product(ys, [m[0] for m in mats], outs, dts, x)
    for y, (_, W64) in zip(ys, mats):
        assert rel(y, x.double() @ W64.T) <= cut(cols)


@pytest.mark.parametrize("dt", FORMATS, ids=lambda d: d.name)
@pytest.mark.parametrize("tokens,rows,cols", [(64, 512, 256), (64, 512, 1024), (100, 512, 2048), (64, 512, 2304), (64, 512, 3072), (500, 1024, 4096),
                                              (200, 512, 14336)])
@pytest.mark.parametrize("scale", [1.0, 0.05])
def test_prompt_is_no_further_from_64_bits_than_the_expanded_form(dt, tokens, rows, cols, scale):
    """Before: the matrix written out as two F16 matrices and two GEMMs over them, all four products of halves, 4096 columns to an accumulator."""
    W, W64 = matrix(dt, rows, cols, 9)
    x = activations(tokens, cols, 10, by=10.0) * scale
    ref = x.double() @ W64.T
    y, old = torch.zeros(tokens, rows, device="cuda"), torch.zeros(tokens, rows, device="cuda")
    blocks_product([y], [W], [rows], [dt], x)
    hi, lo = torch.zeros(rows, cols, dtype=torch.float16, device="cuda"), torch.zeros(rows, cols, dtype=torch.float16, device="cuda")
    ws = torch.empty(lib().nt_b200_gemm_f16_tc_workspace_bytes(tokens, cols), dtype=torch.uint8, device="cuda")
    lib().nt_b200_split_activations(ws.data_ptr(), x.data_ptr(), tokens, cols, stream())
    lib().nt_b200_dequant_split(hi.data_ptr(), lo.data_ptr(), W.data_ptr(), int(dt), 0, rows, cols, stream())
    for half, add in ((hi, 0), (lo, 1)):
        assert lib().nt_b200_gemm_f16_tc_ws(old.data_ptr(), ws.data_ptr(), half.data_ptr(), tokens, rows, cols, add, stream()) == 0
    torch.cuda.synchronize()
    print("%s %d x %d x %d, activations x %g: %.2e here, %.2e expanded" % (dt.name, tokens, rows, cols, scale, rel(y, ref), rel(old, ref)))
    assert rel(y, ref) <= 1.02 * rel(old, ref)


@pytest.mark.parametrize("dt,cols", [(DType.Q4_0, 1024), (DType.Q4_0, 4096), (DType.Q4_0, 14336), (DType.Q6_K, 1280), (DType.Q6_K, 11008)], ids=str)
@pytest.mark.parametrize("wild,by", [(0.0, 1.0), (0.01, 10.0), (0.01, 100.0)])       # the tracked workloads' activations, without and with wilder ones
def test_single_token_is_no_further_from_64_bits_than_the_general_path(dt, cols, wild, by):
    """Q4_0, and Q6_K rows off 16 bytes, were multiplied by the F32 vector (the path that a vector off 16 bytes still takes).  Q4_0 takes 32-bit integers of the
    activations, Q6_K 24-bit ones: 2^-24 of a 32-block's largest number, so one far above its neighbours (a hundred times) costs it more than F32."""
    if dt == DType.Q6_K and by > 10:
        pytest.skip("24-bit integers of a block")
    rows = 2048
    W, W64 = matrix(dt, rows, cols, 13)
    x = activations(1, cols + 1, 14, wild, by)[0]
    y, old = torch.zeros(rows, device="cuda"), torch.zeros(rows, device="cuda")
    off = torch.empty(cols + 1, device="cuda")
    off[1:] = x[:cols]
    K.launch_gemv(y, W, x[:cols], rows, cols, dt)
    K.launch_gemv(old, W, off.data_ptr() + 4, rows, cols, dt)
    torch.cuda.synchronize()
    ref = W64 @ x[:cols].double()
    print("%s %d x %d, %g of them x %g: %.2e here, %.2e general" % (dt.name, rows, cols, wild, by, rel(y, ref), rel(old, ref)))
    assert rel(y, ref) <= 1.02 * rel(old, ref)
