"""The GEMM over blocks in its form for up to 32 tokens (csrc/prefill_blocks.cu, gemm_blocks_few_kernel): the edges of its token tiles, runs of a single super-block, tiles
shared by several CTAs, and formats with and without minima in one launch."""
import pytest

torch = pytest.importorskip("torch")
from ntransformer_b200.dtypes import DType  # noqa: E402
from test_block_products_gpu import FORMATS, activations, matrix, rel, rows_product  # noqa: E402
from test_block_tokens_gpu import bound, product  # noqa: E402

pytestmark = [pytest.mark.gpu]


@pytest.mark.parametrize("dts", [(d,) for d in FORMATS] + [(DType.Q4_K_M, DType.Q4_K_M, DType.Q6_K), (DType.Q6_K, DType.Q5_K), (DType.Q8_0, DType.Q4_K_M, DType.Q4_0)],
                         ids=lambda d: "+".join(t.name for t in d))
@pytest.mark.parametrize("tokens", [1, 16, 17, 32, 33])
@pytest.mark.parametrize("rows,cols", [(128, 256), (300, 512), (129, 7168), (20000, 512)])
def test_products(dts, tokens, rows, cols):
    outs = [rows, 33, 128][: len(dts)]
    mats = [matrix(d, o, cols, o) for d, o in zip(dts, outs)]
    x = activations(tokens, cols, cols + tokens)
    ys = [torch.full((tokens + 1, o), 7.0, device="cuda") for o in outs]
    product(ys, [m[0] for m in mats], outs, dts, x, fine=True)
    for y, d, (_, W64) in zip(ys, dts, mats):
        assert rel(y[:tokens], x.double() @ W64.T) <= bound(d, 64) and (y[tokens] == 7.0).all()


# formats without minima side by side: one kernel with those that have them, but no columns of tensor memory for their sums (3 stages of 16 tokens fill it to 480 of 512)
@pytest.mark.parametrize("dts", [(DType.Q8_0, DType.Q4_0), (DType.Q4_0, DType.Q6_K), (DType.Q6_K, DType.Q8_0), (DType.Q8_0, DType.Q6_K, DType.Q4_0)], ids=lambda d: "+".join(t.name for t in d))
@pytest.mark.parametrize("tokens", [1, 9, 16, 17, 32])
@pytest.mark.parametrize("rows,cols", [(128, 256), (300, 4096), (20000, 512)])
def test_formats_without_minima_side_by_side(dts, tokens, rows, cols):
    test_products(dts, tokens, rows, cols)


# tokens in blocks whose weights are pairs of halves: together from 9 (large matrices) and 17 tokens on, as exact as gemv_rows' 24-bit integers
@pytest.mark.parametrize("dt", [DType.Q8_0, DType.Q4_0], ids=lambda d: d.name)
@pytest.mark.parametrize("tokens,cols", [(9, 4096), (31, 14336)])
def test_pairs_are_as_exact_as_integers(dt, tokens, cols):
    W, W64 = matrix(dt, 700, cols, 3)
    x = activations(tokens, cols, 5, wild=0.01)
    ys = [torch.zeros(tokens, 700, device="cuda") for _ in range(2)]
    product(ys[:1], [W], [700], [dt], x, fine=True)
    rows_product(ys[1:], [W], [700], [dt], x)
    ref = x.double() @ W64.T
    assert rel(ys[0], ref) <= 1.05 * rel(ys[1], ref)
