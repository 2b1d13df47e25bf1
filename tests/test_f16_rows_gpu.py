"""One vector times F16 rows behind the launcher boundary (csrc/dense.cu): how many warps share a row, rows that end inside a piece of work, matrices with many rounds to a CTA."""
import pytest

torch = pytest.importorskip("torch")
from ntransformer_b200._lib import lib  # noqa: E402
from ntransformer_b200.dtypes import DType  # noqa: E402
from test_block_products_gpu import activations, rel, stream  # noqa: E402

pytestmark = [pytest.mark.gpu]


# one row; eight, four, two and one warps to a row; fewer columns than a warp's piece of work; rows of 3 and of 1.1 pieces of work; long rows; more than sixteen rounds
@pytest.mark.parametrize("rows,cols", [(1, 28672), (17, 28672), (150, 8192), (300, 5000), (600, 4096), (1184, 2048), (5, 8), (33, 1128), (700, 16392), (5000, 16384), (80000, 512)])
@pytest.mark.parametrize("dt,torch_type", [(DType.F16, torch.float16)])
def test_products(rows, cols, dt, torch_type):
    g = torch.Generator(device="cuda").manual_seed(rows)
    W = (torch.randn(rows, cols, generator=g, device="cuda") * cols ** -0.5).to(torch_type)
    x = activations(1, cols, cols)[0]
    y = torch.full((rows + 1,), 7.0, device="cuda")
    lib().nt_b200_gemv(y.data_ptr(), W.data_ptr(), x.data_ptr(), rows, cols, int(dt), stream())
    torch.cuda.synchronize()
    # F32 sums of cols products, 32 lanes of each row by themselves
    assert rel(y[:rows], W.double() @ x.double()) <= (cols / 32) ** 0.5 * 2.0 ** -24 + 2.0 ** -22 and y[rows] == 7.0


# rows of three pieces: few, many, and a little more than a round of gemv_dense's, with and without what is there already
@pytest.mark.parametrize("rows,cols", [(4095, 2304), (4096, 2304), (9000, 2560), (4736, 3072), (4737, 3072), (5684, 3072)])
def test_rows_of_three_pieces(rows, cols):
    test_products(rows, cols, DType.F16, torch.float16)
    g = torch.Generator(device="cuda").manual_seed(rows)
    W, x = (torch.randn(rows, cols, generator=g, device="cuda") * cols ** -0.5).half(), activations(1, cols, cols)[0]
    y = torch.full((rows + 1,), 3.0, device="cuda")
    lib().nt_b200_gemv_add(y.data_ptr(), W.data_ptr(), x.data_ptr(), rows, cols, int(DType.F16), stream())
    torch.cuda.synchronize()
    assert rel(y[:rows], 3.0 + W.double() @ x.double()) <= (cols / 32) ** 0.5 * 2.0 ** -24 + 2.0 ** -22 and y[rows] == 3.0
