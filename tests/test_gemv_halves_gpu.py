"""SwiGLU over gate and up in one launch (csrc/gemv_kquant.cu): pairs of 16-row groups, and groups of 8 rows of each where the number of rounds falls, over rows that
end inside a group, one and several rounds, every format and one mix; and long rows on the form with two stages of fewer, larger teams."""
import pytest

torch = pytest.importorskip("torch")
from ntransformer_b200 import kernels as K  # noqa: E402
from ntransformer_b200.dtypes import DType  # noqa: E402
from test_block_products_gpu import FORMATS, activations, matrix, rel  # noqa: E402

pytestmark = [pytest.mark.gpu]


# 592 teams of 4 warps on 148 SMs: 8-row groups at 20, 2372 + 5 and 28480 + 3 rows, 16-row pairs at 14336 and 9999
@pytest.mark.parametrize("dt", FORMATS, ids=lambda d: d.name)
@pytest.mark.parametrize("rows,cols", [(20, 256), (2377, 2048), (9999, 1024), (14336, 512), (28483, 512)])
def test_swiglu(dt, rows, cols):
    if dt == DType.Q6_K:
        cols = 2048                                                # the entry takes rows on 16 bytes
    (G, G64), (U, U64) = matrix(dt, rows, cols, 1), matrix(dt, rows, cols, 2)
    x, g = activations(1, cols, 3)[0], 1 + 0.1 * activations(1, cols, 4)[0]
    y = torch.full((rows + 8,), 7.0, device="cuda")
    K.gemv_fused_f32([y, y], [G, U], [rows, rows], [dt, dt], cols, x, epilogue=2, norm_w=g, eps=1e-5)
    torch.cuda.synchronize()
    u = x.double() / (x.double().pow(2).mean() + 1e-5).sqrt() * g.double()
    # two products (24-bit integers of a block's largest, F32 sums) and the fast-math sigmoid
    assert rel(y[:rows], torch.nn.functional.silu(G64 @ u) * (U64 @ u)) <= 4e-6 and (y[rows:] == 7.0).all()


def test_swiglu_of_two_formats():
    rows, cols = 2377, 1024
    (G, G64), (U, U64) = matrix(DType.Q4_K_M, rows, cols, 1), matrix(DType.Q5_K, rows, cols, 2)
    x = activations(1, cols, 3)[0]
    y = torch.full((rows + 8,), 7.0, device="cuda")
    K.gemv_fused_f32([y, y], [G, U], [rows, rows], [DType.Q4_K_M, DType.Q5_K], cols, x, epilogue=2)
    torch.cuda.synchronize()
    assert rel(y[:rows], torch.nn.functional.silu(G64 @ x.double()) * (U64 @ x.double())) <= 4e-6 and (y[rows:] == 7.0).all()


@pytest.mark.parametrize("dt", FORMATS, ids=lambda d: d.name)
def test_long_rows_of_many_groups(dt):
    rows, cols = 4113, 28672
    W, W64 = matrix(dt, rows, cols, 5)
    x = activations(1, cols, 6)[0]
    y = torch.zeros(rows, device="cuda")
    K.launch_gemv(y, W, x, rows, cols, dt)
    torch.cuda.synchronize()
    assert rel(y, W64 @ x.double()) <= 1e-6
