"""The matrix-instruction GEMV (csrc/gemv_kquant.cu) where its tiling can go wrong: rows around a 16-row group, few and many groups, rows of 1, 2, 4, 5, 9
and 43 super-blocks (partly filled stages; Q6_K rows whose bytes start at any even address), the matrix's last bytes, vectors of both long-row forms."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from ntransformer_b200 import kernels as K  # noqa: E402
from ntransformer_b200.dtypes import DType, dtype_row_size  # noqa: E402
from ntransformer_b200.synth import random_blocks_np  # noqa: E402
from oracle import oracle as O  # noqa: E402

pytestmark = [pytest.mark.gpu]
FORMATS = [DType.Q4_K_M, DType.Q5_K, DType.Q6_K, DType.Q8_0, DType.Q4_0]


def close(got, raw, x, rows, cols, dt):
    """The vector is held in 24-bit integers of its 32-blocks (2^-24 of their largest value), products are exact, sums F32: the error of a row is
    below 2^-24 * sum |w| (blockmax + |x| * log2(cols)), far below 3e-6 of sum |w| |x|; the rows here have random signs, so compare with their scale."""
    ref = O.gemv(raw, x, rows, cols, int(dt))
    scale = np.abs(x).max() * np.sqrt(cols) * 0.02
    assert np.abs(got - ref).max() <= 4e-6 * scale, np.abs(got - ref).max() / scale


@pytest.mark.parametrize("dt", FORMATS, ids=lambda d: d.name)
@pytest.mark.parametrize("rows,cols", [(1, 256), (15, 512), (16, 1024), (17, 1280), (33, 2304), (2400, 1024), (2353, 4096), (4736, 256), (40, 11008), (4113, 8448), (19, 28672)])
def test_rows_and_stages(dt, rows, cols):
    rng = np.random.default_rng(rows * 7 + cols)
    raw = random_blocks_np(dt, rows, cols, rng)
    x = (rng.standard_normal(cols) * np.where(rng.random(cols) < 0.02, 10, 1)).astype(np.float32)
    y = torch.full((rows + 1,), 7.0, device="cuda")
    K.launch_gemv(y, torch.from_numpy(raw).cuda(), torch.from_numpy(x).cuda(), rows, cols, dt)
    torch.cuda.synchronize()
    got = y.cpu().numpy()
    assert got[rows] == 7.0
    close(got[:rows], raw, x, rows, cols, dt)


# Rows as long as the kernel takes: what is left of shared memory beside the vector holds one to three stages.  More and fewer than 256 row groups.
@pytest.mark.parametrize("dt,rows,cols", [(DType.Q4_K_M, 4113, 49152), (DType.Q4_K_M, 40, 49152), (DType.Q5_K, 4113, 42240), (DType.Q5_K, 2400, 49152),
                                          (DType.Q6_K, 4113, 48896), (DType.Q8_0, 4113, 48384), (DType.Q8_0, 33, 49152), (DType.Q4_0, 4113, 49152)], ids=str)
def test_longest_rows(dt, rows, cols):
    rng = np.random.default_rng(cols + rows)
    block = random_blocks_np(dt, 64, cols, rng)                        # rows repeat: the oracle walks 64 of them
    raw = torch.from_numpy(block).cuda().reshape(64, -1).repeat((rows + 63) // 64, 1)[:rows].contiguous()
    x = (rng.standard_normal(cols) * np.where(rng.random(cols) < 0.02, 10, 1)).astype(np.float32)
    xd = torch.from_numpy(x).cuda()
    ref = np.resize(O.gemv(block, x, 64, cols, int(dt)), rows)
    ys = [torch.zeros(rows, device="cuda")]
    K.launch_gemv(ys[0], raw, xd, rows, cols, dt)
    if dtype_row_size(dt, cols) % 16 == 0:                             # the entry over a pre-quantised vector (22 bits: four times the rounding)
        ys.append(torch.zeros(rows, device="cuda"))
        xq = torch.zeros(K.xq_bytes(cols), dtype=torch.uint8, device="cuda")
        K.quantize_x(xd, xq, cols)
        K.gemv_fused([ys[1]], [raw], [rows], [dt], cols, xq)
    torch.cuda.synchronize()
    scale = np.abs(x).max() * np.sqrt(cols) * 0.02
    for y, wide in zip(ys, (1, 4)):
        assert np.abs(y.cpu().numpy() - ref).max() <= 4e-6 * wide * scale


@pytest.mark.parametrize("special", ["zeros", "one", "tiny", "huge"])
def test_vectors_at_the_ends_of_the_range(special):
    rng = np.random.default_rng(3)
    rows, cols = 50, 1024
    raw = random_blocks_np(DType.Q4_K_M, rows, cols, rng)
    x = rng.standard_normal(cols).astype(np.float32)
    x[32:64] = 0
    if special == "zeros":
        x[:] = 0
    elif special == "one":
        x[:] = 0
        x[777] = -3
    else:
        x *= np.float32(1e-30 if special == "tiny" else 1e30)
    y = torch.zeros(rows, device="cuda")
    K.launch_gemv(y, torch.from_numpy(raw).cuda(), torch.from_numpy(x).cuda(), rows, cols, DType.Q4_K_M)
    torch.cuda.synchronize()
    close(y.cpu().numpy(), raw, x, rows, cols, DType.Q4_K_M)


# Rows of 3 super-blocks: in Q6_K they start at any even address, and were multiplied by the vector in F32 before there was this kernel (as Q4_0's)
@pytest.mark.parametrize("dt", FORMATS, ids=lambda d: d.name)
def test_nan_infinity_and_the_smallest_numbers(dt):
    rows, cols = 70, 768
    rng = np.random.default_rng(11)
    raw = random_blocks_np(dt, rows, cols, rng)
    W = np.stack([O.gemv(raw, e, rows, cols, int(dt)) for e in np.eye(cols, dtype=np.float32)], 1).astype(np.float64)

    def run(x):
        y = torch.zeros(rows, device="cuda")
        K.launch_gemv(y, torch.from_numpy(raw).cuda(), torch.from_numpy(x).cuda(), rows, cols, dt)
        torch.cuda.synchronize()
        return y.cpu().numpy().astype(np.float64)

    x = rng.standard_normal(cols).astype(np.float32)
    for at in (0, 37, 750):
        nan = x.copy()
        nan[at] = np.nan
        assert np.isnan(run(nan)).all()
        for v in (np.inf, -np.inf):
            inf = x.copy()
            inf[at] = v
            got = run(inf)
            if dt not in (DType.Q4_0, DType.Q6_K):         # an infinite scale over zeros, or the offset's infinity taken off the codes': not a number
                assert not np.isfinite(got).any()
            else:                                          # as in 64 bits: the infinity of the weight's sign, not a number where the weight is 0
                with np.errstate(invalid="ignore"):
                    ref = W[:, at] * v
                assert ((got == ref) | (np.isnan(got) & np.isnan(ref))).all()
    # numbers whose scale would be denormal: integers of 2^-126, so an element is off by 2^-127 at most; and a lane's share of a super-block below 2^-126 is
    # flushed before it counts 256
    for size in (3e-32, 1e-32, 1e-33):
        t = (x * np.float32(size)).astype(np.float32)
        bound = 2.0 ** -126 * (np.abs(W).sum(1) + 256 * 4 * cols / 256) + 4e-6 * np.abs(W) @ np.abs(t).astype(np.float64)
        assert (np.abs(run(t) - W @ t.astype(np.float64)) <= bound).all()


def test_nan_in_a_vector_that_is_quantised_by_a_launch_of_its_own():
    rng = np.random.default_rng(12)
    rows, cols = 40, 2048
    x = rng.standard_normal(cols).astype(np.float32)
    x[500] = np.nan
    for dt in FORMATS:
        raw, y = random_blocks_np(dt, rows, cols, rng), torch.zeros(rows, device="cuda")
        xq = torch.zeros(K.xq_bytes(cols), dtype=torch.uint8, device="cuda")
        K.quantize_x(torch.from_numpy(x).cuda(), xq, cols)
        K.gemv_fused([y], [torch.from_numpy(raw).cuda()], [rows], [dt], cols, xq)
        torch.cuda.synchronize()
        assert torch.isnan(y).all()


def test_vector_that_is_not_16_byte_aligned_takes_the_general_path():
    rng = np.random.default_rng(4)
    rows, cols = 40, 512
    raw = random_blocks_np(DType.Q6_K, rows, cols, rng)
    x = rng.standard_normal(cols + 1).astype(np.float32)
    xd = torch.from_numpy(x).cuda()
    y = torch.zeros(rows, device="cuda")
    K.launch_gemv(y, torch.from_numpy(raw).cuda(), xd.data_ptr() + 4, rows, cols, DType.Q6_K)
    torch.cuda.synchronize()
    close(y.cpu().numpy(), raw, x[1:], rows, cols, DType.Q6_K)


@pytest.mark.parametrize("dts", [(DType.Q4_K_M, DType.Q4_K_M, DType.Q6_K), (DType.Q4_K_M, DType.Q5_K), (DType.Q8_0, DType.Q8_0), (DType.Q4_0, DType.Q6_K)])
@pytest.mark.parametrize("pre", [False, True])
def test_matrices_of_one_launch(dts, pre):
    """Mixed formats share a launch's ring; `pre`: the vector in the pre-quantised form (22 bits for each element: four times the rounding)."""
    rng = np.random.default_rng(5)
    cols = 2048
    outs = [40, 33, 16][: len(dts)]
    raws = [random_blocks_np(d, o, cols, rng) for d, o in zip(dts, outs)]
    x = rng.standard_normal(cols).astype(np.float32)
    ys = [torch.zeros(o, device="cuda") for o in outs]
    Ws = [torch.from_numpy(r).cuda() for r in raws]
    xd = torch.from_numpy(x).cuda()
    if pre:
        xq = torch.zeros(K.xq_bytes(cols), dtype=torch.uint8, device="cuda")
        K.quantize_x(xd, xq, cols)
        K.gemv_fused(ys, Ws, outs, dts, cols, xq)
    else:
        K.gemv_fused_f32(ys, Ws, outs, dts, cols, xd)
    torch.cuda.synchronize()
    for y, r, o, d in zip(ys, raws, outs, dts):
        close(y.cpu().numpy() / (4 if pre else 1), r, x / np.float32(4 if pre else 1), o, cols, d)


def test_entries_that_answer_with_a_code_still_refuse_unaligned_rows():
    cols = 43 * 256
    assert dtype_row_size(DType.Q6_K, cols) % 16
    W = torch.zeros(16 * dtype_row_size(DType.Q6_K, cols), dtype=torch.uint8, device="cuda")
    y, x = torch.zeros(16, device="cuda"), torch.zeros(cols, device="cuda")
    with pytest.raises(ValueError):
        K.gemv_fused_f32([y], [W], [16], [DType.Q6_K], cols, x)
