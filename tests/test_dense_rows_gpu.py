"""Dense GEMV at the edges of its walk (pieces of a row, warps to a row), against 64 bits and against the general path (the same rows off 16 bytes)."""
import pytest
import torch

from ntransformer_b200._lib import lib
from ntransformer_b200.dtypes import DType

pytestmark = pytest.mark.gpu
TORCH_DT = {DType.F32: torch.float32, DType.F16: torch.float16, DType.BF16: torch.bfloat16}


def stream():
    return torch.cuda.current_stream().cuda_stream


def off_16_bytes(t):
    """the same numbers one element behind a 16-byte boundary"""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")
    buf[1:] = t.reshape(-1)
    return buf[1:].view(t.shape)


# K: a piece alone, whole and ragged chunks of 128 pieces; rows: fewer than a launch's places, just over them (two warps to a row), an odd number
@pytest.mark.parametrize("dt,K", [(DType.BF16, 8), (DType.BF16, 1032), (DType.BF16, 2048), (DType.F16, 4096), (DType.BF16, 4104), (DType.BF16, 14336),
                                  (DType.BF16, 24584), (DType.F32, 1028), (DType.F32, 4096)])
@pytest.mark.parametrize("outs", [(5, 1, 2), (4099, 37, 601)])
def test_gemv_dense_shared_rows(dt, K, outs):
    g = torch.Generator(device="cuda").manual_seed(K)
    rnd = lambda *n: torch.randn(*n, device="cuda", generator=g)   # noqa: E731
    Ws = [(rnd(o, K) * K ** -0.5).to(TORCH_DT[dt]) for o in outs]
    up = (rnd(outs[0], K) * K ** -0.5).to(TORCH_DT[dt])
    x, gain, y0 = rnd(K), rnd(outs[0]), rnd(outs[0])
    # F32 sums: a product joins at most K / (32 * 4) + 8 additions of 2^-24 relative to the sum of magnitudes
    bound = lambda W: (W.double().abs() @ x.double().abs()) * 2.0 ** -24 * (K / 128 + 24)   # noqa: E731

    def run(aligned):
        M = [w if aligned else off_16_bytes(w) for w in Ws + [up]]
        ys = [torch.full((o,), 7.0, device="cuda") for o in outs]
        lib().nt_b200_gemv_dense(*[y.data_ptr() for y in ys], *[m.data_ptr() for m in M[:3]], *outs, 3, K, x.data_ptr(), int(dt), 0, None, 1.0, stream())
        add, plain, glu = y0.clone(), y0.clone(), torch.zeros(outs[0], device="cuda")
        one = (None, None, M[0].data_ptr(), None, None, outs[0], 0, 0, 1, K, x.data_ptr(), int(dt))
        lib().nt_b200_gemv_dense(add.data_ptr(), *one, 2, gain.data_ptr(), 0.7, stream())
        lib().nt_b200_gemv_dense(plain.data_ptr(), *one, 1, None, 1.0, stream())
        lib().nt_b200_gemv_dense(glu.data_ptr(), None, None, M[0].data_ptr(), M[3].data_ptr(), None, outs[0], outs[0], 0, 2, K, x.data_ptr(), int(dt), 3, None, 1.0,
                                 stream())
        torch.cuda.synchronize()
        return ys + [add, plain, glu]

    if dt != DType.F32:        # an infinity or a NaN in the last piece reaches a row once: the same kind as in 64 bits, on both paths
        for v in (float("inf"), float("nan")):
            keep = x[-3].item()
            x[-3] = v
            for got in (run(True), run(False)):
                for y, W in zip(got, Ws):
                    ref = W.double()[:, -3] * v
                    assert (torch.isnan(y) == torch.isnan(ref)).all() and (torch.isnan(ref) | (y.double() == ref)).all()
            x[-3] = keep

    p = [W.double() @ x.double() for W in Ws + [up]]
    b = [bound(W) for W in Ws + [up]]
    silu = torch.nn.functional.silu(p[0])
    ref = p[:3] + [y0.double() + 0.7 * gain.double() * p[0], y0.double() + p[0], silu * p[3]]
    tol = b[:3] + [0.7 * gain.double().abs() * b[0], b[0], 1.1 * b[0] * p[3].abs() + silu.abs() * b[3]]
    for got in (run(True), run(False)):
        for y, r, t in zip(got, ref, tol):
            assert ((y.double() - r).abs() <= t + r.abs() * 2.0 ** -21 + 1e-7).all()
