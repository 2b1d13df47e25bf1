"""What a launch reads may be written by the launch before it until that one ends: behind one that lets the next start at once and writes late, every launch of the
boundary gives what it gives on inputs that lie there already."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
from ntransformer_b200 import kernels as K  # noqa: E402
from ntransformer_b200._lib import lib  # noqa: E402
from ntransformer_b200.dtypes import DType  # noqa: E402
from ntransformer_b200.synth import random_blocks_np  # noqa: E402

pytestmark = [pytest.mark.gpu]
LATE = 30000      # nanoseconds


def stream():
    return torch.cuda.current_stream().cuda_stream


def check(call, inputs, outs):
    """call(): launches; inputs: what it reads; outs(): fresh outputs -> list.  One input after the other comes late, as other numbers were there before."""
    want = outs()
    call(want)
    torch.cuda.synchronize()
    for t in inputs:
        new = t.clone()
        old = torch.flip(new.reshape(-1), [0]).reshape(new.shape).contiguous() if t.dtype != torch.int32 else new + 3
        for _ in range(3):
            got = outs()
            t.copy_(old)
            torch.cuda.synchronize()
            lib().nt_b200_late_copy(t.data_ptr(), new.data_ptr(), t.numel() * t.element_size(), LATE, stream())
            call(got)
            torch.cuda.synchronize()
            assert all(torch.equal(a, b) for a, b in zip(want, got)), (tuple(t.shape), t.dtype)


def randn(*shape):
    return torch.randn(*shape, device="cuda")


@pytest.mark.parametrize("hidden", [512, 4096, 9216])
def test_norms(hidden):
    x, w = randn(2, hidden), randn(hidden)
    check(lambda o: K.launch_rmsnorm(o[0], x, w, 2, hidden, 1e-5), [x, w], lambda: [torch.zeros(2, hidden, device="cuda")])
    check(lambda o: K.launch_rmsnorm_f16(o[0], x, w, 2, hidden, 1e-5), [x, w], lambda: [torch.zeros(2, hidden, device="cuda", dtype=torch.float16)])


def test_elementwise():
    a, b = randn(4096), randn(4096)
    zeros = lambda: [torch.zeros(4096, device="cuda")]   # noqa: E731
    check(lambda o: K.launch_silu_mul(o[0], a, b, 4096), [a, b], zeros)
    check(lambda o: K.launch_add(o[0], a, b, 4096), [a, b], zeros)
    check(lambda o: K.launch_add_inplace(o[0], b, 4096), [b], zeros)
    check(lambda o: K.launch_add_bias(o[0], b, 4096), [b], zeros)
    check(lambda o: K.launch_copy(o[0], a, 4096), [a], zeros)
    check(lambda o: K.launch_softmax(o[0], a, 4, 1024), [a], zeros)
    check(lambda o: K.launch_cosine_similarity(o[0], a, b, 4096), [a, b], lambda: [torch.zeros(1, device="cuda")])


@pytest.mark.parametrize("interleaved", [False, True])
def test_rope_and_cache(interleaved):
    q, k, v, pos = randn(3, 8, 128), randn(3, 2, 128), randn(3, 2, 128), torch.tensor([5, 6, 7], dtype=torch.int32, device="cuda")
    q0, k0 = q.clone(), k.clone()

    def rope(o):
        lib().nt_b200_rope(o[0].data_ptr(), o[1].data_ptr(), pos.data_ptr(), 1, 3, 8, 2, 128, 1e4, 1.0, int(interleaved), stream())

    check(rope, [pos], lambda: [q0.clone(), k0.clone()])
    check(lambda o: K.launch_copy_to_kv_cache(o[0], o[1], k, v, 3, 2, 128, 1, 8), [k, v], lambda: [torch.zeros(8, 2, 128, device="cuda", dtype=torch.float16) for _ in range(2)])


@pytest.mark.parametrize("dt", [DType.Q4_0, DType.Q8_0, DType.Q4_K_M, DType.Q5_K, DType.Q6_K, DType.F16, DType.F32], ids=lambda d: d.name)
@pytest.mark.parametrize("rows,cols", [(64, 512), (3000, 2048), (256, 11008)])
def test_gemv(dt, rows, cols):
    if dt == DType.F32:
        W = randn(rows, cols)
    elif dt == DType.F16:
        W = randn(rows, cols).half()
    else:
        W = torch.from_numpy(random_blocks_np(dt, rows, cols, np.random.default_rng(1))).cuda()
    other = W.reshape(rows, -1).flip(0).contiguous()               # whole rows: blocks stay blocks
    x = randn(cols)
    for call in (K.launch_gemv, K.launch_gemv_add):
        check(lambda o: call(o[0], W, x, rows, cols, dt), [x], lambda: [torch.zeros(rows, device="cuda")])
    want, got = torch.zeros(rows, device="cuda"), torch.zeros(rows, device="cuda")
    K.launch_gemv(want, W, x, rows, cols, dt)
    new = W.clone()
    W.copy_(other.view(W.shape))
    torch.cuda.synchronize()
    lib().nt_b200_late_copy(W.data_ptr(), new.data_ptr(), W.numel() * W.element_size() // 4 * 4, LATE, stream())
    K.launch_gemv(got, W, x, rows, cols, dt)
    torch.cuda.synchronize()
    assert torch.equal(want, got)


@pytest.mark.parametrize("ctx", [40, 900])
@pytest.mark.parametrize("heads,kv,dim", [(8, 2, 128), (4, 4, 64)])
def test_decode_attention(ctx, heads, kv, dim):
    q, kc, vc = randn(heads, dim), randn(ctx, kv, dim).half(), randn(ctx, kv, dim).half()
    check(lambda o: K.launch_attention_decode(o[0], q, kc, vc, ctx, heads, kv, dim, ctx, dim ** -0.5), [q, kc, vc], lambda: [torch.zeros(heads, dim, device="cuda")])


@pytest.mark.parametrize("heads,kv,dim,tokens", [(8, 2, 128, 40), (8, 2, 64, 40), (152, 76, 128, 40), (153, 51, 64, 200), (8, 2, 128, 5)])
def test_prompt_attention(heads, kv, dim, tokens):
    q, kc, vc = randn(tokens, heads, dim), randn(tokens + 9, kv, dim).half(), randn(tokens + 9, kv, dim).half()
    check(lambda o: K.launch_attention_prefill(o[0], q, kc, vc, tokens, 9, heads, kv, dim, tokens + 9, dim ** -0.5), [q, kc, vc],
          lambda: [torch.zeros(tokens, heads, dim, device="cuda")])


@pytest.mark.parametrize("dt", [DType.Q4_K_M, DType.Q6_K], ids=lambda d: d.name)
@pytest.mark.parametrize("fine", [0, 1])
def test_tokens_over_blocks(dt, fine):
    tokens, rows, cols = 20, 300, 1024
    W = torch.from_numpy(random_blocks_np(dt, rows, cols, np.random.default_rng(1))).cuda()
    x, g = randn(tokens, cols), randn(cols)

    def call(o):
        one = lambda t: (C.c_void_p * 1)(t.data_ptr())   # noqa: E731
        assert lib().nt_b200_gemm_blocks(1, one(o[0]), one(W), (C.c_int * 1)(rows), (C.c_int * 1)(int(dt)), cols, x.data_ptr(), g.data_ptr(), 1e-5, tokens, fine, 0, stream()) == 0

    zeros = lambda: [torch.zeros(tokens, rows, device="cuda")]   # noqa: E731
    check(call, [x, g], zeros)
    new = W.clone()
    want, got = zeros(), zeros()
    call(want)
    W.copy_(new.flip(0))
    torch.cuda.synchronize()
    lib().nt_b200_late_copy(W.data_ptr(), new.data_ptr(), W.numel() // 4 * 4, LATE, stream())
    call(got)
    torch.cuda.synchronize()
    assert torch.equal(want[0], got[0])
