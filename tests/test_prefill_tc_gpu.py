"""Causal attention of prompt tokens on tcgen05 (csrc/attention_prefill_tc.cu) against 64 bits, and against the form on mma.sync that queries off 16 bytes still take:
tiles of 128 queries and steps of 128 keys with remainders, one head to a key head (two runs of queries to a CTA), an odd and an even number of them, both widths."""
import pytest

torch = pytest.importorskip("torch")
from ntransformer_b200 import kernels as K  # noqa: E402
from ntransformer_b200._lib import lib  # noqa: E402

pytestmark = [pytest.mark.gpu]


def inputs(heads, kv, dim, tokens, start, by=1.0):
    g = torch.Generator(device="cuda").manual_seed(heads * 1000 + tokens + start)
    keys = start + tokens
    kc, vc = (torch.randn(keys + 70, kv, dim, device="cuda", generator=g).half() for _ in range(2))
    return torch.randn(tokens, heads, dim, device="cuda", generator=g) * by, kc, vc


def exact(q, kc, vc, start, scale):
    tokens, heads, _ = q.shape
    k, v = (c[: start + tokens].double().repeat_interleave(heads // c.shape[1], 1) for c in (kc, vc))
    s = torch.einsum("thd,shd->hts", q.double(), k) * scale
    hidden = torch.arange(start + tokens, device="cuda")[None] > torch.arange(tokens, device="cuda")[:, None] + start
    return torch.einsum("hts,shd->thd", torch.softmax(s.masked_fill(hidden, -float("inf")), 2), v)


def attend(q, kc, vc, start, scale, off=False):
    tokens, heads, dim = q.shape
    out = torch.full((tokens + 1, heads, dim), 7.0, device="cuda")
    if off:                                                        # the same numbers 8 bytes on: what TMA and 16-byte loads do not take
        room = torch.empty(q.numel() + 2, device="cuda")
        room[2:] = q.reshape(-1)
        src = room.data_ptr() + 8
    else:
        src = q
    K.launch_attention_prefill(out, src, kc, vc, tokens, start, heads, kc.shape[1], dim, kc.shape[0], scale)
    torch.cuda.synchronize()
    assert (out[tokens] == 7.0).all()
    return out[:tokens]


def form(q, kc, start):
    tokens, heads, dim = q.shape
    return lib().nt_b200_attention_prefill_form(*[0x1000] * 4, tokens, start, heads, kc.shape[1], dim, kc.shape[0])


def rel(a, b):
    return float(((a.double() - b).norm() / b.norm()).item())


@pytest.mark.parametrize("heads,kv,dim", [(8, 2, 128), (8, 8, 128), (6, 2, 64), (4, 1, 64), (2, 1, 128)])
@pytest.mark.parametrize("tokens,start", [(16, 0), (128, 0), (129, 127), (257, 1), (300, 500), (17, 1400), (640, 0)])
def test_prompt(heads, kv, dim, tokens, start):
    q, kc, vc = inputs(heads, kv, dim, tokens, start)
    want = exact(q, kc, vc, start, dim ** -0.5)
    kc[start + tokens:] = float("nan")                             # rows of the cache that no query sees
    vc[start + tokens:] = float("inf")
    # scores: dim / 16 additions of each half, cut by 2/3 of 2^-24 of up to |s| = 8 or so, in the exponent: 5e-6 at most, mostly cancelling; halves' pairs 2^-22
    got = attend(q, kc, vc, start, dim ** -0.5)
    assert rel(got, want) <= 5e-6
    assert torch.equal(got, attend(q, kc, vc, start, dim ** -0.5))


@pytest.mark.parametrize("heads,kv", [(152, 76), (153, 51), (152, 152)])      # more than a wave of mma.sync's tiles: the tcgen05 form at any length
@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("tokens,start", [(16, 0), (128, 0), (129, 127), (257, 1), (300, 500), (17, 1400)])
def test_prompt_of_many_heads(heads, kv, dim, tokens, start):
    q, kc, vc = inputs(heads, kv, dim, tokens, start)
    want = exact(q, kc, vc, start, dim ** -0.5)
    kc[start + tokens:] = float("nan")
    vc[start + tokens:] = float("inf")
    assert form(q, kc, start) == 2
    got = attend(q, kc, vc, start, dim ** -0.5)
    assert rel(got, want) <= 5e-6                                  # as above
    assert torch.equal(got, attend(q, kc, vc, start, dim ** -0.5))


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("by", [1e-3, 0.05, 1.0, 4.0])
def test_no_further_from_64_bits_than_the_form_before(dim, by):
    q, kc, vc = inputs(32, 8, dim, 260, 700, by)
    assert form(q, kc, 700) == 2
    want = exact(q, kc, vc, 700, dim ** -0.5)
    got, old = attend(q, kc, vc, 700, dim ** -0.5), attend(q, kc, vc, 700, dim ** -0.5, off=True)
    print("dim %d, queries x %g: %.2e here, %.2e before" % (dim, by, rel(got, want), rel(old, want)))
    assert rel(got, want) <= rel(old, want)


def test_a_nan_stays_in_its_row_and_wide_scores():
    q, kc, vc = inputs(152, 76, 128, 200, 50, 30.0)                # one key takes most of a row's weight
    q[7, 1, 3] = float("nan")
    q[8] = 0
    assert form(q, kc, 50) == 2
    got, want = attend(q, kc, vc, 50, 128 ** -0.5), exact(q, kc, vc, 50, 128 ** -0.5)
    assert torch.isnan(got[7, 1]).all()
    keep = torch.ones(200, 152, dtype=torch.bool, device="cuda")
    keep[7, 1] = False
    assert torch.isfinite(got[keep]).all() and rel(got[keep], want[keep]) <= 5e-5       # scores of up to 100: 2^-22 of them in the exponent


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("scale", [0.0, -0.0, -0.1, -1.0, 1e-30])
@pytest.mark.parametrize("tokens,start", [(200, 50), (130, 0)])
def test_a_scale_of_any_sign(dim, scale, tokens, start):
    q, kc, vc = inputs(153, 51, dim, tokens, start)                # (three heads to a key head: runs of queries, whose first tile has whole steps behind it)
    assert form(q, kc, start) == 2
    got, want = attend(q, kc, vc, start, scale), exact(q, kc, vc, start, scale)
    # in the exponent: 2 * dim / 16 additions, each cut by 2/3 of 2^-24 of a score, and halves' pairs, 2^-22 of it; weights as above
    most = abs(scale) * float((q.norm(dim=2).max() * kc[: start + tokens].float().norm(dim=2).max()).item())
    assert torch.isfinite(got).all() and rel(got, want) <= 5e-6 + (dim / 8 * 2 / 3 * 2.0**-24 + 2.0**-22) * most


@pytest.mark.parametrize("rows", [1, 250, 299])
def test_positions_behind_the_cache_stay_inside_it(rows):
    """Such keys are the cache's last row, as in the form on mma.sync; what lies behind the cache is not read."""
    q, kc, vc = inputs(8, 2, 128, 200, 100)
    kc[rows:], vc[rows:] = float("nan"), float("nan")              # (the allocation goes on)
    inside = torch.arange(300, device="cuda").clamp(max=rows - 1)
    out = torch.empty_like(q)
    K.launch_attention_prefill(out, q, kc, vc, 200, 100, 8, 2, 128, rows, 128 ** -0.5)
    torch.cuda.synchronize()
    assert rel(out, exact(q, kc[inside], vc[inside], 100, 128 ** -0.5)) <= 2e-5      # the form on mma.sync: queries and weights as pairs of halves without a power of two


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("heads,kv,tokens,start", [(152, 76, 200, 70), (153, 51, 300, 0), (152, 76, 16, 1000)])
def test_an_infinite_or_nan_value_reaches_the_queries_that_see_it_and_no_others(dim, heads, kv, tokens, start):
    q, kc, vc = inputs(heads, kv, dim, tokens, start)
    assert form(q, kc, start) == 2
    want = exact(q, kc, vc, start, dim ** -0.5)
    last = start + tokens - 1
    for head, key, channel, value in ((0, last - 9, 3, "inf"), (1, start + 7, dim - 1, "nan"), (2, last, 0, "-inf")):
        vc[key, head, channel] = float(value)
    got = attend(q, kc, vc, start, dim ** -0.5)
    bad = torch.zeros(tokens, heads, dim, dtype=torch.bool, device="cuda")
    for head, key, channel in ((0, last - 9, 3), (1, start + 7, dim - 1), (2, last, 0)):
        bad[key - start:, head * (heads // kv):(head + 1) * (heads // kv), channel] = True
    assert torch.equal(~torch.isfinite(got), bad)
    keep = torch.where(bad, torch.zeros_like(got), got)
    assert rel(keep, torch.where(bad, torch.zeros_like(want), want)) <= 5e-6
