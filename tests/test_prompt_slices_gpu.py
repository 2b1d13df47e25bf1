"""Prompt attention in slices of the keys (csrc/attention_prefill_mma.cu, csrc/attention.cu attention_prefill_slices_for) against 64 bits."""
import pytest

torch = pytest.importorskip("torch")
from ntransformer_b200 import kernels as K  # noqa: E402
from test_prefill_tc_gpu import attend, exact, inputs, rel  # noqa: E402

pytestmark = [pytest.mark.gpu]


def sliced(q, kc, vc, start, scale):
    before = K.launch_count()
    got = attend(q, kc, vc, start, scale)
    assert K.launch_count() - before == 2                          # the slices' launch and the merge's
    assert torch.equal(got.nan_to_num(7.5), attend(q, kc, vc, start, scale).nan_to_num(7.5))
    return got


# the last tile of keys whole and with one key; sixteen slices, some without a tile; early queries that see the first slices alone; one head to a key head, and three
@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("heads,kv,tokens,start", [(4, 2, 16, 496), (4, 2, 17, 496), (1, 1, 20, 1005), (2, 1, 64, 4000), (6, 2, 70, 500), (2, 2, 600, 0), (8, 8, 129, 900), (4, 1, 1000, 41), (64, 8, 17, 1000)])
def test_slices(dim, heads, kv, tokens, start):
    q, kc, vc = inputs(heads, kv, dim, tokens, start)
    want = exact(q, kc, vc, start, dim ** -0.5)
    kc[start + tokens:] = float("nan")                             # rows of the cache that no query sees
    vc[start + tokens:] = float("inf")
    # the high halves' products: dim / 32 + 4 additions, each cut by up to 2^-23 of the sum so far, two in three of it on average, and halves' pairs, 2^-22; measured 2e-7 to 4e-7
    assert rel(sliced(q, kc, vc, start, dim ** -0.5), want) <= 1e-6


@pytest.mark.parametrize("by", [1e-30, 1e-3, 1e4])
@pytest.mark.parametrize("scale", [0.0, -0.1, 128 ** -0.5])
def test_queries_and_scales_of_any_size(by, scale):
    q, kc, vc = inputs(4, 2, 128, 100, 700, by)
    scale = scale / by if by > 1 else scale
    most = abs(scale) * float((q.norm(dim=2).max() * kc.float().norm(dim=2).max()).item())
    got = sliced(q, kc, vc, 700, scale)
    assert torch.isfinite(got).all() and rel(got, exact(q, kc, vc, 700, scale)) <= 1e-6 + 2.0**-22 * most


def test_values_that_a_row_does_not_see_and_nan():
    q, kc, vc = inputs(4, 2, 128, 100, 700)
    q[7, 1, 3] = float("nan")
    vc[760, 0, 5], vc[760, 1, 100] = float("inf"), float("nan")    # token 60 of the prompt: rows 0 to 59 do not see it
    got, want = sliced(q, kc, vc, 700, 128 ** -0.5), exact(q, kc, torch.where(torch.isfinite(vc), vc, 0), 700, 128 ** -0.5)
    assert torch.isnan(got[7, 1]).all()
    keep = torch.isfinite(want) & ~torch.isnan(q).any(2, keepdim=True)
    keep[60:, :2, 5] = keep[60:, 2:, 100] = False
    assert torch.isfinite(got[keep]).all() and rel(got[keep], want[keep]) <= 1e-6
    assert torch.isinf(got[60:, :2, 5]).all() and torch.isnan(got[60:, 2:, 100]).all()


# keys whose scores are NaN, each seen first by the row at its own position: the first of a slice (no other of that slice for the row), one inside, and one whose slice has no weight beside
# the others'; an infinite value there
@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("at", [704, 705, 767])
def test_keys_that_are_nan_reach_every_row_that_sees_them(dim, at):
    q, kc, vc = inputs(4, 2, dim, 100, 700)
    kc[at, 0, 3] = float("nan")
    got, want = sliced(q, kc, vc, 700, dim ** -0.5), exact(q, torch.where(torch.isfinite(kc), kc, 0), vc, 700, dim ** -0.5)
    assert torch.isnan(got[at - 700:, :2]).all()                   # heads 0 and 1 share the key head
    keep = torch.ones_like(want, dtype=torch.bool)
    keep[at - 700:, :2] = False
    assert rel(got[keep], want[keep]) <= 1e-6


@pytest.mark.parametrize("dim", [64, 128])
def test_slices_without_weight(dim):
    q, kc, vc = inputs(4, 2, dim, 100, 700)
    q, kc = q.abs(), kc.abs() * 0.1
    kc[1] = 60.0                                                   # every query's weight, all but nothing else's
    vc[400, 0, 7] = float("inf")
    kc[401, 1, 2] = float("nan")
    got = sliced(q, kc, vc, 700, 1.0)
    assert not torch.isfinite(got[:, :2, 7]).any() and torch.isnan(got[:, 2:]).all()
    keep = torch.arange(dim, device="cuda") != 7
    assert rel(got[:, :2][:, :, keep], vc[1, 0].double()[keep].expand(100, 2, dim - 1)) <= 1e-6
