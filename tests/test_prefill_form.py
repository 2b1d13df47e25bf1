"""Which form a call of prompt attention takes (csrc/attention.cu attention_prefill_form): the choice alone, no device."""
import pytest

from ntransformer_b200._lib import lib

QUERIES, MMA, TC = 0, 1, 2


def form(tokens, start, heads=32, kv=8, dim=128, rows=None, out=0x1000, q=0x2000, k=0x3000, v=0x4000):
    return lib().nt_b200_attention_prefill_form(out, q, k, v, tokens, start, heads, kv, dim, start + tokens if rows is None else rows)


@pytest.mark.parametrize("tokens,start", [(500, 0), (1000, 1023)])
def test_positions_behind_the_cache(tokens, start):
    """The maps of the tcgen05 form have a row for every key; the form on mma.sync stays inside the cache whatever the positions."""
    assert form(tokens, start) == TC and form(tokens, start, rows=4096) == TC
    for rows in (start + tokens - 1, start, 1):
        assert form(tokens, start, rows=rows) == MMA
    assert form(tokens, -1, rows=4096) == MMA and form(tokens, 2**31 - 100, rows=2**31 - 1) == MMA


def test_pointers_and_widths():
    assert form(1000, 0, dim=64) == TC and form(1000, 0, dim=96) == QUERIES and form(15, 0) == QUERIES and form(1000, 0, heads=30) == QUERIES
    for name in ("out", "q", "k", "v"):
        assert form(1000, 0, **{name: 0x1008}) == MMA


# measured where the two forms take turns (us on tcgen05, on mma.sync): neither side of the line by more than a few per cent
@pytest.mark.parametrize("dim,heads,kv,start,tokens,want", [
    (128, 32, 8, 0, 17, MMA),          # 10.9, 8.4
    (128, 64, 8, 0, 26, MMA),          # 10.9, 8.2
    (128, 4, 2, 0, 167, MMA),          # 13.5, 10.8
    (128, 32, 8, 300, 17, MMA),        # 16.8, 14.5
    (128, 32, 8, 300, 40, TC),         # 16.9, 18.6
    (128, 32, 8, 300, 100, MMA),       # 21.1, 18.8
    (128, 32, 8, 0, 256, MMA),         # 15.5, 14.0
    (128, 32, 8, 0, 500, TC),          # 21.3, 32.2: more than a wave there
    (128, 4, 4, 1000, 17, TC),         # 30.1, 35.6
    (128, 4, 4, 0, 1000, TC),          # 32.4, 35.7
    (64, 8, 2, 24, 231, MMA),          # 12.7, 10.3
    (64, 16, 4, 0, 115, MMA),          # 8.0, 7.2
    (64, 32, 8, 1000, 17, TC),         # 22.9, 24.7
    (64, 16, 16, 300, 500, MMA),       # 22.9, 20.8
    (64, 64, 8, 0, 200, TC),           # 10.6, 12.5
])
def test_the_faster_form(dim, heads, kv, start, tokens, want):
    assert form(tokens, start, heads, kv, dim) == want
