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
