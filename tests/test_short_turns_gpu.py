"""A few tokens behind a context (csrc/attention.cu launch_rows): one slice of the keys, several, and as many as the scratch has room for, against the same tokens one by one."""
import dataclasses

import numpy as np
import pytest

pytest.importorskip("torch")
from test_short_prompt_gpu import ODD, both  # noqa: E402

pytestmark = [pytest.mark.gpu]
ONE_IN_EIGHT = dataclasses.replace(ODD, hidden_size=1024, n_heads=8, n_kv_heads=1, max_seq_len=1600)      # one CTA to a query and a slice
FOUR = dataclasses.replace(ODD, hidden_size=1024, n_heads=16, n_kv_heads=4, head_dim=128, max_seq_len=1600)


@pytest.mark.parametrize("cfg", [ONE_IN_EIGHT, FOUR, dataclasses.replace(ODD, max_seq_len=1600)])
@pytest.mark.parametrize("n,before", [(2, 31), (2, 1500), (5, 700), (19, 200), (31, 1569)])
def test_together_equals_one_by_one(cfg, n, before):
    toks = np.random.default_rng(n).integers(0, cfg.vocab_size, size=n + before).tolist()
    both(cfg, "Q6_K", toks[:before], toks[before:], [0, n - 1])
