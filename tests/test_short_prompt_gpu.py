"""A few tokens together (csrc/gemv_rows.cu, Model::prefill_short) against the same tokens one decode step at a time: every block format, passes of 8 tokens
and their remainders, rows that are not whole tiles of 32, contexts in front, chunks of 64 where the tensor-core prompt pass does not take the shape."""
import dataclasses

import numpy as np
import pytest

pytest.importorskip("torch")
from ntransformer_b200 import kernels as K  # noqa: E402
from ntransformer_b200.engine import Model  # noqa: E402
from ntransformer_b200.model_spec import TINY  # noqa: E402

pytestmark = [pytest.mark.gpu]
# rows of 3, 4 and 5 super-blocks (Q6_K: 630 and 1050 bytes, so rows start at any even address)
ODD = dataclasses.replace(TINY, intermediate_size=1280, hidden_size=768, n_heads=12, n_kv_heads=4, max_seq_len=400, vocab_size=520)
# 64 rows of keys: no tensor-core tile of 128, so prompts of any length come here; three layers of 16-row remainders
ONE_KV = dataclasses.replace(ODD, n_heads=4, n_kv_heads=1, head_dim=64)


def both(cfg, mix, before, tokens, want):
    out = []
    for together in (True, False):
        m = Model.synthetic(cfg, mix, seed=5)
        m.set_prefill_min_tokens(32 if together else 0)
        if before:
            m.forward(before, 0)
        n0 = K.launch_count()
        out.append((m.forward_logits(tokens, len(before), want).copy(), K.launch_count() - n0))
        m.close()
    (a, na), (b, nb) = out
    assert na < nb, "the tokens ran one at a time"
    # same products and 24-bit activations; sums in another order (1e-6) may round a cached key or value to its other F16 neighbour (2^-11 of it)
    assert np.abs(a - b).max() <= 3e-4 * np.abs(b).max(), np.abs(a - b).max() / np.abs(b).max()


@pytest.mark.parametrize("mix", ["Q4_K_M", "Q4_K", "Q5_K", "Q6_K", "Q8_0", "Q4_0"])
@pytest.mark.parametrize("n,before", [(3, 0), (8, 5), (9, 0), (31, 40)])
def test_together_equals_one_by_one(mix, n, before):
    rng = np.random.default_rng(n)
    toks = rng.integers(0, ODD.vocab_size, size=n + before).tolist()
    both(ODD, mix, toks[:before], toks[before:], [0, n // 2, n - 1])


@pytest.mark.parametrize("n", [65, 150])
def test_long_prompt_of_a_shape_without_tensor_core_tiles(n):
    toks = np.random.default_rng(1).integers(0, ONE_KV.vocab_size, size=n).tolist()
    both(ONE_KV, "Q6_K", [], toks, [1, 64, n - 1] if n > 65 else [1, 64])
