"""The tensor-core GEMM over GGUF blocks (csrc/prefill_blocks.cu) through the batched prompt pass, against the decode step's arithmetic: every format, token
counts around its tiles (one tile of 32, ragged, two column tiles, more than a wave), K of one and of several accumulators, Q6_K rows at any even address."""
import dataclasses

import numpy as np
import pytest

pytest.importorskip("torch")
from ntransformer_b200.engine import Model  # noqa: E402
from ntransformer_b200.model_spec import TINY  # noqa: E402

pytestmark = [pytest.mark.gpu]
# rows are multiples of 128; K of 768 (3 super-blocks: Q6_K rows of 630 bytes) and 2304 = 9 * 256 (two accumulators, the second with 4 k-blocks)
CFG = dataclasses.replace(TINY, hidden_size=768, n_heads=12, n_kv_heads=4, intermediate_size=2304, max_seq_len=700, vocab_size=520, n_layers=2)


def logits(mix, batched, before, tokens, want):
    m = Model.synthetic(CFG, mix, seed=11)
    m.set_prefill_min_tokens(32 if batched else 0)
    if before:
        m.forward(before, 0)
    out = m.forward_logits(tokens, len(before), want).copy()
    m.close()
    return out


@pytest.mark.parametrize("mix", ["Q4_K_M", "Q4_K", "Q5_K", "Q6_K", "Q8_0", "Q4_0"])
@pytest.mark.parametrize("n,before", [(32, 0), (45, 7), (300, 0)])
def test_batched_prompt_equals_one_by_one(mix, n, before):
    toks = np.random.default_rng(n).integers(0, CFG.vocab_size, size=n + before).tolist()
    want = [0, 31, n // 2, n - 1]
    want = sorted(set(want))
    a, b = (logits(mix, k, toks[:before], toks[before:], want) for k in (True, False))
    # 96 products onto one accumulator, each truncated at 2^-24 of it, and weights and activations as pairs of F16 (2^-22): below 1e-5 a product; two layers
    # and cached keys that round to the other F16 neighbour: 5e-4 of the largest logit
    assert np.abs(a - b).max() <= 5e-4 * np.abs(b).max(), np.abs(a - b).max() / np.abs(b).max()
