"""Decode steps whose feed-forward is so wide that the down projection takes a vector quantised by a launch of its own (Model::down_over_xq), against the oracle:
widths on both sides of the rule, the longest that the block GEMVs take, and a format whose rows the pre-quantised kernel does not take."""
import dataclasses

import numpy as np
import pytest

pytest.importorskip("torch")
from ntransformer_b200.engine import Model  # noqa: E402
from ntransformer_b200.gguf_write import synthetic_tensors_np, write_gguf  # noqa: E402
from ntransformer_b200.model_spec import TINY  # noqa: E402
from oracle import oracle as O  # noqa: E402

pytestmark = [pytest.mark.gpu]


# mixed: attention in F16, so that the step is not the short chain of launches
@pytest.mark.parametrize("mix,inter,mixed", [("Q4_K", 28672, False), ("Q4_K", 32768, False), ("Q8_0", 26368, False), ("Q8_0", 28672, False), ("Q6_K", 32768, False),
                                             ("Q6_K", 33024, False), ("Q4_0", 36864, False), ("Q5_K", 49152, False), ("Q8_0", 49152, False), ("Q4_K", 32768, True)])
def test_wide_feed_forward(tmp_path, mix, inter, mixed):
    cfg = dataclasses.replace(TINY, intermediate_size=inter, n_layers=2)
    tensors = synthetic_tensors_np(cfg, mix, seed=7)
    if mixed:
        tensors.update({n: t for n, t in synthetic_tensors_np(cfg, "F16", seed=8).items() if "attn_" in n})
    write_gguf(tmp_path / "m.gguf", cfg, tensors)
    m = Model.load(tmp_path / "m.gguf", cfg.max_seq_len)
    om = O.Model(cfg.dict(), {n: (np.ascontiguousarray(a), int(dt)) for n, (a, dt, r, c) in tensors.items()})
    for pos, tok in enumerate([1, 17, 300 % cfg.vocab_size, 5]):
        got, want = m.forward([tok], pos).copy(), om.forward([tok], pos)
        assert np.abs(got - want).max() <= 1e-3 * np.abs(want).max()
    m.close()
