"""NT_B200_NO_PDL: no launch of a Model is programmatic, in steps, turns and prompts (csrc/kernels_internal.h Launches)."""
import numpy as np
import pytest

pytest.importorskip("torch")
from ntransformer_b200 import kernels as K  # noqa: E402
from ntransformer_b200._lib import lib  # noqa: E402
from ntransformer_b200.engine import Model  # noqa: E402
from ntransformer_b200.model_spec import TINY  # noqa: E402

pytestmark = [pytest.mark.gpu]


@pytest.mark.parametrize("graph", ["", "1"])
@pytest.mark.parametrize("mix", ["Q4_K_M", "Q8_0", "F16"])
def test_the_switch_reaches_every_launch(mix, graph, monkeypatch):
    if graph:
        monkeypatch.setenv("NT_B200_NO_GRAPH", graph)
    toks = np.random.default_rng(1).integers(3, TINY.vocab_size, size=80).tolist()
    out = []
    for off in (False, True):
        if off:
            monkeypatch.setenv("NT_B200_NO_PDL", "1")
        m = Model.synthetic(TINY, mix, seed=2)
        got, at = [], 0
        for n in (40, 1, 1, 12, 3):
            edges, launches = lib().nt_b200_programmatic_count(), K.launch_count()
            got.append(m.forward(toks[at:at + n], at).copy())
            at += n
            assert K.launch_count() > launches
            assert lib().nt_b200_programmatic_count() == edges if off else True
        if not off:
            assert lib().nt_b200_programmatic_count() > 0
        m.close()
        out.append(got)
    assert all(np.array_equal(a, b) for a, b in zip(*out))
