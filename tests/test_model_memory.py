"""Every buffer of Model::PrefillBuffers (csrc/engine/model.h) that is an allocation of its own is given back by ~Model (csrc/engine/model.cu)."""
import re
from pathlib import Path

ENGINE = Path(__file__).resolve().parent.parent / "ntransformer_b200" / "csrc" / "engine"


def test_prefill_buffers_are_freed():
    struct = re.search(r"struct PrefillBuffers \{(.*?)\n    \} pf_;", (ENGINE / "model.h").read_text(), re.S).group(1)
    struct = re.sub(r"//[^\n]*", "", struct)
    names = set(re.findall(r"\*\s*(\w+) = nullptr", struct))
    assert {"x", "ws2", "count", "wide"} <= names
    destructor = re.search(r"\nModel::~Model\(\) \{(.*?)\n\}", (ENGINE / "model.cu").read_text(), re.S).group(1)
    freed = set(re.findall(r"pf_\.(\w+)", destructor))
    assert names <= freed, names - freed
