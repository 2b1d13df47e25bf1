"""The launcher boundary's extension (csrc/fast_call.cpp) hands every entry the arguments that ctypes hands it, and leaves to ctypes what it does not take."""
import ctypes as C
import sys
import sysconfig

import numpy as np
import pytest
import torch

import ntransformer_b200
from ntransformer_b200 import _fast, kernels
from ntransformer_b200._lib import SIGNATURES, lib


class Owner:
    """Stands for a tensor."""
    def __init__(self, address, cuda=True, flat=True):
        self.address, self.is_cuda, self.flat = address, cuda, flat

    def is_contiguous(self):
        return self.flat

    def data_ptr(self):
        return self.address


class Stream:
    cuda_stream = 0x7F0000000010


@pytest.fixture
def entries():
    """The extension bound to callbacks that note what they get; the library's own again afterwards."""
    got, other, keep, table = [], [], [], {}
    for n in _fast.ENTRIES:
        f = C.CFUNCTYPE(None, *SIGNATURES["nt_b200_" + n][1])(lambda *a, n=n: got.append((n, a)))
        keep.append(f)
        table[n] = C.cast(f, C.c_void_p).value
    _fast.bind(Owner, lambda d: 0x5000 + d, lambda: 3, lambda: None, lambda n, a: other.append((n, a)), table)
    yield got, other
    kernels._entries = None
    kernels._fast()


@pytest.mark.parametrize("name", _fast.ENTRIES)
def test_arguments_arrive(entries, name):
    got, other = entries
    types = SIGNATURES["nt_b200_" + name][1]
    address = 0xFFFF800000001000                              # above a signed 64-bit integer
    values = {C.c_void_p: [Owner(address), address, 16], C.c_int: [7, -1, 2**31 - 1], C.c_float: [0.1, 3, float("inf")]}
    for i in range(3):
        args = [values[t][i] for t in types[:-1]]
        want = tuple(address if isinstance(a, Owner) else C.c_float(a).value if t is C.c_float else a for a, t in zip(args, types))
        for stream, s in ((None, 0x5003), (Stream, Stream.cuda_stream), (0, None), (0x40, 0x40)):
            getattr(_fast, name)(*args, stream)
            assert got.pop() == (name, want + (s,))
    getattr(_fast, name)(*[None if t is C.c_void_p else True for t in types])
    assert got.pop()[1] == tuple(None if t is C.c_void_p else 1 for t in types[:-1]) + (0x5003,)
    assert not got and not other
    with pytest.raises(TypeError):
        getattr(_fast, name)(*[1] * (len(types) - 1))


def test_other_forms_go_through_ctypes(entries):
    got, other = entries
    for args in ((C.c_void_p(8), 8, 8, 4, 0), (8, 8, 8, np.int64(4), 0), (8, 8, 8, 4.5, 0), (8, 8, 8, 4, np.int64(3))):
        _fast.add(*args)
        assert other.pop() == ("add", args)
    _fast.softmax(8, 8, torch.tensor(3), 4, 0)
    assert other.pop()[0] == "softmax"
    for bad in (Owner(8, cuda=False), Owner(8, flat=False)):
        with pytest.raises(AssertionError, match="contiguous CUDA tensor"):
            _fast.add(8, 8, bad, 4, 0)
    assert not got and not other


def test_the_other_route_refuses_as_before():
    with pytest.raises(C.ArgumentError):
        kernels.launch_add(None, None, None, 4.5, 0)
    assert kernels._fast() is _fast and lib() is not None


def test_without_the_extension_launches_go_through_ctypes(monkeypatch):
    got = []

    class Library:
        def __getattr__(self, name):
            return lambda *a: got.append((name, a))

    monkeypatch.delattr(ntransformer_b200, "_fast")
    monkeypatch.setitem(sys.modules, "ntransformer_b200._fast", None)         # an ImportError
    monkeypatch.setattr(kernels, "_entries", None)
    monkeypatch.setattr(kernels, "lib", Library)
    kernels.launch_rope(8, None, 16, 1, 2, 3, 4, 64, 1e4, 1.0, True, stream=5)
    kernels.launch_add(8, 16, 24, 7, Stream)
    assert got == [("nt_b200_rope", (8, None, 16, 1, 2, 3, 4, 64, 1e4, 1.0, 1, 5)), ("nt_b200_add", (8, 16, 24, 7, Stream.cuda_stream))]


def test_the_extension_is_of_this_interpreter_alone():
    assert _fast.__file__.endswith(sysconfig.get_config_var("EXT_SUFFIX"))


@pytest.mark.gpu
def test_forms_of_arguments_on_the_device():
    a, b = torch.arange(100.0, device="cuda"), torch.full((100,), 0.5, device="cuda")
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    for n, stream, pointer in ((100, None, lambda t: t), (np.int32(100), side, lambda t: t.data_ptr()), (100, side.cuda_stream, lambda t: C.c_void_p(t.data_ptr()))):
        out = torch.zeros(100, device="cuda")
        torch.cuda.synchronize()
        kernels.launch_add(pointer(out), pointer(a), pointer(b), n, stream)
        torch.cuda.synchronize()
        assert torch.equal(out, a + b)
    with torch.cuda.stream(side):                             # the current stream is looked up at each call
        torch.cuda._sleep(20_000_000)
        c = torch.zeros(100, device="cuda")
        kernels.launch_add(c, a, b, 100)
    side.synchronize()
    assert torch.equal(c, a + b)
