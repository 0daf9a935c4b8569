"""Torch tensors that no kernel may be given an address of are refused before the library is called (no GPU: the library is a stand-in that
counts its calls)."""
import ctypes

import pytest
import torch

from jitnn_b200 import DType, Gguf, Quant, Tensor, _lib


class Library:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def entry(*args):
            self.calls.append(name)
            return 0
        return entry


@pytest.fixture()
def library(monkeypatch):
    lib = Library()
    monkeypatch.setattr(_lib, "load", lambda: lib)
    return lib


@pytest.fixture()
def weight(library):
    w = Tensor(ctypes.c_void_p(1), DType.Q4_K, (4, 256), 0)
    yield w
    w._h = None


# on the CPU; another type, of the same size too; too small; strided
@pytest.mark.parametrize("out,message", [(torch.empty(4, 256), "output on cpu"), (torch.empty(4, 256, dtype=torch.float64), "FP32"),
                                         (torch.empty(4, 256, dtype=torch.int32), "FP32"), (torch.empty(4, 255), "1024 values"),
                                         (torch.empty(256, 4).T, "strided")])
def test_dequantize(library, weight, out, message):
    with pytest.raises(ValueError, match=message):
        Gguf.dequantize(weight, out)
    assert library.calls == []


@pytest.mark.parametrize("call", [lambda w, x: Gguf.linear(x, w), lambda w, x: Gguf.linearBf16(x.to(torch.bfloat16), w),
                                  lambda w, x: Gguf.linearBackward(x[:, :4].contiguous(), w), lambda w, x: Quant.quantizeQ8Blocks(x)])
def test_host_tensors(library, weight, call):
    with pytest.raises(ValueError, match="on cpu"):
        call(weight, torch.zeros(2, 256))
    assert library.calls == []
