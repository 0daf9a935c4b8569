"""The native front of calls on torch tensors against the general code in ops.py: the same bits for everything it takes, and it takes only plain cases."""
import threading

import numpy as np
import pytest
import torch

from jitnn_b200 import DType, Gguf, Quant, Tensor, ops, synth
from jitnn_b200.ops import _linear

pytestmark = pytest.mark.gpu

N, K = 96, 512


@pytest.fixture(scope="module")
def weight():
    raw = synth.random_valid_blocks("Q8_0", N, K, seed=1).numpy().reshape(-1)
    w = Tensor.quantized("Q8_0", raw, N, K)
    Gguf.linear(torch.zeros(1, K, device="cuda"), w)  # (the front comes in with the first torch tensor)
    assert ops._front is not None
    return w


class Slow:
    """ops without the front."""
    def __enter__(self):
        self.front, ops._front = ops._front, None

    def __exit__(self, *a):
        ops._front = self.front


def both(call):
    fast = call()
    with Slow():
        return fast, call()


@pytest.mark.parametrize("shape", [(K,), (1, K), (3, K), (2, 5, K), (0, K), (4, 0, K)])
def test_the_same_results(weight, shape):
    x = torch.randn(*shape, generator=torch.Generator().manual_seed(1)).cuda()
    b = torch.randn(N, generator=torch.Generator().manual_seed(2)).cuda()
    calls = [lambda: Gguf.linear(x, weight), lambda: Gguf.linear(x, weight, b), lambda: Quant.linear(x, weight, bias=b),
             lambda: Gguf.linear(torch.nn.Parameter(x), weight, torch.nn.Parameter(b)), lambda: Gguf.linearBf16(x.bfloat16(), weight, b),
             lambda: Gguf.linearBackward(x[..., :N].contiguous(), weight), lambda: Gguf.dequantize(weight, torch.empty(N, K, device="cuda"))]
    if x.numel() > 0:
        calls.append(lambda: Quant.quantizeQ8Blocks(x))
    for call in calls:
        fast, slow = both(call)
        assert type(fast) is torch.Tensor and fast.dtype == slow.dtype and fast.shape == slow.shape and fast.stride() == slow.stride()
        assert fast.device == slow.device and not fast.requires_grad and torch.equal(fast, slow)


def test_what_is_not_plain_goes_on_to_the_general_code(weight):
    f, x = ops._front, torch.randn(2, K, device="cuda")
    b = torch.zeros(N, device="cuda")

    class Sub(torch.Tensor):
        pass

    for args in ((x.double(), weight, None), (x.cpu(), weight, None), (x[:, :256].contiguous(), weight, None), (x.T.contiguous().T, weight, None), (x[0, 0], weight, None),
                 (x.numpy(force=True), weight, None), (x, "w", None), (x, weight, b.double()), (x, weight, b[:5]), (x, weight, b.cpu()), (x, weight, [0.0] * N),
                 (x.as_subclass(Sub), weight, None), (x, weight), (x.to_sparse(), weight, None)):
        assert f.linear(*args) is None
    assert f.quantize(x[:, :33].contiguous()) is None and f.quantize(x.T) is None and f.quantize(x[:0]) is None
    assert f.dequantize(weight, None) is None and f.dequantize(weight, torch.empty(N, K - 1, device="cuda")) is None
    assert f.backward(x, weight) is None
    strided = torch.randn(K, 2, device="cuda").T  # what the general code takes, it still takes
    assert torch.equal(Gguf.linear(strided, weight), Gguf.linear(strided.contiguous(), weight))
    for bad in (x.double(), x.cpu(), x[:, :256].contiguous()):
        with pytest.raises(ValueError):
            Gguf.linear(bad, weight)
    with pytest.raises(ValueError, match="16-byte"):  # an error of the library itself
        Gguf.linear(torch.randn(K + 1, device="cuda")[1:], weight)
    other = Tensor.quantized("Q8_0", synth.random_valid_blocks("Q8_0", 32, 64, seed=1).numpy().reshape(-1), 32, 64)
    other.release()
    assert f.linear(torch.zeros(1, 64, device="cuda"), other, None) is None
    with pytest.raises(RuntimeError, match="released"):
        Gguf.linear(torch.zeros(1, 64, device="cuda"), other)


def test_while_torch_calls_are_intercepted(weight):
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode
    x, seen = torch.randn(2, K, device="cuda"), []

    class Dispatch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    class Function(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    want = Gguf.linear(x, weight)
    with Dispatch():
        assert ops._front.linear(x, weight, None) is None
        assert torch.equal(Gguf.linear(x, weight), want)
    assert any("new_empty" in s or "empty" in s for s in seen)  # the general code's calls are seen, as before
    with Function():
        assert ops._front.linear(x, weight, None) is None
    assert ops._front.linear(x, weight, None) is not None
    taken = []

    def f(row):
        taken.append(ops._front.linear(row, weight, None) is None)
        return row

    torch.func.vmap(f)(x)
    assert taken == [True]
    with torch.inference_mode():
        assert Gguf.linear(x, weight).is_inference()


def test_streams_and_threads(weight):
    xs = [torch.randn(2, K, device="cuda") for _ in range(4)]
    want = [Gguf.linear(x, weight) for x in xs]
    torch.cuda.synchronize()
    bad = []

    def work(i):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for _ in range(200):
                y = Gguf.linear(xs[i], weight)
            s.synchronize()
            if not torch.equal(y, want[i]):
                bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert bad == []
