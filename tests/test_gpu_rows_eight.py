"""The rows kernel with up to 8 rows of x, and the formats whose scales its sums are multiplied by, where they can go wrong.

The reference is the product of the oracle's dequantised weights in double. x keeps 22 bits of the largest of its 256 neighbours (up to four standard deviations),
products are exact, sums of at most 256 terms are taken by the tensor core. So an element is off by some 4 x 2^-22 / sqrt(12) = 2.8e-7 of the root of its terms' squares,
and one in a hundred thousand by five times that: 1.5e-6 at most, 3.5e-7 of the result's norm, measured over these shapes.
"""
import ctypes

import numpy as np
import pytest
import torch

import jitnn_b200
from conftest import LINEAR_TYPES
from jitnn_b200 import Gguf, Tensor, device_status, synth
from oracle import oracle

pytestmark = pytest.mark.gpu

REL = 1e-5  # where a few blocks make up a result
NORM, ELEMENT = 1e-6, 3e-6  # ordinary weights
GROUPED = ["Q6_K", "Q8_0", "Q4_0", "Q4_1"]
# One row of W; a second tile's first row; fewer units than ranges; clusters of 2, 4 and 8; two waves; two launches.
SHAPES = [(1, 256), (129, 512), (128, 2816), (1024, 8192), (4096, 4096), (6400, 4096), (19000, 2048), (9500, 8192)]


def product(t, n, k, seed):
    raw = synth.random_valid_blocks(t, n, k, seed=seed).numpy().reshape(-1)
    return raw, Tensor.quantized(t, raw, n, k), torch.from_numpy(oracle.dequantize(t, raw).reshape(n, k)).cuda().double()


@pytest.mark.parametrize("n,k", SHAPES)
@pytest.mark.parametrize("t", GROUPED)
def test_up_to_eight_rows(t, n, k):
    raw, w, wd = product(t, n, k, n)
    b = torch.randn(n, generator=torch.Generator().manual_seed(n)).cuda()
    for m in (3, 5, 8):
        x = torch.randn(m, k, generator=torch.Generator().manual_seed(m)).cuda()
        ref, of = x.double() @ wd.T + b.double(), ((x.double() ** 2) @ (wd ** 2).T + b.double() ** 2).sqrt()
        y = Gguf.linear(x, w, b)
        assert float((y.double() - ref).norm() / ref.norm()) <= NORM
        assert float(((y.double() - ref).abs() / of).max()) <= ELEMENT  # (a single column or the edge of a tile would be lost in the norm)
        for _ in range(5):
            assert torch.equal(Gguf.linear(x, w, b), y)
        if n > 128:  # a row shard gives the bits of the whole weight, whatever its launches are
            shard = Tensor.quantized(t, raw, n, k, rows=(0, n // 3))
            assert torch.equal(Gguf.linear(x, shard, b[:n // 3]), y[:, :n // 3])
            shard.release()
    assert device_status(0) == 0


@pytest.mark.parametrize("m", [8, 16])
@pytest.mark.parametrize("t", GROUPED)
def test_scales_of_every_size(t, m):
    """Block scales from the smallest subnormal half to the largest half, side by side; each row of W is held against its own size."""
    n, k = 200, 1024
    raw = synth.random_valid_blocks(t, n, k, seed=5).numpy().reshape(n, -1).copy()
    size = {"Q6_K": 210, "Q8_0": 34, "Q4_0": 18, "Q4_1": 20}[t]
    blocks = raw.reshape(-1, size)
    d = np.exp2(np.random.default_rng(2).uniform(-24, 15.9, blocks.shape[0])).astype(np.float16)
    for at in {"Q6_K": [208], "Q8_0": [0], "Q4_0": [0], "Q4_1": [0, 2]}[t]:
        blocks[:, at:at + 2] = d.view(np.uint8).reshape(-1, 2)
    raw = raw.reshape(-1)
    w, wd = Tensor.quantized(t, raw, n, k), torch.from_numpy(oracle.dequantize(t, raw).reshape(n, k)).cuda().double()
    x = torch.randn(m, k, generator=torch.Generator().manual_seed(3)).cuda()
    y, ref, size = Gguf.linear(x, w).double(), x.double() @ wd.T, (x.double() ** 2) @ (wd ** 2).T
    assert float(((y - ref).abs() / size.sqrt()).max()) <= REL


@pytest.mark.parametrize("t", LINEAR_TYPES)
def test_nan_and_inf_reach_their_rows_alone(t):
    n, k, m = 300, 1024, 8
    _, w, wd = product(t, n, k, 3)
    x = torch.randn(m, k, generator=torch.Generator().manual_seed(1)).cuda()
    x[2, 17], x[7, 1000] = float("nan"), float("inf")
    x[4] = 0.0
    y = Gguf.linear(x, w)
    bad = ~torch.isfinite(y)
    assert bool(bad[2].all()) and bool(bad[7].all()) and bool((y[4] == 0).all())
    rows = [r for r in range(m) if r not in (2, 7)]
    ref = x[rows].double() @ wd.T
    assert float((y[rows].double() - ref).norm() / ref.norm()) <= NORM


@pytest.mark.parametrize("t", ["Q8_0", "Q4_0", "Q4_1"])
def test_three_rows_are_captured_after_a_call_with_one(t):
    """The row count at which the kernel changes needs no scratch buffer that a call with one row has not left."""
    n, k = 512, 28672
    _, w, _ = product(t, n, k, 4)
    stream = torch.cuda.Stream()
    x = torch.randn(4, k, generator=torch.Generator().manual_seed(1)).cuda()
    want = Gguf.linear(x, w)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        Gguf.linear(x[:1], w)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        y = Gguf.linear(x, w)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)


# k that is no multiple of 256, of which the decode kernels take no rows; k of which those of Q8_0 take one row but not two; a call with fewer rows in front of both
@pytest.mark.parametrize("t,k", [("Q8_0", 1056), ("Q4_0", 1056), ("Q8_0", 24576)])
@pytest.mark.parametrize("first,then", [((8,), 4), ((4,), 8), ((16,), 3), ((1, 4), 8), ((1,), 3)])
def test_a_call_with_other_rows_leaves_the_scratch_for_a_capture(t, k, first, then):
    if k == 1056 and first == (1,):
        pytest.skip("one row has no scratch")
    n = 512
    _, w, _ = product(t, n, k, 4)
    handle = ctypes.c_void_p()  # of a stream that no other test has used: torch hands out the same few again
    assert int(torch.cuda.cudart().cudaStreamCreate(ctypes.addressof(handle))) == 0
    stream = torch.cuda.ExternalStream(handle.value)
    x = torch.randn(16, k, generator=torch.Generator().manual_seed(1)).cuda()
    want = Gguf.linear(x[:then], w)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        for m in first:
            Gguf.linear(x[:m], w)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        y = Gguf.linear(x[:then], w)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)
