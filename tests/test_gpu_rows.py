"""The FP32 product of up to 16 rows of x on the tensor cores (rows kernel) where its tiles, ranges of k and launches end.

The reference is the product of the oracle's dequantised weights in double. x keeps 22 significant bits, products are exact, sums of at most 256
terms are taken by the tensor core before they are added up in FP32 registers: 2e-7 of the result's norm on ordinary weights, and 1e-5
leaves room for cancellation.
"""
import numpy as np
import pytest
import torch

import jitnn_b200
from conftest import LINEAR_TYPES
from jitnn_b200 import Gguf, Tensor, device_status, synth
from jitnn_b200._lib import JQ_MEM_DEVICE, check
from oracle import oracle

pytestmark = pytest.mark.gpu

REL = 1e-5

# One row of W; a second tile's first row; one unit of k, fewer units than ranges, no multiple of the ranges; few tiles with k over 8, 4 and 2 thread blocks;
# two waves of whole tiles whose scales of x stay from tile to tile; whole tiles and what is left in two launches; a cluster launch in front of another.
# (test_rows_plan.py has the launches of each.)
SHAPES = [(1, 256, 9), (129, 512, 16), (128, 2816, 10), (4096, 4096, 13), (1024, 8192, 16), (2000, 16384, 9), (19000, 2048, 12), (30000, 1024, 16),
          (6400, 4096, 12), (18950, 2560, 10), (23200, 3584, 15), (9500, 8192, 11), (4300, 14080, 14)]
TWO_LAUNCHES, THREE_LAUNCHES = (9500, 8192), (28500, 11264)


@pytest.mark.parametrize("n,k,m", SHAPES)
@pytest.mark.parametrize("t", LINEAR_TYPES)
def test_against_the_oracle(t, n, k, m):
    raw = synth.random_valid_blocks(t, n, k, seed=n + m).numpy().reshape(-1)
    w, wd = Tensor.quantized(t, raw, n, k), torch.from_numpy(oracle.dequantize(t, raw).reshape(n, k)).cuda().double()
    g = torch.Generator().manual_seed(k)
    x, b = torch.randn(m, k, generator=g).cuda(), torch.randn(n, generator=g).cuda()
    ref = x.double() @ wd.T + b.double()
    y = Gguf.linear(x, w, b)
    assert float((y.double() - ref).norm() / ref.norm()) <= REL
    for _ in range(20):
        assert torch.equal(Gguf.linear(x, w, b), y)
    assert device_status(0) == 0


@pytest.mark.parametrize("t", LINEAR_TYPES)
def test_nan_and_inf_reach_their_rows_alone(t):
    n, k, m = 300, 1024, 16
    raw = synth.random_valid_blocks(t, n, k, seed=3).numpy().reshape(-1)
    w, wd = Tensor.quantized(t, raw, n, k), torch.from_numpy(oracle.dequantize(t, raw).reshape(n, k)).cuda().double()
    x = torch.randn(m, k, generator=torch.Generator().manual_seed(1)).cuda()
    x[2, 17], x[15, 1000] = float("nan"), float("inf")
    x[7] = 0.0
    y = Gguf.linear(x, w)
    bad = ~torch.isfinite(y)
    assert bool(bad[2].all()) and bool(bad[15].all()) and bool((y[7] == 0).all())
    rows = [r for r in range(m) if r not in (2, 15)]
    ref = x[rows].double() @ wd.T
    assert float((y[rows].double() - ref).norm() / ref.norm()) <= REL


@pytest.mark.parametrize("t", LINEAR_TYPES)
def test_calls_on_other_x_in_turn(t):
    """Products in two and in three launches, the ones behind reading an image of x that they do not wait for: x is written by the kernel in front of the
    call, its image lies where that of the call before lay (another x, scales a thousand times larger, another k), y holds NaN until its launches write it,
    and the kernel behind the call reads it."""
    L = jitnn_b200.load()
    m, g = 16, torch.Generator().manual_seed(1)
    stream = torch.cuda.current_stream().cuda_stream
    products = []  # weight, x in use, y, [(x, the result of a call alone)]
    for n, k in (TWO_LAUNCHES, THREE_LAUNCHES):
        raw = synth.random_valid_blocks(t, n, k, seed=n).numpy().reshape(-1)
        w, values = Tensor.quantized(t, raw, n, k), torch.from_numpy(oracle.dequantize(t, raw).reshape(n, k)).cuda()
        results = []
        for size in (1.0, 1000.0):
            x = torch.randn(m, k, generator=g).cuda() * size
            y = Gguf.linear(x, w)
            torch.cuda.synchronize()
            ref = torch.cat([x.double() @ part.double().T for part in values.split(4096)], dim=1)
            assert float((y.double() - ref).norm() / ref.norm()) <= REL
            results.append((x, y))
        products.append((w, torch.empty(m, k, device="cuda"), torch.empty(m, n, device="cuda"), results))
    got = []
    for i in range(40):
        w, x, y, results = products[i // 2 % 2 if i < 20 else i % 2]
        use = results[(i + i // 4) % 2]
        x.copy_(use[0])
        y.fill_(float("nan"))
        check(L.jq_linear_f32(w._handle(), x.data_ptr(), m, None, y.data_ptr(), JQ_MEM_DEVICE, stream))
        got.append((y.clone(), use[1]))
    assert all(torch.equal(y, alone) for y, alone in got)
    assert device_status(0) == 0
