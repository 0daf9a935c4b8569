"""The FP32 product of up to 16 rows of x on the tensor cores (rows kernel) where its tiles, ranges of k and launches end.

The reference is the product of the oracle's dequantised weights in double. x keeps 22 significant bits, products are exact, sums of at most 256
terms are taken by the tensor core before they are added up in FP32 registers: 2e-7 of the result's norm on ordinary weights, and 1e-5
leaves room for cancellation.
"""
import numpy as np
import pytest
import torch

from conftest import LINEAR_TYPES
from jitnn_b200 import Gguf, Tensor, device_status, synth
from oracle import oracle

pytestmark = pytest.mark.gpu

REL = 1e-5

# One row of W; a second tile's first row; one unit of k, fewer units than ranges, no multiple of the ranges; few tiles with k over 8, 4 and 2 thread blocks;
# two waves of whole tiles whose scales of x stay from tile to tile; whole tiles and what is left in two launches; a cluster launch in front of another.
# (test_rows_plan.py has the launches of each.)
SHAPES = [(1, 256, 9), (129, 512, 16), (128, 2816, 10), (4096, 4096, 13), (1024, 8192, 16), (2000, 16384, 9), (19000, 2048, 12), (30000, 1024, 16),
          (6400, 4096, 12), (18950, 2560, 10), (23200, 3584, 15), (9500, 8192, 11), (4300, 14080, 14)]


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
