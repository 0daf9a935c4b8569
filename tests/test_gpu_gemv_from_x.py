"""The decode GEMVs of Q6_K and the 32-element formats at the line between building x's image themselves and reading that of an image kernel.

Both make the same digits of x and sum in the same order, so that neighbours across the line differ by nothing but the launches. The reference is the product
of the oracle's dequantised weights in double; x keeps 22 bits of the largest of its 256 neighbours, 4e-7 of what is added up on ordinary weights.
"""
import numpy as np
import pytest
import torch

import jitnn_b200
from jitnn_b200 import Gguf, Tensor, device_status, synth
from oracle import oracle

pytestmark = pytest.mark.gpu

REL = 1e-5
LINE = 8192  # values of x


@pytest.mark.parametrize("n", [1, 16, 17, 5000])
@pytest.mark.parametrize("k,m", [(256, 1), (256, 2), (2048, 2), (2304, 1), (4096, 2), (4352, 2), (8192, 1), (8448, 1)])
@pytest.mark.parametrize("t", ["Q6_K", "Q8_0", "Q4_0", "Q4_1"])
def test_one_launch_up_to_the_line(t, k, m, n):
    L = jitnn_b200.load()
    raw = synth.random_valid_blocks(t, n, k, seed=k + n).numpy().reshape(-1)
    w, wd = Tensor.quantized(t, raw, n, k), torch.from_numpy(oracle.dequantize(t, raw).reshape(n, k)).cuda().double()
    g = torch.Generator().manual_seed(m)
    x, b = torch.randn(m, k, generator=g).cuda(), torch.randn(n, generator=g).cuda()
    before = L.jq_launch_count()
    y = Gguf.linear(x, w, b)
    assert L.jq_launch_count() - before == (1 if m * k <= LINE else 2)
    ref, size = x.double() @ wd.T + b.double(), ((x.double() ** 2) @ (wd ** 2).T).sqrt() + b.double().abs()  # (what is added up, as a result may be next to zero)
    assert float(((y.double() - ref).abs() / size).max()) <= REL
    # host arrays: the image kernel reads x once, the same digits
    assert np.array_equal(Gguf.linear(x.cpu().numpy(), w, b.cpu().numpy()), y.cpu().numpy())
    assert device_status(0) == 0


@pytest.mark.parametrize("t", ["Q6_K", "Q8_0", "Q4_0", "Q4_1"])
def test_x_of_every_size_and_of_the_kernel_in_front(t):
    """Zeros, subnormals, the largest floats, ties of the fixed point, NaN and Inf, in x that the kernel in front of the call writes."""
    n, k = 64, 1024
    raw = synth.random_valid_blocks(t, n, k, seed=2).numpy().reshape(-1)
    w, wd = Tensor.quantized(t, raw, n, k), torch.from_numpy(oracle.dequantize(t, raw).reshape(n, k)).cuda().double()
    base = torch.randn(2, k, generator=torch.Generator().manual_seed(1)).cuda()
    x = torch.empty_like(base)
    cases = [base * 0.0, base * 1e-39, base * 1e30, torch.round(base * 64) + 0.5, base.clone(), base.clone()]
    cases[4][0, 300], cases[5][1, 1023] = float("nan"), float("-inf")
    for i, c in enumerate(cases):
        x.copy_(c)
        y = Gguf.linear(x, w)
        ref = c.double() @ wd.T
        for row in range(2):
            if not bool(torch.isfinite(c[row]).all()):
                assert not bool(torch.isfinite(y[row]).any())
            elif i in (0, 1):  # below the smallest scale of the image x is rounded to a fixed grid of 2^-124
                assert float((y[row].double() - ref[row]).abs().max()) <= 2.0 ** -124 * float(wd.abs().sum(1).max())
            else:
                assert float((y[row].double() - ref[row]).norm() / ref[row].norm()) <= REL
