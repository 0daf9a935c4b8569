"""Dequantisation of all ten formats where a thread block's work ends, bit for bit: rows in fours, steps of 256 (warps go on from one row group to the next), and
the 2048 values of a thread block of the formats that are dequantised only."""
import numpy as np
import pytest
import torch

from jitnn_b200 import DType, Gguf, Tensor
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [d.name for d in DType])
@pytest.mark.parametrize("n,steps", [(1, 1), (3, 3), (4, 8), (5, 9), (7, 17), (130, 5)])
def test_ends_of_thread_blocks(t, n, steps):
    d = DType[t]
    for k in ([steps * 256] if d.blockValues() == 256 else [steps * 256, steps * 256 - 32]):
        raw = np.random.default_rng(n + k).integers(0, 256, (n * k // d.blockValues(), d.blockBytes()), dtype=np.uint8)
        for at in {"Q5_0": [0], "Q5_1": [0, 2], "Q2_K": [80, 82], "Q3_K": [108], "Q4_K": [0, 2], "Q5_K": [0, 2], "Q6_K": [208], "Q8_0": [0], "Q4_0": [0], "Q4_1": [0, 2]}[t]:
            raw[:, at + 1] &= 0xBB  # no NaN or Inf among the scales: their bits depend on the machine
        w = Tensor.quantized(t, raw.reshape(-1), n, k)
        out = torch.full((n * k + 8,), 7.0, device="cuda")
        Gguf.dequantize(w, out)
        want = oracle.dequantize(t, raw.reshape(-1))
        assert np.array_equal(out[:n * k].cpu().numpy().view(np.uint32), want.reshape(-1).view(np.uint32)), k
        assert bool((out[n * k:] == 7.0).all())


def test_the_kernel_in_front_still_reads_its_output():
    """The output is the input of the kernel in front of the call: its weights may be loaded early, its stores may not come early."""
    n, k = 512, 4096
    raw = np.random.default_rng(1).integers(0, 100, (n * k // 32, 34), dtype=np.uint8)
    w = Tensor.quantized("Q8_0", raw.reshape(-1), n, k)
    out, big = torch.empty(n, k, device="cuda"), torch.empty(16, n, k, device="cuda")
    for i in range(20):
        out.fill_(float(i))
        for part in big:
            part.copy_(out)
        Gguf.dequantize(w, out)
        assert bool((big == float(i)).all())
