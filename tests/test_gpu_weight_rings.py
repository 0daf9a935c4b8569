"""The decode kernels' rings of weights in shared memory: a slot is filled again only when what was in it has been read.

A copy that lands on values which a warp has yet to read shows as weights of another block. Two x in turn, nothing between the calls but the order of
the stream: every result has the bits of a call alone, which is close to the product of the oracle's dequantised weights in double (the kernels keep
22 significant bits of x and are off by 3e-7 of the result's norm; 1e-5 leaves room for cancellation).
"""
import pytest
import torch

import jitnn_b200
from jitnn_b200 import Gguf, Tensor, device_status, synth
from oracle import oracle

pytestmark = pytest.mark.gpu

REL = 1e-5


def calls_in_turn(t, n, k, m):
    raw = synth.random_valid_blocks(t, n, k, seed=n + m).numpy().reshape(-1)
    w, wd = Tensor.quantized(t, raw, n, k), torch.from_numpy(oracle.dequantize(t, raw).reshape(n, k)).cuda().double()
    xs = [torch.randn(m, k, generator=torch.Generator().manual_seed(s)).cuda() * 10.0 ** s for s in range(2)]
    alone = []
    for x in xs:
        y = Gguf.linear(x, w)
        torch.cuda.synchronize()
        ref = x.double() @ wd.T
        assert float((y.double() - ref).norm() / ref.norm()) <= REL
        alone.append(y)
    for _ in range(10):
        ys = [Gguf.linear(xs[i % 2], w) for i in range(20)]
        assert all(torch.equal(y, alone[i % 2]) for i, y in enumerate(ys))
    assert device_status(0) == 0


# instances for 1, 2 and 4 rows of x, many tiles per thread block and few, one super-block of k and so many that x's image comes in slices
@pytest.mark.parametrize("n,k,m", [(11008, 4096, 1), (32000, 4096, 4), (4096, 11008, 2), (300, 256, 1), (2000, 28672, 4)])
def test_q6_k(n, k, m):
    calls_in_turn("Q6_K", n, k, m)


# instances for 1, 2, 4 and 8 rows of x, and the forms of 8 and 16 warps
@pytest.mark.parametrize("t", ["Q4_K", "Q5_K"])
@pytest.mark.parametrize("n,k,m", [(11008, 4096, 1), (32000, 4096, 8), (4096, 11008, 2), (300, 256, 1), (2000, 28672, 4)])
def test_q4_k_q5_k(t, n, k, m):
    calls_in_turn(t, n, k, m)


# the tcgen05 GEMV, whose ring of x's image holds the weights and sums that its epilogue reads: more than 8 rows, or a k whose image does not stay in
# shared memory; tiles of one thread block, of two and of more
@pytest.mark.parametrize("t,n,k,m", [("Q4_K", 11008, 4096, 16), ("Q5_K", 4096, 11008, 8), ("Q5_K", 1000, 8192, 16), ("Q4_K", 4096, 28672, 1)])
def test_tcgen05_gemv(t, n, k, m):
    L = jitnn_b200.load()
    L.jq_set_option(b"gemv_tcgen05", 1)
    try:
        calls_in_turn(t, n, k, m)
    finally:
        L.jq_set_option(b"gemv_tcgen05", 0)


@pytest.mark.parametrize("t", ["Q8_0", "Q4_0", "Q4_1"])
@pytest.mark.parametrize("n,k,m", [(11008, 4096, 1), (4096, 11008, 2), (300, 256, 1)])
def test_32_element_formats(t, n, k, m):
    calls_in_turn(t, n, k, m)
