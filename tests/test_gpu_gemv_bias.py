"""A decode linear with and without a bias: for Q4_K and Q5_K these are two instances of a kernel. The bias is added to the finished sum, so the one is the other plus the
bias, rounded once: the same bits."""
import pytest
import torch

from jitnn_b200 import Gguf, Tensor, synth

pytestmark = pytest.mark.gpu

# one row of W; a tile's rest; several tiles a thread block; k that is made into an image inside, in front, and in slices
SHAPES = [(1, 256), (17, 4096), (130, 8192), (9001, 512), (300, 40960)]


@pytest.mark.parametrize("n,k", SHAPES)
@pytest.mark.parametrize("t", ["Q4_K", "Q5_K", "Q6_K", "Q8_0"])
def test_bias_is_added_to_the_same_sums(t, n, k):
    w = Tensor.quantized(t, synth.random_valid_blocks(t, n, k, seed=n).numpy().reshape(-1), n, k)
    g = torch.Generator(device="cuda").manual_seed(k)
    b = torch.randn(n, generator=g, device="cuda")
    for m in range(1, 9):
        x = torch.randn(m, k, generator=g, device="cuda")
        none = Gguf.linear(x, w)
        assert torch.equal(Gguf.linear(x, w, b), none + b), m
        assert torch.equal(Gguf.linear(x, w), none), m


# one launch whose contraction is shared by thread blocks; whole tiles and such a launch behind them; the matrix kernel, both precisions
@pytest.mark.parametrize("t,n,k,m,bf16", [("Q6_K", 1000, 8192, 8, False), ("Q4_K", 2049, 4096, 16, False), ("Q8_0", 19000, 2048, 8, False), ("Q4_K", 1001, 4096, 24, False),
                                          ("Q4_K", 1000, 8192, 64, False), ("Q6_K", 1004, 8192, 64, True)])
def test_a_bias_that_the_kernel_in_front_writes(t, n, k, m, bf16):
    """Split contractions add the bias in an epilogue of their own, also by threads that have not waited for the kernel in front themselves."""
    w = Tensor.quantized(t, synth.random_valid_blocks(t, n, k, seed=n).numpy().reshape(-1), n, k)
    wb = Tensor.quantized("Q8_0", synth.random_valid_blocks("Q8_0", n, 256, seed=k).numpy().reshape(-1), n, 256)
    g = torch.Generator(device="cuda").manual_seed(k)
    x = torch.randn(m, k, generator=g, device="cuda")
    linear = Gguf.linearBf16 if bf16 else Gguf.linear
    x = x.to(torch.bfloat16) if bf16 else x
    none, z = linear(x, w), torch.randn(40, 1, 256, generator=g, device="cuda")
    ys, bs = [], []
    for i in range(len(z)):
        b = Gguf.linear(z[i], wb).view(n)
        ys.append(linear(x, w, b))
        bs.append(b.clone())
    for y, b in zip(ys, bs):
        assert torch.equal(y, none + b)
