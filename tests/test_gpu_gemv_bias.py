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
