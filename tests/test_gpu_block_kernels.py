"""Whole-weight kernels at the edges of their tiles: dequantisation of weights whose rows and steps of k do not fill a tile, and the
quantiser on values next to its rounding boundaries. Both are bit-exact with the oracle, so no tolerance is involved."""
import numpy as np
import pytest
import torch

from jitnn_b200 import Gguf, Quant, Tensor, synth
from oracle import oracle

pytestmark = pytest.mark.gpu

SMALL_BLOCKS = ["Q8_0", "Q4_0", "Q4_1", "Q5_0", "Q5_1"]
SUPER_BLOCKS = ["Q4_K", "Q5_K", "Q6_K", "Q2_K", "Q3_K"]


# k: one block; a step of 256 short of one block, and one block over; nine warps' worth of steps. n: around 4 rows a warp, 128 a tile.
@pytest.mark.parametrize("t,n,k", [(t, n, k) for t in SMALL_BLOCKS for n, k in [(1, 32), (3, 224), (5, 288), (129, 96), (130, 2336)]] +
                         [(t, n, k) for t in SUPER_BLOCKS for n, k in [(1, 256), (5, 512), (129, 2304), (257, 768)]])
def test_dequantize_partial_tiles(t, n, k):
    raw = synth.random_valid_blocks(t, n, k, seed=n + k).numpy()
    w = Tensor.quantized(t, raw, n, k)
    out = torch.full((n, k), float("nan"), device="cuda")
    got = Gguf.dequantize(w, out).cpu().numpy().reshape(-1)
    want = oracle.dequantize(t, raw)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    assert np.array_equal(w.blocks(), raw.reshape(-1))


# blocks: fewer than, exactly and one more than a thread block's 128; offset 4 bytes: buffers that are not 16-byte aligned
@pytest.mark.parametrize("blocks", [1, 127, 128, 129, 1000])
@pytest.mark.parametrize("aligned", [True, False])
def test_quantize_rounding_boundaries(blocks, aligned):
    rng = np.random.default_rng(blocks)
    x = rng.standard_normal((blocks, 32)).astype(np.float32)
    q = rng.integers(-127, 128, (blocks, 32)).astype(np.float64)
    # half of the blocks hold values a rounding step from (q + 1/2) d, on both sides and exactly there
    amax = np.abs(x).max(axis=1).astype(np.float64)
    d = (amax / 127.0).astype(np.float32).astype(np.float64)
    near = ((np.abs(q) - 0.5) * np.sign(q) * d[:, None]).astype(np.float32)
    step = rng.integers(-2, 3, near.shape).astype(np.int32)
    near = (near.view(np.int32) + np.where(near != 0, step, 0)).view(np.float32)
    near[:, 0] = amax
    x[::2] = near[::2]
    if blocks > 3:
        x[1] = 0.0
        x[3] *= np.float32(1e-41)  # subnormal values and scale
    buf = torch.zeros(blocks * 32 + 4, device="cuda")
    view = buf[:-4] if aligned else buf[1:-3]
    view.copy_(torch.from_numpy(x.reshape(-1)))
    got = Quant.quantizeQ8Blocks(view.reshape(blocks, 32)).cpu().numpy()
    assert np.array_equal(got, oracle.quantize_q8_0(x).reshape(-1))
