"""The tensor-core matrix kernel (FP32 products with many rows of x, and the input gradient) where its tiles, ranges and rings end, and the values
that are hard on it and, with up to 16 rows of x, on the rows kernel.

The reference is the product of the oracle's dequantised weights in double. Both operands of the kernel keep 22 significant bits (2^-22 each),
and sums of at most 272 terms are taken in FP32 by the tensor core before they are added up in FP32 registers: 3e-7 of the result's norm or
less on ordinary weights (the last test), and 1e-5 leaves room for cancellation.
"""
import numpy as np
import pytest
import torch

from conftest import LINEAR_TYPES
from jitnn_b200 import Gguf, Quant, Tensor, device_status, synth
from oracle import oracle

pytestmark = pytest.mark.gpu

REL = 1e-5


def weight(t, n, k, seed, edit=None):
    raw = synth.random_valid_blocks(t, n, k, seed=seed).numpy().reshape(-1)
    if edit is not None:
        edit(raw)
    return Tensor.quantized(t, raw, n, k), torch.from_numpy(oracle.dequantize(t, raw).reshape(n, k)).cuda().double()


def close(y, ref):
    assert device_status(0) == 0
    err = float((y.double() - ref).norm() / ref.norm())
    assert err <= REL, err


# one feature; one row of a second 128-feature tile; one unit of k and more units than rings hold; the widths of the two instances (32 rows of
# x) and of a tile (128); few enough tiles for k in ranges (1, 2, 4 of them); more tiles than SMs (persistent CTAs)
SHAPES = [(1, 256, 17), (129, 512, 32), (128, 2816, 33), (257, 4096, 128), (640, 1024, 129), (4096, 4096, 40), (20000, 512, 150)]


@pytest.mark.parametrize("n,k,m", SHAPES)
@pytest.mark.parametrize("t", LINEAR_TYPES)
def test_linear(t, n, k, m):
    w, wd = weight(t, n, k, seed=n + m)
    g = torch.Generator().manual_seed(k)
    x, b = torch.randn(m, k, generator=g).cuda(), torch.randn(n, generator=g).cuda()
    close(Gguf.linear(x, w, b), x.double() @ wd.T + b.double())
    close(Gguf.linear(x, w), x.double() @ wd.T)


@pytest.mark.parametrize("n,k,m", [(1, 256, 1), (130, 256, 3), (64, 2816, 32), (4096, 512, 33), (200, 4096, 128), (512, 1024, 300), (300, 20480, 65)])
@pytest.mark.parametrize("t", LINEAR_TYPES)
def test_backward(t, n, k, m):
    w, wd = weight(t, n, k, seed=n + m)
    g = torch.randn(m, n, generator=torch.Generator().manual_seed(k)).cuda()
    close(Gguf.linearBackward(g, w), g.double() @ wd)


# products cut by features into several launches, each with its own tiles: 150 tiles for 9 rows (two more than a wave; the rows kernel), 86 x 2 for 200 rows,
# and the backward form, with an even and an odd first tile of features
@pytest.mark.parametrize("t,n,k,m,bwd", [("Q4_K", 19100, 8192, 9, False), ("Q6_K", 19100, 8192, 9, False), ("Q4_K", 11000, 4096, 200, False),
                                         ("Q6_K", 11000, 4096, 500, False), ("Q8_0", 4096, 11008, 128, True), ("Q4_K", 16384, 5120, 128, True)])
def test_cut_by_features(t, n, k, m, bwd):
    w, wd = weight(t, n, k, seed=m)
    g = torch.Generator().manual_seed(k)
    if bwd:
        x = torch.randn(m, n, generator=g).cuda()
        close(Gguf.linearBackward(x, w), x.double() @ wd)
    else:
        x, b = torch.randn(m, k, generator=g).cuda(), torch.randn(n, generator=g).cuda()
        close(Gguf.linear(x, w, b), x.double() @ wd.T + b.double())


# up to 16 rows (the rows kernel) the sums are taken in eight ranges of k whatever the number of thread blocks that share it: a row shard, whose k is
# split over a larger cluster, gives bitwise the outputs of the whole weight. k: fewer units than ranges, more, and not a multiple
@pytest.mark.parametrize("k", [768, 2048, 2816, 11008])
@pytest.mark.parametrize("t", LINEAR_TYPES)
def test_row_shards_are_bitwise_equal(t, k):
    n, m = 5000, 13
    raw = synth.random_valid_blocks(t, n, k, seed=k).numpy().reshape(-1)
    whole = Tensor.quantized(t, raw, n, k)
    x = torch.randn(m, k, generator=torch.Generator().manual_seed(k)).cuda()
    y = Gguf.linear(x, whole)
    for lo, hi in [(0, 100), (2048, 2560), (3000, 5000)]:
        shard = Tensor.quantized(t, raw, n, k, rows=(lo, hi))
        assert torch.equal(Gguf.linear(x, shard), y[:, lo:hi])
    wd = torch.from_numpy(oracle.dequantize(t, raw).reshape(n, k)).cuda().double()
    close(y, x.double() @ wd.T)


# 32-element formats: k that does not fill a step of 256, or not even a multiple of 4 x 32 (13 rows: the rows kernel where rows x k is large enough)
@pytest.mark.parametrize("m", [20, 13])
@pytest.mark.parametrize("k", [32, 96, 224, 288, 1056])
@pytest.mark.parametrize("t", ["Q8_0", "Q4_0", "Q4_1"])
def test_partial_steps(t, k, m):
    n = 150
    w, wd = weight(t, n, k, seed=k)
    g = torch.Generator().manual_seed(k)
    x, gy = torch.randn(m, k, generator=g).cuda(), torch.randn(m, n, generator=g).cuda()
    close(Gguf.linear(x, w), x.double() @ wd.T)
    close(Gguf.linearBackward(gy, w), gy.double() @ wd)


@pytest.mark.parametrize("m", [64, 13])
def test_wide_ranges(m):
    """Scales and mins of very different sizes within a row's block and across rows, zero and subnormal scales, x over 80 powers of two."""
    n, k = 256, 512
    for t in LINEAR_TYPES:
        block = {"Q8_0": 34, "Q4_0": 18, "Q4_1": 20, "Q4_K": 144, "Q5_K": 176, "Q6_K": 210}[t]
        fields = {"Q8_0": [0], "Q4_0": [0], "Q4_1": [0, 2], "Q4_K": [0, 2], "Q5_K": [0, 2], "Q6_K": [208]}[t]

        def edit(raw):
            blocks = raw.reshape(-1, block)
            rng = np.random.default_rng(1)
            for f in fields:
                v = (2.0 ** rng.uniform(-24, 4, len(blocks))).astype(np.float16)
                v[rng.random(len(blocks)) < 0.1] = 0
                blocks[:, f:f + 2] = v.view(np.uint8).reshape(-1, 2)

        w, wd = weight(t, n, k, 7, edit)
        x = torch.randn(m, k, generator=torch.Generator().manual_seed(3)).cuda() * (2.0 ** torch.linspace(-40, 40, m))[:, None].cuda()
        y = Gguf.linear(x, w)
        ref = x.double() @ wd.T
        # per output: relative to the sum of the magnitudes of what is added up
        assert float(((y.double() - ref).abs() / (x.double().abs() @ wd.abs().T + 1e-300)).max()) <= REL
        assert device_status(0) == 0


def test_nan_and_inf_reach_their_rows():
    w, wd = weight("Q4_K", 256, 1024, 5)
    x = torch.randn(40, 1024, generator=torch.Generator().manual_seed(3)).cuda()
    x[3, 17], x[20, 1000] = float("nan"), float("inf")
    y = Gguf.linear(x, w)
    bad = ~torch.isfinite(y)
    assert bool(bad[3].all()) and bool(bad[20].all())
    rows = [r for r in range(40) if r not in (3, 20)]
    close(y[rows], x[rows].double() @ wd.T)


# 32-element formats with a k that the decode kernels decline: up to 16 rows the choice of the kernel must not depend on the number of output rows
# either, or a shard would add up in another order than the whole weight (5000 x 1056 and 100 x 1056 lie on both sides of any line in products)
@pytest.mark.parametrize("k", [288, 1056, 2080])
@pytest.mark.parametrize("t", ["Q8_0", "Q4_0", "Q4_1"])
def test_row_shards_are_bitwise_equal_for_partial_steps(t, k):
    n = 5000
    raw = synth.random_valid_blocks(t, n, k, seed=k).numpy().reshape(-1)
    whole = Tensor.quantized(t, raw, n, k)
    shards = [(lo, hi, Tensor.quantized(t, raw, n, k, rows=(lo, hi))) for lo, hi in [(0, 100), (2048, 2560), (2500, 5000)]]
    for m in range(1, 17):
        x = torch.randn(m, k, generator=torch.Generator().manual_seed(k + m)).cuda()
        y = Gguf.linear(x, whole)
        for lo, hi, shard in shards:
            assert torch.equal(Gguf.linear(x, shard), y[:, lo:hi]), (m, lo, hi)


def test_wide_ranges_backward():
    """Features whose blocks are far smaller than their neighbours' in the same 128 rows: outputs of their own, to their own precision."""
    n, k, m = 300, 512, 40
    for t in ["Q8_0", "Q4_0", "Q4_1"]:
        block, fields = {"Q8_0": (34, [0]), "Q4_0": (18, [0]), "Q4_1": (20, [0, 2])}[t]

        def edit(raw):
            blocks = raw.reshape(n, k // 32, block)
            for f in fields:
                for b in range(k // 32):
                    blocks[:, b, f:f + 2] = np.full(n, 1.25 * 2.0 ** (3 - 3 * (b % 8)), np.float16).view(np.uint8).reshape(-1, 2)

        w, wd = weight(t, n, k, 7, edit)
        g = torch.randn(m, n, generator=torch.Generator().manual_seed(3)).cuda() * (2.0 ** torch.linspace(-40, 40, m))[:, None].cuda()
        y, ref = Gguf.linearBackward(g, w), g.double() @ wd
        # 2^-22 of each operand and what the tensor cores cut off
        assert float(((y.double() - ref).abs() / (g.double().abs() @ wd.abs() + 1e-300)).max()) <= 2e-6
        assert device_status(0) == 0


def k_scales(sc, mn):
    """The 12 bytes of a Q4_K or Q5_K block that hold eight 6-bit scales and mins (GgufKernels.java:74-83)."""
    b = [sc[j] | (sc[j + 4] >> 4) << 6 for j in range(4)] + [mn[j] | (mn[j + 4] >> 4) << 6 for j in range(4)]
    return np.array(b + [(sc[j + 4] & 15) | (mn[j + 4] & 15) << 4 for j in range(4)], np.uint8)


# mins far above the scales beside sub-blocks whose min is 0 or 1: every weight keeps its own 22 bits. All quants of a sub-block are equal and x is
# positive, so an error of a weight does not average out. ratio = dmin / d, 0: d is zero
@pytest.mark.parametrize("m", [20, 13])
@pytest.mark.parametrize("ratio", [30.0, 900.0, 1001.0, 1100.0, 20000.0, 1.0e6, 0.0])
@pytest.mark.parametrize("t", ["Q4_K", "Q5_K"])
def test_mins_far_above_the_scales(t, ratio, m):
    n, k = 64, 512
    block, quants = {"Q4_K": (144, 16), "Q5_K": (176, 16)}[t]
    d = 0.0 if ratio == 0.0 else (2.0 ** -14 if ratio > 30000 else 2.0 ** -9)
    dmin = float(np.float16(d * ratio if ratio else 0.37))
    parts = np.empty((n * k // 256, 8))  # of a sub-block's weights: d scale q + dmin min

    def edit(raw):
        rng = np.random.default_rng(int(ratio))
        for i, b in enumerate(raw.reshape(-1, block)):
            scales, mins = rng.integers(1, 64, 8), rng.integers(0, 2, 8) * (i % 3 != 0)
            if i % 3 == 2:
                mins[i % 8] = 63
            b[0:4] = np.array([d, dmin], np.float16).view(np.uint8)
            b[4:16] = k_scales([int(v) for v in scales], [int(v) for v in mins])
            b[quants:] = 0xff if i % 2 == 0 else 0x77  # Q5_K: the fifth bits too
            q = np.full(8, 15 if i % 2 == 0 else 7) + (0 if t == "Q4_K" else 16 * np.array([(b[quants] >> j) & 1 for j in range(8)]))
            parts[i] = d * scales * q + dmin * mins

    w, wd = weight(t, n, k, 3, edit)
    size = torch.from_numpy(np.repeat(parts, 32, axis=1).reshape(n, k)).cuda()
    assert bool((wd.abs() <= size * 1.0000001).all())
    x = torch.rand(m, k, generator=torch.Generator().manual_seed(9)).cuda() + 0.5
    # one sub-block at a time, so that the large ones do not hide the small ones
    for sub in range(16):
        part = torch.zeros_like(x)
        part[:, 32 * sub:32 * sub + 32] = x[:, 32 * sub:32 * sub + 32]
        y, ref = Gguf.linear(part, w).double(), part.double() @ wd.T
        # 2^-22 of the two parts of each weight, 2^-22 of x, and what the tensor cores cut off: some 2^-23 a step
        assert float(((y - ref).abs() / (part.double() @ size.T + 1e-30)).max()) <= 2e-6, (sub, ratio)
    assert device_status(0) == 0


# Q4_1: one min far above the others of the same 256, and x in one block of 32 at a time, so that the large min does not hide the others: what is the same
# for a block (8 d + min) goes as two halves under one power of two for all eight, which keep 22 bits of each down to 2^-17 of the largest
@pytest.mark.parametrize("m", [20, 13])
@pytest.mark.parametrize("ratio", [30.0, 1000.0, 30000.0])
def test_one_min_far_above_the_others(ratio, m):
    n, k = 64, 512
    parts = np.empty((n, k // 32))  # of a block's weights: d q + min

    def edit(raw):
        rng = np.random.default_rng(int(ratio))
        for row, blocks in enumerate(raw.reshape(n, k // 32, 20)):
            mins = rng.uniform(0.5, 1.0, k // 32) * 2.0 ** -9
            mins[row % 8::8] *= ratio
            mins = mins.astype(np.float16)
            blocks[:, 0:2] = np.full(k // 32, 2.0 ** -9, np.float16).view(np.uint8).reshape(-1, 2)
            blocks[:, 2:4] = mins.view(np.uint8).reshape(-1, 2)
            blocks[:, 4:] = 0xff if row % 2 == 0 else 0x77
            parts[row] = 2.0 ** -9 * (15 if row % 2 == 0 else 7) + mins.astype(np.float64)

    w, wd = weight("Q4_1", n, k, 3, edit)
    assert bool((wd == torch.from_numpy(np.repeat(parts, 32, axis=1)).cuda()).all())  # all weights of a block are the same
    x = torch.rand(m, k, generator=torch.Generator().manual_seed(9)).cuda() + 0.5
    for block in range(k // 32):
        part = torch.zeros_like(x)
        part[:, 32 * block:32 * block + 32] = x[:, 32 * block:32 * block + 32]
        y, ref = Gguf.linear(part, w).double(), part.double() @ wd.T
        # as above: 2^-22 of the two parts of each weight, 2^-22 of x, and what the tensor cores cut off
        assert float(((y - ref).abs() / ref).max()) <= 2e-6, (block, ratio)
    assert device_status(0) == 0


# What the decode kernels and plain FP32 sums of the same products keep: 3.2e-7 of the result's norm (measured: the decode GEMVs 2.8 to 3.2e-7 for
# every format, FP32 fused multiply-adds on CUDA cores 1.8 to 2.4e-7). The tensor cores cut sums off towards zero, a bias that grows with the
# number of MMAs that go into one accumulator.
@pytest.mark.parametrize("t", LINEAR_TYPES)
def test_error_is_no_larger_than_the_decode_kernels(t):
    n, k = 1024, 4096
    g = torch.Generator(device="cuda").manual_seed(5)
    wf = torch.randn(n, k, generator=g, device="cuda") * 0.02
    raw = (Quant.quantizeQ8Blocks(wf) if t == "Q8_0" else synth.QUANTIZERS[t](wf)).cpu().numpy().reshape(-1)
    w = Tensor.quantized(t, raw, n, k)
    wd = torch.from_numpy(oracle.dequantize(t, raw).reshape(n, k)).cuda().double()
    worst = {}
    for m in (5, 9, 16, 20, 33, 64, 100, 128, 200):
        x, gy = torch.randn(m, k, generator=g, device="cuda"), torch.randn(m, n, generator=g, device="cuda")
        for name, y, ref in (("forward", Gguf.linear(x, w), x.double() @ wd.T), ("backward", Gguf.linearBackward(gy, w), gy.double() @ wd)):
            worst[name, m] = float((y.double() - ref).norm() / ref.norm())
    assert max(v for (name, _), v in worst.items() if name == "forward") <= 3.2e-7, worst
    assert max(v for (name, _), v in worst.items() if name == "backward") <= 1.8e-7, worst


# Many units through the ring of raw blocks, back to back: a unit that is copied over while a warp still reads it shows as weights of another unit
# (so did the backward form of every format but Q4_K and Q4_1, and the bfloat16 one of Q8_0, in up to nine calls of ten).
@pytest.mark.parametrize("t,n,k,m,kind", [("Q4_0", 11008, 4096, 128, "backward"), ("Q8_0", 11008, 4096, 128, "backward"), ("Q5_K", 11008, 4096, 128, "backward"),
                                          ("Q6_K", 11008, 4096, 128, "backward"), ("Q4_1", 11008, 4096, 100, "backward"), ("Q4_K", 11008, 4096, 128, "backward"),
                                          ("Q8_0", 4096, 4096, 512, "bf16"), ("Q6_K", 4096, 4096, 512, "bf16"), ("Q4_K", 11008, 4096, 200, "forward"),
                                          ("Q8_0", 11008, 4096, 16, "forward"), ("Q4_0", 11008, 4096, 24, "forward"), ("Q5_K", 11008, 4096, 32, "forward"),
                                          ("Q6_K", 11008, 4096, 100, "forward"), ("Q8_0", 11008, 4096, 200, "forward"), ("Q4_1", 11008, 4096, 300, "forward"),
                                          ("Q4_K", 4096, 11008, 100, "bf16"), ("Q5_K", 11008, 4096, 300, "bf16")])
def test_repeated_calls_give_the_same_bits(t, n, k, m, kind):
    w, _ = weight(t, n, k, seed=2)
    x = torch.randn(m, n if kind == "backward" else k, generator=torch.Generator().manual_seed(4)).cuda()
    call = {"backward": lambda: Gguf.linearBackward(x, w), "forward": lambda: Gguf.linear(x, w), "bf16": lambda: Gguf.linearBf16(x.to(torch.bfloat16), w)}[kind]
    call()
    torch.cuda.synchronize()
    alone = call()  # with nothing before or behind it
    torch.cuda.synchronize()
    for _ in range(5):
        ys = [call() for _ in range(20)]
        assert all(torch.equal(y, alone) for y in ys)
    assert device_status(0) == 0
