"""The decode GEMVs of Q6_K and the 32-element formats at the lines between building x's image themselves and reading that of an image kernel.

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
    """Zeros, subnormals, large floats, ties of the fixed point, NaN and Inf, in x that the kernel in front of the call writes."""
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


# the first and the last number of rows of W with which the rule looks at more than the values of x, and those beside them
@pytest.mark.parametrize("n", [512, 513, 2368, 2369])
@pytest.mark.parametrize("k,m", [(6144, 1), (3072, 2), (6400, 1), (3328, 2), (8192, 1), (4096, 2)])
@pytest.mark.parametrize("t", ["Q6_K", "Q8_0", "Q4_1"])
def test_the_image_kernel_between_few_and_many_rows(t, k, m, n):
    """Which of the two routes a launched and a captured call take, and that all give the same bits."""
    L = jitnn_b200.load()
    raw = synth.random_valid_blocks(t, n, k, seed=k + n).numpy().reshape(-1)
    w, wd = Tensor.quantized(t, raw, n, k), torch.from_numpy(oracle.dequantize(t, raw).reshape(n, k)).cuda().double()
    x = torch.randn(m, k, generator=torch.Generator().manual_seed(m)).cuda()
    between = m * k > 6144 and 512 < n <= 2368
    stream = torch.cuda.Stream()
    counts = []
    with torch.cuda.stream(stream):
        stream.wait_stream(torch.cuda.default_stream())
        before = L.jq_launch_count()
        y = Gguf.linear(x, w)
        counts.append(L.jq_launch_count() - before)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        before = L.jq_launch_count()
        z = Gguf.linear(x, w)
        counts.append(L.jq_launch_count() - before)
    graph.replay()
    torch.cuda.synchronize()
    assert counts == [2 if between and m == 1 and t == "Q4_1" else 1, 2 if between and (m == 2 or t != "Q6_K") else 1]
    assert torch.equal(y, z) and np.array_equal(Gguf.linear(x.cpu().numpy(), w), y.cpu().numpy())
    ref, size = x.double() @ wd.T, ((x.double() ** 2) @ (wd ** 2).T).sqrt()
    assert float(((y.double() - ref).abs() / size).max()) <= REL


@pytest.mark.parametrize("m", [1, 2, 3, 8, 16, 20])
@pytest.mark.parametrize("t", ["Q4_K", "Q5_K", "Q6_K", "Q8_0", "Q4_0", "Q4_1"])
def test_in_place(t, m):
    """y on x with n = k: no thread block still reads x when another stores y. Products on a second stream let the call's thread blocks start one after the other."""
    n = {1: 8192, 2: 4096}.get(m, 2048)  # (8192 values of x, which would become digits inside the GEMV)
    w = Tensor.quantized(t, synth.random_valid_blocks(t, n, n, seed=m).numpy().reshape(-1), n, n)
    L, x = jitnn_b200.load(), torch.randn(m, n, generator=torch.Generator().manual_seed(m)).cuda()
    want, other, side = Gguf.linear(x, w), torch.randn(2048, 2048, device="cuda"), torch.cuda.Stream()
    zs = [x.clone() for _ in range(50)]
    torch.cuda.synchronize()
    for z in zs:
        with torch.cuda.stream(side):
            torch.mm(other, other)
        assert L.jq_linear_f32(w._handle(), z.data_ptr(), m, None, z.data_ptr(), 1, torch.cuda.current_stream().cuda_stream) == 0
    assert all(torch.equal(z, want) for z in zs)


@pytest.mark.parametrize("m", [1, 2])
@pytest.mark.parametrize("t", ["Q4_K", "Q5_K", "Q6_K", "Q8_0", "Q4_0", "Q4_1"])
def test_x_up_to_the_largest_float(t, m):
    """Magnitudes from 2^127 to the largest float, with weights small enough for a finite result; made inside the GEMV, and by the image kernel (host arrays)."""
    n, k = 64, 1024
    raw = synth.random_valid_blocks(t, n, k, seed=2).numpy().reshape(-1).copy()
    size, at = {"Q4_K": (144, [0, 2]), "Q5_K": (176, [0, 2]), "Q6_K": (210, [208]), "Q8_0": (34, [0]), "Q4_0": (18, [0]), "Q4_1": (20, [0, 2])}[t]
    for a in at:
        raw.reshape(-1, size)[:, a:a + 2] = np.array([2.0 ** -22], np.float16).view(np.uint8)
    w, wd = Tensor.quantized(t, raw, n, k), torch.from_numpy(oracle.dequantize(t, raw).reshape(n, k)).cuda().double()
    g = torch.Generator().manual_seed(m)
    x = (torch.rand(m, k, generator=g) + 1.0) * 2.0 ** 127 * (torch.randint(0, 2, (m, k), generator=g) * 2 - 1)
    x[0, 5] = torch.finfo(torch.float32).max
    x = x.clamp(-torch.finfo(torch.float32).max, torch.finfo(torch.float32).max).cuda()
    ref, of = x.double() @ wd.T, ((x.double() ** 2) @ (wd ** 2).T).sqrt()
    for y in (Gguf.linear(x, w), torch.from_numpy(Gguf.linear(x.cpu().numpy(), w)).cuda()):
        assert float(((y.double() - ref).abs() / of).max()) <= REL
