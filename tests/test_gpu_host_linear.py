"""Host arrays of the linear below, at and above the size that goes through page-locked staging memory (512 KB for x, bias and y)."""
import threading

import numpy as np
import pytest
import torch

from conftest import LINEAR_TYPES, close_like_reference
from jitnn_b200 import Gguf, Tensor, synth
from oracle import oracle

pytestmark = pytest.mark.gpu


# staged; a row longer than y may be staged (16 KB) but x may; x, bias and y just under and just over 512 KB; a k the decode kernels do not
# take (not a multiple of 256)
@pytest.mark.parametrize("n,k,m", [(1, 256, 1), (300, 512, 2), (5000, 256, 1), (64, 8192, 15), (64, 8192, 16), (64, 8192, 17), (96, 96, 3)])
@pytest.mark.parametrize("t", LINEAR_TYPES)
def test_sizes(t, n, k, m):
    if k % oracle.block_values(t) != 0:
        pytest.skip("k is not a whole number of blocks")
    raw = synth.random_valid_blocks(t, n, k, seed=n + k).numpy().reshape(-1)
    w = Tensor.quantized(t, raw, n, k)
    rng = np.random.default_rng(m)
    x, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    for bias in (None, b):
        close_like_reference(oracle.linear(t, raw, x, bias, n=n), Gguf.linear(x, w, bias), "%s %dx%d m=%d" % (t, n, k, m))


def test_a_thread_gives_back_what_it_held():
    """Staging memory, page-locked memory and stream of a thread that has made host calls."""
    n, k, m = 1024, 4096, 512  # 10 MB of staging
    w = Tensor.quantized("Q4_0", synth.random_valid_blocks("Q4_0", n, k, seed=1).numpy().reshape(-1), n, k)
    x = np.zeros((m, k), np.float32)

    def work():
        Gguf.linear(x, w)
        Gguf.linear(x[:1], w)

    def threads(count):
        for _ in range(count):
            t = threading.Thread(target=work)
            t.start()
            t.join()
        return torch.cuda.mem_get_info()[0]

    before = threads(2)
    assert before - threads(20) < 64 << 20
