"""The Q8_0 quantiser around a thread block's 64 blocks and a thread's eight, where one thread makes a block's scale for its neighbours; NaN and Inf stay in their block."""
import numpy as np
import pytest
import torch

from jitnn_b200 import Quant
from oracle import oracle
from test_gpu_block_kernels import test_quantize_rounding_boundaries as check_boundaries

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks", [3, 7, 8, 9, 63, 64, 65, 4097])
@pytest.mark.parametrize("aligned", [True, False])
def test_ends_of_thread_blocks(blocks, aligned):
    check_boundaries(blocks, aligned)


def test_a_bad_block_leaves_its_neighbours_alone():
    x = np.random.default_rng(1).standard_normal((130, 32)).astype(np.float32)
    want = oracle.quantize_q8_0(x).reshape(130, 34)
    x[5, 3], x[77, 31] = np.nan, np.inf
    got = Quant.quantizeQ8Blocks(torch.from_numpy(x).cuda()).cpu().numpy().reshape(130, 34)
    rows = [r for r in range(130) if r not in (5, 77)]
    assert np.array_equal(got[rows], want[rows])
