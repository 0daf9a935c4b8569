"""How the rows kernel's tiles go into launches (jitnn_b200/csrc/jq_rows_cut.cuh), without a GPU but for the last test: the shapes of its GPU tests reach
every kind of plan."""
import ctypes
import os
import shutil
import subprocess

import pytest
import torch

import jitnn_b200
from conftest import LINEAR_TYPES, ROOT
from jitnn_b200 import Gguf, Tensor, synth
from oracle.oracle import TYPES
from test_gpu_rows import SHAPES, THREE_LAUNCHES, TWO_LAUNCHES

CALL = """
#include "jq_rows_cut.cuh"
extern "C" int plan(int type, int tiles, int units, int* out) {
    jq::rows::Parts p;
    jq::rows::cut(tiles, units, jq::rows::unit_ns(type), jq::rows::MAX_PARTS, p);
    for (int i = 0; i < p.count; i++) {
        out[2 * i] = p.tiles[i];
        out[2 * i + 1] = p.ksplit[i];
    }
    return p.count;
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    compiler = shutil.which("g++") or pytest.skip("no C++ compiler")
    at = tmp_path_factory.mktemp("plan")
    (at / "plan.cpp").write_text(CALL)
    subprocess.run([compiler, "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "jitnn_b200", "csrc"), str(at / "plan.cpp"), "-o", str(at / "plan.so")], check=True)
    lib = ctypes.CDLL(str(at / "plan.so"))

    def launches(t, n, k):
        out = (ctypes.c_int * 6)()
        count = lib.plan(TYPES[t], (n + 127) // 128, (k + 255) // 256, out)
        return [(out[2 * i], out[2 * i + 1]) for i in range(count)]

    return launches


# (tiles, thread blocks that share k) of each launch; Q4_K's where its units, the fastest, make another choice
PLANS = {
    (1, 256): [(1, 1)], (129, 512): [(2, 1)], (128, 2816): [(1, 4)], (4096, 4096): [(32, 4)], (1024, 8192): [(8, 8)], (2000, 16384): [(16, 4)],
    (19000, 2048): [(148, 1), (1, 4)], (30000, 1024): [(235, 1)], (6400, 4096): [(50, 2)], (18950, 2560): [(148, 1), (1, 4)],
    (23200, 3584): [(148, 1), (34, 2)], (9500, 8192): [(74, 2), (1, 8)], (4300, 14080): [(33, 4), (1, 8)], (28500, 11264): [(148, 1), (74, 2), (1, 8)],
}
PLANS_Q4_K = {(19000, 2048): [(149, 1)], (4300, 14080): [(34, 2)]}


@pytest.mark.parametrize("t", LINEAR_TYPES)
def test_launches_of_the_tested_shapes(plan, t):
    for n, k in [s[:2] for s in SHAPES] + [TWO_LAUNCHES, THREE_LAUNCHES]:
        want = PLANS_Q4_K.get((n, k), PLANS[n, k]) if t == "Q4_K" else PLANS[n, k]
        assert plan(t, n, k) == want, (n, k)


@pytest.mark.parametrize("t", LINEAR_TYPES)
def test_launches_hold_every_tile_once_and_fit_the_chip(plan, t):
    for n in (1, 128, 129, 4096, 9472, 9473, 18944, 18945, 28673, 40000, 128256, 300000):
        for k in (32, 256, 288, 1024, 4096, 8192, 28672):
            parts = plan(t, n, k)
            assert 1 <= len(parts) <= 3 and sum(tiles for tiles, _ in parts) == (n + 127) // 128
            for tiles, ks in parts:
                assert tiles > 0 and (ks == 1 or (ks in (2, 4, 8) and tiles * ks <= 148 and (k + 255) // 256 >= 2 * ks))


@pytest.mark.gpu
@pytest.mark.parametrize("t", LINEAR_TYPES)
def test_the_tested_shapes_are_the_rows_kernels(t):
    """x's image and the launches of the plan: no shape goes to the decode kernels instead (32-element formats, Q6_K: from 5 rows on, Q4_K and Q5_K: from 9)."""
    L = jitnn_b200.load()
    for n, k, m in SHAPES:
        raw = synth.random_valid_blocks(t, n, k, seed=1).numpy().reshape(-1)
        w, x = Tensor.quantized(t, raw, n, k), torch.zeros(m, k, device="cuda")
        before = L.jq_launch_count()
        Gguf.linear(x, w)
        want = PLANS_Q4_K.get((n, k), PLANS[n, k]) if t == "Q4_K" else PLANS[n, k]
        assert L.jq_launch_count() - before == 1 + len(want), (n, k, m)
        w.release()
