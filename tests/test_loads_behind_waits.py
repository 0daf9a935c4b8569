"""What a kernel behind a programmatic launch declares as read-only (no GPU).

Loads from `const __restrict__` memory and through __ldg depend on nothing that the wait for the kernel in front says it touches, and may be moved in front of it. So a kernel
that waits declares only what no kernel in front of it on its stream writes: weights, tables, a decoder's position. Images are read by asynchronous copies (asm volatile), which stay where they are.
"""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "jitnn_b200", "csrc")
NOT_WRITTEN_IN_FRONT = {"table", "w", "cos_t", "sin_t", "pos0", "peerp"}
READ_BY_ASYNCHRONOUS_COPIES = {"image"}
# __ldg of: the weights' formats; norm weights; cached keys of earlier positions, in front of the wait
LDG_IN = {"jq_formats.cuh": None, "jq_dequant.cu": None, "jq_gemv.cu": None, "jq_decoder.cu": 2}


def kernels(text):
    for m in re.finditer(r"__global__ void", text):
        head = text[m.end():text.index("{", m.end())]
        depth, at = 0, m.end() + len(head)
        while True:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
            if depth == 0:
                break
        yield head, text[m.end() + len(head):at]


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))), ids=os.path.basename)
def test_read_only_parameters(path):
    with open(path) as f:
        text = f.read()
    for head, body in kernels(text):
        if "griddepcontrol.wait" in body or "pdl_enter()" in body:
            names = set(re.findall(r"const [\w:]+\* __restrict__ (\w+)", head))
            assert names <= NOT_WRITTEN_IN_FRONT | READ_BY_ASYNCHRONOUS_COPIES, head
            for name in names & READ_BY_ASYNCHRONOUS_COPIES:
                assert not re.search(r"\*\s*%s\b|\b%s\[" % (name, name), body), head
    name, count = os.path.basename(path), len(re.findall(r"__ldg\(", text))
    assert count == 0 or (name in LDG_IN and LDG_IN[name] in (None, count)), count
