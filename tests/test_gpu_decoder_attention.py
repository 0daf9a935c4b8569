"""The general path's attention, rotations, cache and images for the rows kernel: runs of consecutive tokens, which share thread blocks, and batches, against the same
tokens one at a time, where chunks of 64 keys, groups of heads and numbers of rows begin and end.

Both are FP32 throughout and take sums in other orders: 2e-5 of the largest logit (1e-6 and less is seen) leaves room for the layers between.
"""
import numpy as np
import pytest
import torch

import jitnn_b200
from jitnn_b200 import LlamaDecoder, Quant, synth

pytestmark = pytest.mark.gpu

REL = 2e-5
VOCAB = 512


def build(head, heads, kv_heads, fmt, hidden=512, bad_token=None):
    dim = head * heads
    g = torch.Generator(device="cuda").manual_seed(head + heads)

    def lin(n, k, t=fmt):
        w = torch.randn(n, k, generator=g, device="cuda") * 0.05
        return (t, (Quant.quantizeQ8Blocks(w) if t == "Q8_0" else synth.QUANTIZERS[t](w)).cpu().numpy().reshape(-1), n, k)

    kv = head * kv_heads
    w = {"tok_embeddings": torch.randn(VOCAB, dim, generator=g, device="cuda").cpu().numpy(), "norm": np.ones(dim, np.float32), "output": lin(VOCAB, dim)}
    if bad_token is not None:
        w["tok_embeddings"][bad_token] = np.nan
    for layer in range(2):
        p = "layers.%d." % layer
        w[p + "attention_norm"] = (1.0 + 0.1 * torch.randn(dim, generator=g, device="cuda")).cpu().numpy()
        w[p + "ffn_norm"] = (1.0 + 0.1 * torch.randn(dim, generator=g, device="cuda")).cpu().numpy()
        w.update({p + "wq": lin(dim, dim), p + "wk": lin(kv, dim), p + "wv": lin(kv, dim, "Q6_K" if fmt == "Q4_K" else fmt), p + "wo": lin(dim, dim),
                  p + "w1": lin(hidden, dim), p + "w3": lin(hidden, dim), p + "w2": lin(dim, hidden)})
    dec = LlamaDecoder(2, dim, heads, kv_heads, hidden, VOCAB, 320)
    dec.load(w)
    return dec


@pytest.fixture(autouse=True)
def general_kernels():
    jitnn_b200.load().jq_set_option(b"decoder_fused", 0)
    yield
    jitnn_b200.load().jq_set_option(b"decoder_fused", 1)


# heads of 16 (a merge takes fewer than 256 values), 64 and 128, and 96 (other kernels, heads across the merge's 256 values); groups of 1, 2, 8 and 12 heads
@pytest.mark.parametrize("head,heads,kv_heads", [(64, 4, 4), (64, 16, 2), (128, 2, 1), (128, 12, 1), (96, 8, 4), (16, 16, 16)])
@pytest.mark.parametrize("fmt", ["Q4_K", "Q8_0"])
def test_runs_of_tokens(head, heads, kv_heads, fmt):
    dec = build(head, heads, kv_heads, fmt)
    toks = np.random.default_rng(1).integers(0, VOCAB, 160).astype(np.int32)
    alone = np.stack([np.array(dec.forward(toks[i:i + 1], i)[0][0]) for i in range(160)])
    scale = np.abs(alone).max()
    for start in (0, 55, 63, 64, 121):  # in front of, across and behind the ends of chunks
        for n in (2, 3, 5, 8, 9, 16):
            got = dec.forward(toks[start:start + n], start)[0]
            assert np.abs(got - alone[start:start + n]).max() <= REL * scale, (start, n)
    after = np.array(dec.forward(toks[137:138], 137)[0][0])
    assert np.abs(after - alone[137]).max() <= REL * scale
    dec.close()


@pytest.mark.parametrize("head,heads,kv_heads", [(64, 4, 4), (128, 8, 1), (128, 2, 2)])
@pytest.mark.parametrize("fmt,n", [("Q4_K", 3), ("Q4_K", 11), ("Q8_0", 3), ("Q8_0", 16)])
def test_batches(head, heads, kv_heads, fmt, n):
    dec = build(head, heads, kv_heads, fmt)
    dec.set_sequences(n)
    toks = np.random.default_rng(2).integers(0, VOCAB, (n, 70)).astype(np.int32)
    for s in range(n):
        for at in range(0, 62, 16):
            dec.enqueue(toks[s, at:min(at + 16, 62)], at, seq=s)
    got = [np.array(dec.forward_batch(toks[:, p], p)[0]) for p in range(62, 67)]  # (kernel by kernel, captured, replayed)
    for s in range(n):
        for i, p in enumerate(range(62, 67)):
            alone = np.array(dec.forward(toks[s, p:p + 1], p, seq=s)[0][0])
            assert np.abs(got[i][s] - alone).max() <= REL * np.abs(alone).max(), (s, p)
    dec.close()


@pytest.mark.parametrize("head,heads,kv_heads", [(64, 4, 2), (128, 2, 1)])
def test_a_later_token_reaches_nobody_in_front_of_it(head, heads, kv_heads):
    """The last token of a run is all NaN: the tokens in front of it share its thread block and give the bits that they give without it."""
    dec = build(head, heads, kv_heads, "Q8_0", bad_token=7)
    toks = np.random.default_rng(3).integers(8, VOCAB, 80).astype(np.int32)
    dec.enqueue(toks[:16], 0)
    dec.enqueue(toks[16:32], 16)
    want = np.array(dec.forward(toks[32:45], 32)[0])
    bad = toks[32:45].copy()
    bad[12] = 7
    got = np.array(dec.forward(bad, 32)[0])
    assert np.array_equal(got[:12], want[:12]) and np.isfinite(want).all() and not np.isfinite(got[12]).any()
    dec.close()
