"""The captured decode steps where one range of cached positions ends and the next begins, and the page-locked logits arrays."""
import numpy as np
import pytest
import torch

import jitnn_b200
from jitnn_b200 import LlamaDecoder, synth
from oracle import llama_oracle

pytestmark = pytest.mark.gpu


def build(heads, kv_heads, head_dim, max_seq, seed=5):
    dim = heads * head_dim
    cfg = llama_oracle.Config(layers=2, dim=dim, heads=heads, kv_heads=kv_heads, hidden=2 * dim, vocab=8192, max_seq=max_seq)
    dec = LlamaDecoder(cfg.layers, cfg.dim, cfg.heads, cfg.kv_heads, cfg.hidden, cfg.vocab, cfg.max_seq, cfg.eps, cfg.rope_base)
    dec.load(llama_oracle.random_model(cfg, seed))
    return dec


# a graph covers up to 256, 512, ... positions; one, two, four and eight query heads per key/value head; both head sizes; one row and several
@pytest.mark.parametrize("heads,kv_heads,head_dim,n_seqs", [(2, 2, 128, 1), (4, 2, 128, 1), (4, 2, 128, 3), (4, 1, 64, 2), (8, 1, 128, 2)])
def test_captured_steps_across_ranges(heads, kv_heads, head_dim, n_seqs):
    toks = np.random.default_rng(1).integers(0, 8192, (516, n_seqs)).astype(np.int32)
    out = []
    for graph in (0, 1):
        jitnn_b200.load().jq_set_option(b"decoder_graph", graph)
        try:
            dec = build(heads, kv_heads, head_dim, 516)
            if n_seqs > 1:
                dec.set_sequences(n_seqs)
            got = []
            for pos in range(516):
                lg, nxt = dec.forward(toks[pos], pos) if n_seqs == 1 else dec.forward_batch(toks[pos], pos)
                if pos in (0, 63, 64, 254, 255, 256, 257, 511, 512, 515):
                    got.append(np.array(lg))
                    assert np.array_equal(nxt, np.argmax(lg, axis=1))
            out.append(got)
            dec.close()
        finally:
            jitnn_b200.load().jq_set_option(b"decoder_graph", 1)
    # The two forms cut the keys into chunks alike but launch a different number of them; merging an empty chunk multiplies by one and adds
    # zero, so only FP32 rounding in the merge may differ: 2e-4 of the largest logit is the decoder's own bar.
    for a, b in zip(*out):
        assert np.abs(a - b).max() <= 2e-4 * np.abs(a).max()


def test_logits_arrays_stay_valid():
    """More arrays held than page-locked blocks exist; each keeps its step's values, also after the decoder is closed."""
    dec = build(4, 2, 64, 32)
    held, copies = [], []
    for pos in range(9):
        lg, _ = dec.forward([pos + 1], pos)
        held.append(lg)
        copies.append(lg.copy())
    del held[2], copies[2]  # its block is free for the next step
    lg, _ = dec.forward([3], 9)
    held.append(lg)
    copies.append(lg.copy())
    dec.close()
    for a, b in zip(held, copies):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n_seqs", [1, 2])
def test_the_next_range_is_captured_before_it_is_reached(n_seqs):
    """A step past the end of a range finds its graph there: capturing counts the step's launches, replaying does not."""
    dec = build(4, 2, 128, 520)
    if n_seqs > 1:
        dec.set_sequences(n_seqs)
    L = jitnn_b200.load()
    toks = np.zeros(n_seqs, np.int32)
    counts = [L.jq_launch_count()]
    for pos in range(236, 520):
        dec.forward(toks, pos) if n_seqs == 1 else dec.forward_batch(toks, pos)
        counts.append(L.jq_launch_count())
    per_step = np.diff(counts)
    assert per_step[256 - 236] == 0 and per_step[512 - 236] == 0
    assert (per_step > 0).sum() == 2 + 2  # the first step is issued kernel by kernel; one capture each for up to 256, 512 and 520 positions
    dec.close()


# where the norm in front of gate and up stops being made inside their launch: by width, and at 8192 by the rows of both
@pytest.mark.parametrize("dim,hidden", [(7168, 12544), (7424, 9984), (8192, 9984), (8192, 10240)])
def test_norms_inside_and_in_front(dim, hidden):
    """The fused single-token step against the general kernels."""
    heads, vocab = dim // 128, 512
    g = torch.Generator(device="cuda").manual_seed(hidden)

    def lin(n, k):
        return ("Q4_K", synth.quantize_q4_k(torch.randn(n, k, generator=g, device="cuda") * 0.02).cpu().numpy().reshape(-1), n, k)

    w = {"tok_embeddings": torch.randn(vocab, dim, generator=g, device="cuda").cpu().numpy(), "norm": np.ones(dim, np.float32), "output": lin(vocab, dim)}
    for layer in range(2):
        p = "layers.%d." % layer
        w[p + "attention_norm"] = (1.0 + 0.1 * torch.randn(dim, generator=g, device="cuda")).cpu().numpy()
        w[p + "ffn_norm"] = (1.0 + 0.1 * torch.randn(dim, generator=g, device="cuda")).cpu().numpy()
        w.update({p + "wq": lin(dim, dim), p + "wk": lin(128, dim), p + "wv": lin(128, dim), p + "wo": lin(dim, dim), p + "w1": lin(hidden, dim),
                  p + "w3": lin(hidden, dim), p + "w2": lin(dim, hidden)})
    dec = LlamaDecoder(2, dim, heads, 1, hidden, vocab, 8)
    dec.load(w)
    out = []
    for fused in (0, 1):
        jitnn_b200.load().jq_set_option(b"decoder_fused", fused)
        try:
            out.append([np.array(dec.forward([7 * pos + 1], pos)[0]) for pos in range(3)])
        finally:
            jitnn_b200.load().jq_set_option(b"decoder_fused", 1)
    for a, b in zip(*out):
        assert np.abs(a - b).max() <= 1e-5 * np.abs(a).max()  # FP32 throughout, sums in other orders
    dec.close()


# a Q6_K wv beside Q4_K wq and wk, which makes the norm itself: 20 super-blocks (no multiple of its eight warps), the first width with two ring stages in place
# of three (26 super-blocks), the widest
@pytest.mark.parametrize("dim,heads,hidden", [(5120, 40, 2048), (6656, 52, 2048), (8192, 64, 1024)])
def test_a_q6k_wv_makes_its_own_norm(dim, heads, hidden):
    """The fused single-token step against the general kernels; a layer with a Q6_K wv takes one launch more than one whose weights are all Q4_K."""
    vocab, L = 512, jitnn_b200.load()
    g = torch.Generator(device="cuda").manual_seed(dim)
    launches = []
    for fine in ("Q4_K", "Q6_K"):
        def lin(n, k, t="Q4_K"):
            return (t, synth.QUANTIZERS[t](torch.randn(n, k, generator=g, device="cuda") * 0.02).cpu().numpy().reshape(-1), n, k)

        w = {"tok_embeddings": torch.randn(vocab, dim, generator=g, device="cuda").cpu().numpy(), "norm": np.ones(dim, np.float32), "output": lin(vocab, dim)}
        for layer in range(2):
            p = "layers.%d." % layer
            w[p + "attention_norm"] = (1.0 + 0.1 * torch.randn(dim, generator=g, device="cuda")).cpu().numpy()
            w[p + "ffn_norm"] = (1.0 + 0.1 * torch.randn(dim, generator=g, device="cuda")).cpu().numpy()
            w.update({p + "wq": lin(dim, dim), p + "wk": lin(256, dim), p + "wv": lin(256, dim, fine), p + "wo": lin(dim, dim), p + "w1": lin(hidden, dim),
                      p + "w3": lin(hidden, dim), p + "w2": lin(dim, hidden)})
        dec = LlamaDecoder(2, dim, heads, 2, hidden, vocab, 8)
        dec.load(w)
        before = L.jq_launch_count()
        fused = [np.array(dec.forward([1], 0)[0])]  # (the first step is issued kernel by kernel)
        launches.append(L.jq_launch_count() - before)
        fused += [np.array(dec.forward([7 * pos + 1], pos)[0]) for pos in (1, 2)]
        L.jq_set_option(b"decoder_fused", 0)
        try:
            general = [np.array(dec.forward([7 * pos + 1], pos)[0]) for pos in range(3)]
        finally:
            L.jq_set_option(b"decoder_fused", 1)
        for a, b in zip(general, fused):
            assert np.abs(a - b).max() <= 1e-5 * np.abs(a).max()  # FP32 throughout, sums in other orders
        dec.close()
    assert launches[1] - launches[0] == 2


# an odd number of super-blocks: the last width whose norm one thread block makes, and the first that is too wide for it and goes to the general kernels
@pytest.mark.parametrize("heads", [30, 42])
def test_widths_of_an_odd_number_of_super_blocks(heads):
    cfg = llama_oracle.Config(layers=1, dim=128 * heads, heads=heads, kv_heads=2, hidden=1024, vocab=512, max_seq=8)
    dec = LlamaDecoder(cfg.layers, cfg.dim, cfg.heads, cfg.kv_heads, cfg.hidden, cfg.vocab, cfg.max_seq, cfg.eps, cfg.rope_base)
    weights = llama_oracle.random_model(cfg, 3)
    dec.load(weights)
    ref = llama_oracle.Decoder(cfg, weights)
    for pos in range(3):
        want = ref.forward(7 * pos + 1, pos)
        assert np.abs(dec.forward([7 * pos + 1], pos)[0][0] - want).max() <= 2e-4 * np.abs(want).max()
    dec.close()
