"""The prompt path's tensor-core attention where its tiles of 64 queries and 64 keys end, against the FP32 decode path on the same weights.

The attention itself keeps FP32 precision; the linears around it round their inputs to bfloat16, so the bar is the prompt path's own: 1e-2
of the largest logit (tests/test_gpu_decoder_prompt.py).
"""
import numpy as np
import pytest
import torch

from jitnn_b200 import LlamaDecoder
from oracle import llama_oracle

pytestmark = pytest.mark.gpu

TOL = 1e-2


# head sizes 128 and 64; one, two and four query heads per key/value head
@pytest.mark.parametrize("dim,heads,kv_heads", [(512, 4, 4), (512, 4, 2), (256, 4, 1)])
# one query; a tile and one either side; two tiles and a bit. Positions before the run: none, one, a tile less and more one, several tiles
@pytest.mark.parametrize("tokens,pos0", [(1, 0), (1, 64), (63, 1), (64, 0), (64, 64), (65, 63), (129, 65), (140, 200)])
def test_tile_edges(dim, heads, kv_heads, tokens, pos0):
    cfg = llama_oracle.Config(layers=2, dim=dim, heads=heads, kv_heads=kv_heads, hidden=2 * dim, vocab=300, max_seq=pos0 + tokens + 2)
    dec = LlamaDecoder(cfg.layers, cfg.dim, cfg.heads, cfg.kv_heads, cfg.hidden, cfg.vocab, cfg.max_seq, cfg.eps, cfg.rope_base)
    dec.load(llama_oracle.random_model(cfg, tokens + pos0))
    toks = np.random.default_rng(tokens).integers(0, cfg.vocab, pos0 + tokens + 1).astype(np.int32)

    def feed(lo, hi):
        for at in range(lo, hi, 16):
            out = dec.forward(toks[at:min(at + 16, hi)], at)[0]
        return out[-1]

    want = feed(0, pos0 + tokens)
    want_next = feed(pos0 + tokens, pos0 + tokens + 1)
    if pos0 > 0:
        feed(0, pos0)
    got, _ = dec.prompt(toks[pos0:pos0 + tokens], pos0)
    assert np.abs(got - want).max() <= TOL * np.abs(want).max()
    # the keys and values it left in the cache
    got_next = feed(pos0 + tokens, pos0 + tokens + 1)
    assert np.abs(got_next - want_next).max() <= TOL * np.abs(want_next).max()
    dec.close()


def q8_weight(values):
    """Integers -127 .. 127 times 2^-7 as a Q8_0 weight: exact in bfloat16 (up to 8 bits each), so linears on bfloat16 numbers add up exactly."""
    n, k = values.shape
    raw = np.zeros((n, k // 32, 34), np.uint8)
    raw[:, :, :2] = np.full(1, 2.0 ** -7, np.float16).view(np.uint8)
    raw[:, :, 2:] = values.astype(np.int8).view(np.uint8).reshape(n, k // 32, 32)
    return ("Q8_0", raw.reshape(-1), n, k)


def attention_model(heads, kv_heads, hd, seed):
    """One layer whose residual stream after the attention block is embedding + bfloat16(attention), read through an identity output projection.
    Every embedding has a mean square of exactly 1, so that its RMSNorm (eps 0) is itself and exact in bfloat16; wo and the output projection are
    identities, the feed-forward block adds zero."""
    rng = np.random.default_rng(seed)
    dim, kv = heads * hd, kv_heads * hd
    emb = np.empty((dim, dim), np.float32)  # as many tokens as dimensions
    for row in emb:
        row[:] = rng.permutation(np.where(np.arange(dim) < dim * 5 // 16, 1.75, 0.25)) * rng.choice([-1.0, 1.0], dim)
    assert np.array_equal((emb.astype(np.float64) ** 2).mean(1), np.ones(dim))
    w = {"tok_embeddings": emb, "norm": np.ones(dim, np.float32), "layers.0.attention_norm": np.ones(dim, np.float32), "layers.0.ffn_norm": np.ones(dim, np.float32)}
    mats = {"wq": rng.integers(-12, 13, (dim, dim)), "wk": rng.integers(-12, 13, (kv, dim)), "wv": rng.integers(-127, 128, (kv, dim))}
    mats["wv"][::3] //= 16  # dimensions of different sizes
    for name, v in mats.items():
        w["layers.0." + name] = q8_weight(v)
    one = np.zeros((dim, dim), np.int64)
    np.fill_diagonal(one, 64)  # 1/2
    w["layers.0.wo"], w["output"] = q8_weight(one), q8_weight(one)
    for name, n, k in (("w1", 256, dim), ("w3", 256, dim), ("w2", dim, 256)):
        w["layers.0." + name] = q8_weight(np.zeros((n, k), np.int64))
    return emb, mats, w


# The attention's own precision. With q, k and v exact, its result can be worked out in double and rounded to bfloat16; the kernel's result is that
# wherever its error before the rounding (some 2^-22 per operand) does not carry it over the middle between two bfloat16 numbers: 2^-9 of a value
# apart, so about one in a thousand. Operands of one half each (11 bits) would miss one in five.
@pytest.mark.parametrize("heads,kv_heads,hd", [(8, 8, 64), (4, 4, 128), (4, 1, 128)])
def test_precision(heads, kv_heads, hd):
    dim = heads * hd
    emb, mats, w = attention_model(heads, kv_heads, hd, seed=heads + hd)
    dec = LlamaDecoder(1, dim, heads, kv_heads, 256, dim, 400, eps=0.0)
    dec.load(w)
    missed = total = 0
    for T in (1, 2, 33, 63, 64, 65, 100, 127, 128, 129, 200, 257, 300):
        toks = np.random.default_rng(T).integers(0, dim, T).astype(np.int32)
        x = emb[toks].astype(np.float64)
        split = T // 3  # the keys before it come from the cache
        if split:
            dec.prompt(toks[:split], 0)
        got, _ = dec.prompt(toks[split:], split)
        q, k, v = (x @ (mats[name] / 128.0).T for name in ("wq", "wk", "wv"))
        half = hd // 2
        ang = np.arange(T)[:, None] * 10000.0 ** (-2.0 * np.arange(half) / hd)
        c, s = np.cos(ang).astype(np.float32).astype(np.float64)[:, None], np.sin(ang).astype(np.float32).astype(np.float64)[:, None]

        def rope(a):
            a = a.reshape(T, -1, hd)
            return np.concatenate([a[..., :half] * c - a[..., half:] * s, a[..., :half] * s + a[..., half:] * c], -1)

        q, k, v = rope(q)[-1], rope(k), v.reshape(T, kv_heads, hd)
        att = np.empty((heads, hd))
        for h in range(heads):
            sc = k[:, h * kv_heads // heads] @ q[h] / np.sqrt(hd)
            p = np.exp(sc - sc.max())
            att[h] = (p / p.sum()) @ v[:, h * kv_heads // heads]
        want = torch.from_numpy(att.reshape(-1)).to(torch.bfloat16).double().numpy() / 2
        res = x[-1] + want
        # logits = res / rms(res) / 2 in FP32
        rms = np.sqrt((res ** 2).mean())
        err = np.abs(got.astype(np.float64) * 2 * rms - res)
        missed += int((err > np.abs(want) * 2.0 ** -10 + 4e-6 * np.abs(res).max()).sum())
        total += dim
    assert missed <= total // 50, (missed, total)
    dec.close()


# A bad token is seen by the tokens behind it alone, also within a tile of 64 keys. What the earlier ones left in the cache (of every layer) is
# what a run without it leaves.
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("tokens,at", [(40, 39), (40, 20), (100, 70), (130, 129)])
def test_a_bad_token_does_not_reach_back(tokens, at, value):
    cfg = llama_oracle.Config(layers=3, dim=512, heads=4, kv_heads=2, hidden=512, vocab=300, max_seq=tokens + 2)
    model = llama_oracle.random_model(cfg, 1)
    model["tok_embeddings"][7, 100] = value
    dec = LlamaDecoder(cfg.layers, cfg.dim, cfg.heads, cfg.kv_heads, cfg.hidden, cfg.vocab, cfg.max_seq, cfg.eps, cfg.rope_base)
    dec.load(model)
    toks = np.random.default_rng(tokens).integers(8, cfg.vocab, tokens).astype(np.int32)
    dec.prompt(toks, 0)
    want, _ = dec.forward([3], at)  # in the bad token's place
    toks[at] = 7
    got, _ = dec.prompt(toks, 0)
    assert not np.isfinite(got).any()
    got, _ = dec.forward([3], at)
    assert np.isfinite(got).all()
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
    dec.close()
