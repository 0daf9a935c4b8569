"""The prompt path's tensor-core attention where its tiles of 64 queries and 64 keys end, against the FP32 decode path on the same weights.

The attention itself keeps FP32 precision; the linears around it round their inputs to bfloat16, so the bar is the prompt path's own: 1e-2
of the largest logit (tests/test_gpu_decoder_prompt.py).
"""
import numpy as np
import pytest

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
