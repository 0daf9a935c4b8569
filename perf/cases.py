"""The work this library is used for, as cases that can be timed and compared through its public entry points.

A case is a dict of plain values. Its "kind" says which entry point it stands for:

* ``linear``      ``Gguf.linear``: y = x W^T (+ bias) in float32. One row of x is a decode step of one sequence, 2 to 16 rows are
                  a batch of sequences (or a short run of tokens), more rows a prompt or a training batch in full precision.
                  ``host`` takes numpy arrays, as a caller without device memory of its own does.
* ``bf16``        ``Gguf.linearBf16``: the prompt form of the linear, bfloat16 x, tensor cores.
* ``backward``    ``Gguf.linearBackward``: the input gradient, as fine-tuning with frozen quantised weights needs it.
* ``dequantize``  ``Gguf.dequantize`` into a tensor of the caller.
* ``quantize``    ``Quant.quantizeQ8Blocks``: float32 to Q8_0 blocks.
* ``step``        ``LlamaDecoder``: one decode step, ``mode`` "single" (one sequence), "batch" (one token of each of several
                  sequences) or "chunk" (a short run of consecutive tokens of one sequence in full precision).
* ``prompt``      ``LlamaDecoder.prompt``: a whole prompt in one pass over the weights.

Decoders have the widths of whole models and fewer layers; every layer has its own device memory, so a step streams its weights
from device memory as that of the whole model does.
"""
import math

import numpy as np
import torch

from jitnn_b200 import DType, Gguf, Quant, Tensor, synth
from jitnn_b200.decoder import LlamaDecoder

LINEAR_FORMATS = ("Q4_K", "Q6_K", "Q8_0", "Q5_K", "Q4_0", "Q4_1")
# dim, heads, key/value heads, feed-forward width
WIDTHS = {
    "small": (1024, 16, 16, 2816),  # head size 64
    "1b": (2048, 16, 16, 5632),
    "7b": (4096, 32, 32, 11008),
    "7b-gqa": (4096, 32, 8, 14336),
    "70b": (8192, 64, 8, 28672),
}
MAX_SEQ = 2048
MAX_FLOPS = 2.0 * 4096 * 11008 * 2048  # of the largest listed linear
MAX_ELEMENTS = 32000 * 4096


def listed():
    return [
        # one token through an attention projection of a 7B-shaped model: the smallest call, latency counts
        {"name": "linear_q4k_4096x4096_m1", "kind": "linear", "format": "Q4_K", "n": 4096, "k": 4096, "m": 1, "bias": False, "host": False},
        # the same from and to host arrays, with bias: a caller that keeps its activations in host memory
        {"name": "linear_q8_0_4096x4096_m1_host", "kind": "linear", "format": "Q8_0", "n": 4096, "k": 4096, "m": 1, "bias": True, "host": True},
        # the output projection of eight sequences decoded together
        {"name": "linear_q6k_32000x4096_m8", "kind": "linear", "format": "Q6_K", "n": 32000, "k": 4096, "m": 8, "bias": False, "host": False},
        # a ragged run of tokens through a feed-forward projection in full precision (the default of every row count)
        {"name": "linear_q4k_11008x4096_m200", "kind": "linear", "format": "Q4_K", "n": 11008, "k": 4096, "m": 200, "bias": False, "host": False},
        # prompt linears: an ordinary prompt, and a long one through the widest k
        {"name": "bf16_q4k_11008x4096_m512", "kind": "bf16", "format": "Q4_K", "n": 11008, "k": 4096, "m": 512, "bias": False},
        {"name": "bf16_q6k_4096x11008_m2048", "kind": "bf16", "format": "Q6_K", "n": 4096, "k": 11008, "m": 2048, "bias": False},
        # the input gradient of a feed-forward projection for a small training batch
        {"name": "backward_q4k_11008x4096_m128", "kind": "backward", "format": "Q4_K", "n": 11008, "k": 4096, "m": 128},
        # decode and encode of whole weights
        {"name": "dequantize_q6k_4096x11008", "kind": "dequantize", "format": "Q6_K", "n": 4096, "k": 11008},
        {"name": "quantize_q8_0_4096x4096", "kind": "quantize", "n": 4096, "k": 4096},
        # decode steps: one sequence with a 7B-shaped Q4_K / Q6_K mix, sixteen sequences with 70B widths
        {"name": "step_7b_mix_single_pos576", "kind": "step", "mode": "single", "width": "7b", "layers": 8, "mix": "Q4_K_M", "vocab": 32000, "rows": 1,
         "pos": 576, "logits": True},
        {"name": "step_70b_q4k_batch16_pos256", "kind": "step", "mode": "batch", "width": "70b", "layers": 2, "mix": "Q4_K", "vocab": 32000, "rows": 16,
         "pos": 256, "logits": True},
        # a 512-token prompt
        {"name": "prompt_7b_mix_512", "kind": "prompt", "width": "7b", "layers": 8, "mix": "Q4_K_M", "vocab": 32000, "rows": 512, "pos": 0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shape(rng, fmt, step):
    """n and k of a weight: from small layers to the widest of a 7B shape, n of any size, k in whole blocks."""
    while True:
        n = _log_int(rng, 256, 32000)
        if rng.random() < 0.7:
            n = max(64, n // 64 * 64)
        unit = 256 if fmt.endswith("_K") or rng.random() < 0.7 else step
        k = max(unit, _log_int(rng, 512, 14336) // unit * unit)
        if n * k <= MAX_ELEMENTS:
            return n, k


def draw(rng):
    kind = rng.choice(["linear"] * 5 + ["bf16"] * 2 + ["backward"] + ["dequantize"] + ["quantize"] + ["step"] * 2 + ["prompt"])
    fmt = rng.choice(LINEAR_FORMATS)
    if kind == "linear":
        n, k = _shape(rng, fmt, 32)
        where = rng.random()
        m = 1 if where < 0.35 else (rng.randint(2, 16) if where < 0.7 else _log_int(rng, 17, 512))
        m = max(1, min(m, int(MAX_FLOPS / (2.0 * n * k))))
        return {"kind": kind, "format": fmt, "n": n, "k": k, "m": m, "bias": rng.random() < 0.3, "host": m <= 16 and rng.random() < 0.2}
    if kind == "bf16":
        n, k = _shape(rng, fmt, 64)
        m = max(64, min(_log_int(rng, 64, 4096), int(MAX_FLOPS / (2.0 * n * k))))
        return {"kind": kind, "format": fmt, "n": n, "k": k, "m": m, "bias": rng.random() < 0.3}
    if kind == "backward":
        n, k = _shape(rng, fmt, 32)
        m = 1 if rng.random() < 0.2 else _log_int(rng, 2, 512)
        return {"kind": kind, "format": fmt, "n": n, "k": k, "m": m}
    if kind == "dequantize":
        fmt = rng.choice(LINEAR_FORMATS + ("Q5_0", "Q5_1", "Q2_K", "Q3_K"))
        n, k = _shape(rng, fmt, 32)
        return {"kind": kind, "format": fmt, "n": n, "k": k}
    if kind == "quantize":
        n, k = _shape(rng, "Q8_0", 32)
        return {"kind": kind, "n": n, "k": k}
    width = rng.choice(list(WIDTHS))
    layers = rng.randint(1, 2) if width == "70b" else rng.randint(2, 8)
    case = {"kind": kind, "width": width, "layers": layers, "mix": rng.choice(["Q4_K_M", "Q4_K_M", "Q4_K", "Q8_0"]), "vocab": rng.choice([32000, 32000, 8001])}
    if kind == "step":
        mode = rng.choice(["single", "single", "batch", "chunk"])
        case.update(mode=mode, rows=1 if mode == "single" else rng.randint(2, 16), pos=_log_int(rng, 1, 1024), logits=rng.random() < 0.5)
        if mode == "batch":
            case["pos"] = min(case["pos"], 384)
    else:
        case.update(rows=_log_int(rng, 24, 768 if width == "70b" else 1536), pos=rng.choice([0, 0, rng.randint(1, 256)]))
    return case


# ---- what a user's program has in hand ---------------------------------------------------------------------------------------

def _blocks(fmt, n, k, g):
    """GGUF blocks of an [n, k] weight ~ N(0, 0.02), made on the GPU, as host bytes."""
    if fmt in ("Q5_0", "Q5_1", "Q2_K", "Q3_K"):  # no quantiser: random quants with scales of an ordinary size
        qk, nb, offsets = {"Q5_0": (32, 22, [0]), "Q5_1": (32, 24, [0, 2]), "Q2_K": (256, 84, [80, 82]), "Q3_K": (256, 110, [108])}[fmt]
        raw = torch.randint(0, 256, (n * k // qk, nb), generator=g, dtype=torch.uint8, device="cuda")
        for off in offsets:
            scale = torch.rand(raw.shape[0], generator=g, device="cuda") * 0.028 + 0.002
            raw[:, off:off + 2] = scale.to(torch.float16).view(torch.uint8).reshape(-1, 2)
        return raw.cpu().numpy()
    w = torch.randn(n, k, generator=g, device="cuda") * 0.02
    blocks = Quant.quantizeQ8Blocks(w) if fmt == "Q8_0" else synth.QUANTIZERS[fmt](w)
    return blocks.cpu().numpy()


def _decoder(case, g):
    dim, heads, kv_heads, hidden = WIDTHS[case["width"]]
    kv_dim = dim // heads * kv_heads
    base = "Q8_0" if case["mix"] == "Q8_0" else "Q4_K"
    fine = "Q6_K" if case["mix"] == "Q4_K_M" else base
    shapes = {"wq": (base, dim, dim), "wk": (base, kv_dim, dim), "wv": (fine, kv_dim, dim), "wo": (base, dim, dim),
              "w1": (base, hidden, dim), "w3": (base, hidden, dim), "w2": (fine, dim, hidden)}
    sets = [{name: (t, _blocks(t, n, k, g), n, k) for name, (t, n, k) in shapes.items()} for _ in range(min(2, case["layers"]))]
    weights = {"tok_embeddings": torch.randn(case["vocab"], dim, generator=g, device="cuda").cpu().numpy(),
               "output": (fine, _blocks(fine, case["vocab"], dim, g), case["vocab"], dim),
               "norm": (1.0 + 0.1 * torch.randn(dim, generator=g, device="cuda")).cpu().numpy()}
    for layer in range(case["layers"]):
        for name, value in sets[layer % len(sets)].items():
            weights["layers.%d.%s" % (layer, name)] = value
        for name in ("attention_norm", "ffn_norm"):
            weights["layers.%d.%s" % (layer, name)] = (1.0 + 0.1 * torch.randn(dim, generator=g, device="cuda")).cpu().numpy()
    dec = LlamaDecoder(case["layers"], dim, heads, kv_heads, hidden, case["vocab"], MAX_SEQ)
    dec.load(weights)
    return dec


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    state = {"case": case}
    if kind in ("step", "prompt"):
        dec = _decoder(case, g)
        seqs = case["rows"] if kind == "step" and case["mode"] == "batch" else 1
        if seqs > 1:
            dec.set_sequences(seqs)
        tokens = torch.randint(0, case["vocab"], (seqs, case["pos"] + 1), generator=g, device="cuda").cpu().numpy().astype(np.int32)
        for s in range(seqs):  # the keys and values of the positions before this call
            for at in range(0, case["pos"], 16):
                dec.enqueue(tokens[s, at:min(at + 16, case["pos"])], at, seq=s)
        state["decoder"] = dec
        state["tokens"] = torch.randint(0, case["vocab"], (case["rows"],), generator=g, device="cuda").cpu().numpy().astype(np.int32)
        if kind == "step":  # a program that decodes has taken steps before; their results are overwritten
            for _ in range(2):
                run(state)
        return state
    if kind == "quantize":
        state["x"] = torch.randn(case["n"], case["k"], generator=g, device="cuda")
        return state
    n, k = case["n"], case["k"]
    state["w"] = Tensor.quantized(DType[case["format"]], _blocks(case["format"], n, k, g), n, k)
    if kind == "dequantize":
        state["out"] = torch.empty(n, k, device="cuda")
    elif kind == "backward":
        state["g"] = torch.randn(case["m"], n, generator=g, device="cuda")
    else:
        x = torch.randn(case["m"], k, generator=g, device="cuda")
        bias = torch.randn(n, generator=g, device="cuda") if case["bias"] else None
        if kind == "bf16":
            x = x.to(torch.bfloat16)
        elif case["host"]:
            x, bias = x.cpu().numpy(), None if bias is None else bias.cpu().numpy()
        state["x"], state["bias"] = x, bias
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "linear":
        return Gguf.linear(state["x"], state["w"], state["bias"])
    if kind == "bf16":
        return Gguf.linearBf16(state["x"], state["w"], state["bias"])
    if kind == "backward":
        return Gguf.linearBackward(state["g"], state["w"])
    if kind == "dequantize":
        return Gguf.dequantize(state["w"], state["out"])
    if kind == "quantize":
        return Quant.quantizeQ8Blocks(state["x"])
    dec = state["decoder"]
    if kind == "prompt":
        return dec.prompt(state["tokens"], case["pos"])[0]
    if case["mode"] == "batch":
        out = dec.forward_batch(state["tokens"], case["pos"], want_logits=case["logits"])
    else:
        out = dec.forward(state["tokens"], case["pos"], want_logits=case["logits"])
    return list(out)


def _weight_bytes(fmt, n, k):
    t = DType[fmt]
    return n * k // t.blockValues() * t.blockBytes()


def work(case):
    kind = case["kind"]
    if kind in ("step", "prompt"):
        dim, heads, kv_heads, hidden = WIDTHS[case["width"]]
        kv_dim = dim // heads * kv_heads
        base = "Q8_0" if case["mix"] == "Q8_0" else "Q4_K"
        fine = "Q6_K" if case["mix"] == "Q4_K_M" else base
        layer = [(base, dim, dim), (base, kv_dim, dim), (fine, kv_dim, dim), (base, dim, dim), (base, hidden, dim), (base, hidden, dim), (fine, dim, hidden)]
        last = (fine, case["vocab"], dim)
        rows, layers, pos = case["rows"], case["layers"], case["pos"]
        weights = layers * sum(_weight_bytes(*w) for w in layer) + _weight_bytes(*last)
        out_rows = 1 if kind == "prompt" else rows
        flops = 2.0 * (rows * layers * sum(n * k for _, n, k in layer) + out_rows * last[1] * last[2])
        if kind == "step" and case["mode"] == "batch":
            cached, pairs = rows * pos, rows * (pos + 1)
        else:  # consecutive tokens see the cache and each other
            cached, pairs = pos, rows * pos + rows * (rows + 1) // 2
        flops += 4.0 * layers * pairs * dim
        read = 2 * layers * cached * kv_dim * 4
        written = 2 * layers * rows * kv_dim * 4 + (out_rows * case["vocab"] * 4 if case.get("logits", True) else 4 * rows)
        return {"bytes": weights + read + written + rows * dim * 4, "flops": flops}
    n, k = case["n"], case["k"]
    if kind == "quantize":
        return {"bytes": 4 * n * k + n * k // 32 * 34, "flops": 3.0 * n * k}
    weight = _weight_bytes(case["format"], n, k)
    if kind == "dequantize":
        return {"bytes": weight + 4 * n * k, "flops": 2.0 * n * k}
    m = case["m"]
    if kind == "backward":
        return {"bytes": weight + 4 * m * (n + k), "flops": 2.0 * m * n * k}
    x_bytes = 2 if kind == "bf16" else 4
    return {"bytes": weight + x_bytes * m * k + 4 * m * n + (4 * n if case["bias"] else 0), "flops": 2.0 * m * n * k}


def tolerance(case):
    kind = case["kind"]
    if kind in ("dequantize", "quantize"):
        return "exact"
    if kind == "bf16":
        return {"rel": 5e-3}  # operands of 8 significant bits: each is off by up to 2^-9, at random
    if kind == "prompt":
        return {"rel": 2e-2}  # the same at every linear of every layer
    if kind == "step":
        return {"rel": 1e-4}  # float32 throughout; the rounding of every layer is carried on by the ones behind it
    return {"rel": 1e-5}  # float32 sums
