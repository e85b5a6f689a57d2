"""What a user of the package has it do, as timed cases.

The package is a vLLM quantization plugin: its work is the quantized linear layer at every batch size (decode
steps of 1..16 rows, prefill chunks of up to thousands), the quantized expert layer, the decoder that strings them
together, and the quantizer that makes the codes.  Layer shapes are those of the 9B-class decoder and of the
128-expert layer the benchmark uses; the rest of the range (other widths, odd widths, tensor-parallel shards) is
what ``draw`` covers.

Decode steps run both ways a serving engine runs them: captured once in a CUDA graph and replayed (``graph``), or
launched op by op from Python.

    listed()           the cases
    draw(rng)          one more case of the same ranges
    prepare(case, s)   inputs, layers and (for graph cases) the captured step, from the seed alone
    run(state)         one pass through the public entry points; its outputs
    work(case)         bytes and flops the pass cannot do without
    tolerance(case)    how far another correct implementation at the same precision may be off
"""
import math

import torch

from polarengine_vllm_b200.decoder import DecoderConfig, QuantDecoder
from polarengine_vllm_b200.linear_method import PolarQuantLinearMethod
from polarengine_vllm_b200.moe_method import PolarQuantMoEMethod
from polarengine_vllm_b200.packing import pack_codes_half_block
from polarengine_vllm_b200.quantizer import PolarQuantizer
from polarengine_vllm_b200.utils import get_centroids

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}


# ---------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # one small projection for one token, launched from Python: the latency of a single apply() call
        {"name": "linear_1_token", "kind": "linear", "tokens": 1, "out_f": 4096, "in_f": 4096, "bits": 6, "dtype": "fp16", "bias": False},
        # the four projections of a 9B-class decoder layer for one token, the step replayed as a CUDA graph
        {"name": "layer_1_token_graph", "kind": "layer", "tokens": 1, "hidden": 4096, "kv": 1024, "inter": 12288, "graph": True},
        # the same layer for a handful of sequences, launched from Python (enforce_eager serving)
        {"name": "layer_5_tokens", "kind": "layer", "tokens": 5, "hidden": 4096, "kv": 1024, "inter": 12288, "graph": False},
        # ... and for 16 sequences under a graph
        {"name": "layer_16_tokens_graph", "kind": "layer", "tokens": 16, "hidden": 4096, "kv": 1024, "inter": 12288, "graph": True},
        # a short prompt chunk of odd length through a fused q/k/v projection with a bias, width not a multiple of 128
        {"name": "prefill_200_ragged", "kind": "linear", "tokens": 200, "out_f": 6144, "in_f": 4000, "bits": 5, "dtype": "bf16", "bias": True},
        # a large prompt chunk through the widest layer shape: tensor-core bound
        {"name": "prefill_4096", "kind": "linear", "tokens": 4096, "out_f": 12288, "in_f": 4096, "bits": 4, "dtype": "bf16", "bias": False},
        # the expert layer at its three token counts: one token, a decode batch, a prompt chunk
        {"name": "moe_1_token", "kind": "moe", "tokens": 1, "experts": 128, "hidden": 2688, "inter": 1856, "top_k": 8, "graph": False},
        {"name": "moe_64_tokens_graph", "kind": "moe", "tokens": 64, "experts": 128, "hidden": 2688, "inter": 1856, "top_k": 8, "graph": True},
        {"name": "moe_2048_tokens", "kind": "moe", "tokens": 2048, "experts": 128, "hidden": 2688, "inter": 1856, "top_k": 8, "graph": False},
        # a decode step of the whole decoder (fewer layers and a smaller vocabulary than the 9B one) at cache position 512
        {"name": "decode_step_graph", "kind": "decode", "tokens": 1, "layers": 6, "context": 512, "graph": True},
        # the prompt of that decoder
        {"name": "prompt_512", "kind": "prompt", "tokens": 512, "layers": 6},
        # quantizing one bf16 weight matrix (down_proj) to 4 bits: codes, norms, nibble packing
        {"name": "quantize_4bit", "kind": "quantize", "rows": 4096, "cols": 12288, "bits": 4, "dtype": "bf16"},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _width(rng, lo, hi):
    """Mostly whole 128-blocks, as layers are made; every fourth one ragged."""
    n = _log_int(rng, lo, hi)
    return n // 8 * 8 if rng.random() < 0.25 else max(128, n // 128 * 128)


def draw(rng):
    kind = rng.choice(["linear", "linear", "prefill", "prefill", "layer", "layer", "moe", "decode", "prompt", "quantize"])
    if kind in ("linear", "prefill"):
        tokens = _log_int(rng, 1, 16) if kind == "linear" else _log_int(rng, 17, 4096)
        out_f = _log_int(rng, 1024, 24576) // 16 * 16
        in_f = _width(rng, 1024, 12288)
        while tokens * out_f * in_f > 4096 * 12288 * 4096:  # no more than the largest listed one
            out_f //= 2
        return {"kind": "linear", "tokens": tokens, "out_f": out_f, "in_f": in_f, "bits": rng.choice([3, 4, 5, 6]),
                "dtype": rng.choice(["fp16", "bf16"]), "bias": rng.random() < 0.5}
    if kind == "layer":
        hidden = rng.choice([2048, 2560, 3072, 4096, 5120])
        return {"kind": "layer", "tokens": _log_int(rng, 1, 16), "hidden": hidden, "kv": rng.choice([256, 512, 1024]),
                "inter": rng.choice([2, 3, 4]) * hidden, "graph": rng.random() < 0.5}
    if kind == "moe":
        tokens = _log_int(rng, 1, 2048)
        return {"kind": "moe", "tokens": tokens, "experts": rng.choice([16, 32, 64, 128]), "hidden": rng.choice([1024, 2048, 2688]),
                "inter": rng.choice([768, 1024, 1408, 1856]), "top_k": rng.choice([2, 4, 8]), "graph": tokens <= 64 and rng.random() < 0.5}
    if kind == "decode":
        return {"kind": "decode", "tokens": rng.choice([1, 2, 3, 4, 6, 8, 12, 16, 32]), "layers": rng.randint(2, 6), "context": _log_int(rng, 16, 600),
                "graph": rng.random() < 0.7}
    if kind == "prompt":
        return {"kind": "prompt", "tokens": _log_int(rng, 17, 600), "layers": rng.randint(2, 6)}
    return {"kind": "quantize", "rows": _log_int(rng, 256, 8192), "cols": _width(rng, 1024, 12288), "bits": rng.choice([3, 4, 5, 6]),
            "dtype": rng.choice(["fp16", "bf16", "fp32"])}


# ---------------------------------------------------------------------------------------------- inputs
def _codes_and_norms(out_f, kp, bits, dev, gen):
    """What the quantizer makes of Gaussian weights: Lloyd-Max cells of N(0, 1) draws, block norms around
    0.02 * sqrt(128)."""
    ct = get_centroids(bits).to(dev)
    bounds = (ct[1:] + ct[:-1]) / 2
    codes = torch.empty(out_f, kp, dtype=torch.int8, device=dev)
    step = max(1, (1 << 26) // kp)
    for r in range(0, out_f, step):
        z = torch.randn(min(step, out_f - r), kp, device=dev, generator=gen)
        codes[r:r + step] = torch.bucketize(z, bounds, out_int32=True)
    norms = (0.02 * math.sqrt(128) * (1 + 0.05 * torch.randn(out_f, kp // 128, device=dev, generator=gen))).half()
    return codes, norms


def _linear(sections, in_f, bits, dev, gen):
    """A loaded quantized layer, made the way vLLM makes one: create, load, post-process."""
    method = PolarQuantLinearMethod(128, bits)
    layer = torch.nn.Module()
    out_f = sum(sections)
    with torch.device(dev):
        method.create_weights(layer, in_f, list(sections), in_f, out_f, torch.float16)
    codes, norms = _codes_and_norms(out_f, layer.in_f_padded, bits, dev, gen)
    layer.codes.data.copy_(codes)
    layer.norms.data.copy_(norms)
    method.process_weights_after_loading(layer)
    return method, layer


def _captured(step):
    """The step captured in a CUDA graph after a few warm-up calls on the capture stream."""
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        for _ in range(2):
            step()
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            out = step()
    torch.cuda.current_stream().wait_stream(stream)
    return graph, out


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)

    def randn(*shape, dtype=torch.float16):
        return torch.randn(*shape, device=dev, generator=gen).to(dtype)

    kind = case["kind"]
    if kind == "linear":
        method, layer = _linear([case["out_f"]], case["in_f"], case["bits"], dev, gen)
        x = randn(case["tokens"], case["in_f"], dtype=DTYPES[case["dtype"]])
        bias = randn(case["out_f"]) if case["bias"] else None
        step = lambda: method.apply(layer, x, bias)  # noqa: E731
    elif kind == "layer":
        h, kv, inter, t = case["hidden"], case["kv"], case["inter"], case["tokens"]
        qkv = _linear([h, kv, kv], h, 5, dev, gen)
        o = _linear([h], h, 6, dev, gen)
        gate_up = _linear([inter, inter], h, 3, dev, gen)
        down = _linear([h], inter, 4, dev, gen)
        xs = [randn(t, h), randn(t, h), randn(t, h), randn(t, inter)]
        parts = [(m, layer, x) for (m, layer), x in zip((qkv, o, gate_up, down), xs)]
        step = lambda: [m.apply(layer, x) for m, layer, x in parts]  # noqa: E731
    elif kind == "moe":
        e, h, inter = case["experts"], case["hidden"], case["inter"]
        method = PolarQuantMoEMethod(3, 4)
        layer = torch.nn.Module()
        with torch.device(dev):
            method.create_weights(layer, e, h, inter, torch.float16)
        for rows, kp, bits, codes, norms in ((2 * inter, layer.moe_hidden_padded, 3, layer.w13_codes, layer.w13_norms),
                                             (h, layer.moe_inter_padded, 4, layer.w2_codes, layer.w2_norms)):
            c, n = _codes_and_norms(e * rows, kp, bits, dev, gen)
            codes.data.copy_(pack_codes_half_block(c).view(codes.shape))
            norms.data.copy_(n.view(norms.shape))
            del c, n
        method.process_weights_after_loading(layer)
        x, logits, top_k = randn(case["tokens"], h), randn(case["tokens"], e), case["top_k"]
        step = lambda: method.apply(layer, x, logits, top_k, True)  # noqa: E731
    elif kind in ("decode", "prompt"):
        cfg = DecoderConfig(n_layers=case["layers"], vocab=32768)
        batch = case["tokens"] if kind == "decode" else 1
        model = QuantDecoder(cfg, dev, seed=seed, max_len=640, batch=batch)
        t = 1 if kind == "decode" else case["tokens"]
        ids = torch.randint(0, cfg.vocab, (batch, t), device=dev, generator=gen)
        pos = 0
        if kind == "decode":  # a filled cache; the step writes (and rewrites) position `context`
            for cache in (*model.k_cache, *model.v_cache):
                cache[:, :, :case["context"]] = randn(batch, cfg.n_kv_heads, case["context"], cfg.head_dim)
            pos = torch.tensor(case["context"], device=dev, dtype=torch.int64)

        def step():
            logits = model.forward(ids, pos, return_logits=True)
            return {"logits": logits, "k": model.k_cache, "v": model.v_cache}
    else:
        w = 0.02 * randn(case["rows"], case["cols"], dtype=DTYPES[case["dtype"]])
        quantizer, bits = PolarQuantizer(), case["bits"]

        def step():
            q = quantizer.quantize_tensor_gpu(w, bits)
            codes = pack_codes_half_block(q["codes"]) if bits <= 4 else q["codes"]
            return {"codes": codes, "norms": q["norms"], "ct_scaled": q["ct_scaled"]}
    if case.get("graph"):
        graph, out = _captured(step)

        def replay():
            graph.replay()
            return out
        return {"step": replay, "captured": step}  # the graph reads the tensors that `step` holds
    return {"step": step}


def run(state):
    return state["step"]()


# ---------------------------------------------------------------------------------------------- floors, tolerances
def _linear_bytes(out_f, in_f, bits, tokens, out_bytes=2):
    kp = -(-in_f // 128) * 128
    return (out_f * kp // (2 if bits <= 4 else 1) + out_f * (kp // 128) * 2 + (1 << bits) * 4
            + tokens * in_f * 2 + tokens * out_f * out_bytes)


def work(case):
    kind = case["kind"]
    if kind == "linear":
        t, n, k = case["tokens"], case["out_f"], case["in_f"]
        return {"bytes": _linear_bytes(n, k, case["bits"], t), "flops": 2 * t * n * k}
    if kind == "layer":
        t, h, kv, inter = case["tokens"], case["hidden"], case["kv"], case["inter"]
        shapes = ((h + 2 * kv, h, 5), (h, h, 6), (2 * inter, h, 3), (h, inter, 4))
        return {"bytes": sum(_linear_bytes(n, k, b, t) for n, k, b in shapes), "flops": sum(2 * t * n * k for n, k, _ in shapes)}
    if kind == "moe":
        t, e, h, inter = case["tokens"], case["experts"], case["hidden"], case["inter"]
        pairs = t * case["top_k"]
        active = e * (1 - (1 - case["top_k"] / e) ** t)  # experts that uniform routing gives a token
        per = _linear_bytes(2 * inter, h, 3, 0) + _linear_bytes(h, inter, 4, 0)
        return {"bytes": active * per + t * (2 * h + e) * 2, "flops": 2 * pairs * 3 * h * inter}
    if kind in ("decode", "prompt"):
        c = DecoderConfig()
        t, vocab = case["tokens"], 32768
        heads = t if kind == "decode" else 1  # rows that go through the LM head
        h, kv, q = c.hidden, c.n_kv_heads * c.head_dim, c.n_heads * c.head_dim
        shapes = ((q + 2 * kv, h, 5), (h, q, 6), (2 * c.intermediate, h, 3), (h, c.intermediate, 4))
        per = sum(_linear_bytes(n, k, b, 0) for n, k, b in shapes)
        seen = case["context"] + 1 if kind == "decode" else (t + 1) / 2  # cache positions a token attends to, on average
        cache = t * seen * kv * 2 * 2 if kind == "decode" else t * kv * 2 * 2
        flops = case["layers"] * (sum(2 * t * n * k for n, k, _ in shapes) + 4 * t * seen * q) + 2 * heads * vocab * h
        return {"bytes": case["layers"] * (per + cache) + _linear_bytes(vocab, h, 6, heads, 4) + t * h, "flops": flops}
    rows, cols, bits = case["rows"], case["cols"], case["bits"]
    kp = -(-cols // 128) * 128
    return {"bytes": rows * cols * (4 if case["dtype"] == "fp32" else 2) + rows * kp // (2 if bits <= 4 else 1) + rows * (kp // 128) * 2,
            "flops": rows * kp * 9}


def tolerance(case):
    kind, t = case["kind"], case["tokens"] if "tokens" in case else 0
    if kind == "quantize":
        # rotation and norm are fp32 sums: a value on a cell boundary may change its cell, a norm its fp16 rounding
        return {"rel": 1e-4, "max": 2e-3, "differ": 1e-5}
    if kind in ("linear", "layer"):
        # up to 16 rows multiply fp16 operands, more rows bf16 ones; fp16 results
        return {"rel": 2e-3 if t <= 16 else 6e-3}
    # chains of several such products with fp16 (or bf16) operands between them
    return {"rel": 1e-2}
