"""The work that a user of the framework has it do, as measurable cases.

Five kinds, each through its public entry point:

  linear      quantised projections, `QuantisedLinear.forward`: single tokens, small and medium
              decode batches, prefill chunks; all code widths, both 16-bit types, both block sizes
              of the configurations, ragged row counts.  One projection called eagerly
              (`projections` 1), or several of the same shape one after another, each with its own
              weights and activations, replayed from a CUDA graph as a serving loop and the
              framework's own benchmark harness do
  create      quantising a dense weight and laying it out for the kernels (`QuantisedLinear.create`,
              then `tiled()`), what loading a model does once per projection
  dequantise  packed weights back to a dense matrix (`kernels.dequantise`)
  decode      one decode step of a custom-llama over a KV cache (`LlamaDecoder`), replayed from a
              CUDA graph as `fdk.models.benchmark` does
  prefill     the prompt in one pass (`LlamaDecoder.prefill`), called eagerly
"""

from __future__ import annotations

import sys
from pathlib import Path

import torch

sys.path.insert(0, str(Path.cwd() / "fused-dequantisation-kernels_b200"))

from fdk import kernels, llama, models  # noqa: E402

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}

# projections [rows n, columns k] of the custom-llama configurations, by model: q|k|v, o, gate|up, down
WIDTHS = {"4B": (3072, 24, 11264), "12B": (4096, 32, 14336), "31B": (6144, 48, 21504)}


def _linear(name, m, n, k, bits, block=64, dtype="bf16", projections=1):
    return {"name": name, "kind": "linear", "m": m, "n": n, "k": k, "bits": bits, "block": block, "dtype": dtype,
            "projections": projections}


def listed():
    return [
        # single-token decode: the o projection of the smallest model, called eagerly (launch latency is
        # what a user feels) ...
        _linear("linear_m1_3072_4bit", 1, 3072, 3072, 4),
        # ... and the largest square matrix of the kernel sweep, the headline of the benchmark: eight
        # weight sets (285 MB, more than L2) in one graph
        _linear("linear_m1_8192_4bit_graph8", 1, 8192, 8192, 4, projections=8),
        # a handful of sequences decoded together, an odd number of them: a 12B gate projection at 2 bits
        _linear("linear_m5_14336x4096_2bit", 5, 14336, 4096, 2),
        # sixteen sequences, 3-bit codes
        _linear("linear_m16_8192_3bit_graph4", 16, 8192, 8192, 3, projections=4),
        # continuous batching: some dozens of sequences, 4B gate projections
        _linear("linear_m48_11264x3072_4bit_graph4", 48, 11264, 3072, 4, projections=4),
        # a short prompt through a matrix with ragged sizes, 8 bits in fp16, blocks of 64 (batch of the kernel tests)
        _linear("linear_m200_ragged_8bit_fp16", 200, 5003, 3008, 8, 64, "fp16"),
        # a prefill chunk through the fused gate|up projection of the 12B model
        _linear("linear_m2048_28672x4096_4bit", 2048, 28672, 4096, 4),
        # loading: one 4B gate projection quantised to 4 bits
        {"name": "create_11264x3072_4bit", "kind": "create", "n": 11264, "k": 3072, "bits": 4, "block": 64, "dtype": "bf16"},
        # the dense matrix back: export, or a layer outside the kernels' range
        {"name": "dequantise_8192_4bit", "kind": "dequantise", "n": 8192, "k": 8192, "bits": 4, "block": 64, "dtype": "bf16"},
        # The models have the widths of the 4B configuration and fewer layers: every layer does the same
        # work, and through its full depth two correct implementations differ by 4-5 % in the logits of
        # random weights, too much to tell right from wrong.
        # interactive serving: one sequence, a conversation of a thousand tokens in the cache; the
        # output projection quantised too (`skip=None`), so that it keeps the share that it has at full depth
        {"name": "decode_4B_b1_ctx1000", "kind": "decode", "model": "4B", "layers": 8, "batch": 1, "context": 1000, "bits": 4, "quantised_head": True},
        # batched serving: 32 sequences, contexts of two thousand tokens, the default 16-bit output projection
        {"name": "decode_4B_b32_ctx2000", "kind": "decode", "model": "4B", "layers": 8, "batch": 32, "context": 2000, "bits": 4, "quantised_head": False},
        # a prompt of a thousand tokens, not a multiple of any tile
        {"name": "prefill_4B_b1_t1000", "kind": "prefill", "model": "4B", "layers": 4, "batch": 1, "tokens": 1000, "bits": 4, "quantised_head": True},
    ]


def _log_int(rng, low, high):
    return max(low, min(high, round(low * (high / low) ** rng.random())))


def _bits(rng):
    return rng.choice([4, 4, 4, 4, 3, 2, 1, 8])


def draw(rng):
    kind = rng.choices(["linear", "create", "dequantise", "decode", "prefill"], [12, 2, 2, 3, 2])[0]
    if kind in ("linear", "create", "dequantise"):
        block = rng.choice([64, 64, 64, 128])
        n = _log_int(rng, 256, 28672)
        if rng.random() < 0.5:  # half of the row counts are whole tiles, the others are ragged
            n = (n + 63) // 64 * 64
        k = max(1, round(_log_int(rng, 256, 20480) / block)) * block
        case = {"kind": kind, "n": n, "k": k, "bits": _bits(rng), "block": block, "dtype": rng.choice(["bf16", "bf16", "bf16", "fp16"])}
        if kind == "linear":
            case["m"] = min(_log_int(rng, 1, 2048), 2048 * 28672 * 4096 // (n * k))
            case["projections"] = rng.choice([1, 4, 8]) if case["m"] <= 256 else 1
        else:  # a matrix of at most 128 M weights
            case["n"] = min(n, (1 << 27) // k)
        return case
    model = rng.choice(["4B", "4B", "12B"])
    case = {"kind": kind, "model": model, "bits": _bits(rng), "quantised_head": rng.random() < 0.5}
    if kind == "decode":
        case["layers"] = rng.randint(2, 8 if model == "4B" else 6)
        case["batch"] = _log_int(rng, 1, 64)
        case["context"] = _log_int(rng, 16, min(4096, 65536 // case["batch"]))
    else:
        case["layers"] = rng.randint(2, 4)
        case["batch"] = _log_int(rng, 1, 8)
        case["tokens"] = _log_int(rng, 17, (1024 if model == "4B" else 512) // case["batch"])
    return case


def _codebook(bits, dtype, device):
    """Sorted centroids of normal weights, in units of the block scale (the mean magnitude up to 2
    bits, the largest magnitude from 3 bits on); 8-bit codes use the default grid."""
    if bits == 8:
        return None
    c = models.kmeans_like_codebook(bits).float()
    return (c if bits <= 2 else c / c.abs().max()).to(device, dtype)


def _dense(n, k, seed, dtype):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn((n, k), generator=gen, device="cuda") * k**-0.5).to(dtype), gen


def _dims(case):
    dims = models.get_custom_llama_dims(case["model"])
    dims.num_hidden_layers = case["layers"]
    return dims


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("decode", "prefill"):
        return _prepare_model(case, seed)
    dtype = DTYPES[case["dtype"]]
    n, k = case["n"], case["k"]
    weight, gen = _dense(n, k, seed, dtype)
    config = models.QuantisationConfig(case["bits"], case["block"])
    lut = _codebook(case["bits"], dtype, weight.device)
    if kind == "create":
        return {"kind": kind, "weight": weight, "config": config, "lut": lut}
    layer = models.QuantisedLinear.create(weight, config, lut=lut)
    if kind == "dequantise":
        return {"kind": kind, "layer": layer}
    pairs = []
    for i in range(case["projections"]):
        if i > 0:
            weight = torch.randn((n, k), generator=gen, device="cuda").mul_(k**-0.5).to(dtype)
            layer = models.QuantisedLinear.create(weight, config, lut=lut)
        layer.tiled()
        pairs.append((layer, torch.randn((case["m"], k), generator=gen, device="cuda").to(dtype)))
    if len(pairs) == 1:
        return {"kind": kind, "layer": layer, "x": pairs[0][1]}
    graph, stream, outs = _capture(lambda: [layer(x) for layer, x in pairs])
    return {"kind": "graph", "pairs": pairs, "graph": graph, "stream": stream, "outs": outs}


def _capture(step, between=lambda: None):
    """`step` run once (which allocates the stream's workspace) and then captured -> graph, stream, its outputs."""
    graph = torch.cuda.CUDAGraph()
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.no_grad(), torch.cuda.stream(stream):
        step()
        between()
        stream.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            outs = step()
    stream.synchronize()
    return graph, stream, outs


def _prepare_model(case, seed):
    dims = _dims(case)
    bits, batch, device = case["bits"], case["batch"], torch.device("cuda", torch.cuda.current_device())
    config = models.QuantisationConfig(bits, 64, skip=None if case["quantised_head"] else "^lm_head$")
    model = llama.LlamaDecoder.random_init(dims, config, device, seed=seed, lut=_codebook(bits, torch.bfloat16, device))
    gen = torch.Generator(device=device).manual_seed(seed + 1)
    caches = None
    if case["kind"] == "prefill":
        tokens = case["tokens"]
        model.allocate(batch, tokens + 64)  # room for an answer
        ids = torch.randint(0, dims.vocab_size, (batch, tokens), generator=gen, device=device)
        caches = [c[:, :, :tokens] for c in model.k_cache + model.v_cache]
        return {"kind": "prefill", "model": model, "ids": ids, "caches": caches}
    context = case["context"]
    model.allocate(batch, context + 64)
    model.fill_cache_synthetic(context, seed=seed + 2)
    ids = torch.randint(0, dims.vocab_size, (batch,), generator=gen, device=device)
    caches = [c[:, :, context] for c in model.k_cache + model.v_cache]  # what the step appends
    graph, stream, logits = _capture(lambda: model(ids), lambda: model.position.fill_(context))
    return {"kind": "decode", "model": model, "ids": ids, "graph": graph, "stream": stream, "logits": logits,
            "caches": caches, "context": context}


def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["layer"](state["x"])
    if kind == "graph":
        state["graph"].replay()
        return state["outs"]
    if kind == "create":
        layer = models.QuantisedLinear.create(state["weight"], state["config"], lut=state["lut"])
        return layer.weight_data.data, layer.scale.data, layer.lut, layer.tiled()
    if kind == "dequantise":
        layer = state["layer"]
        return kernels.dequantise(layer.weight_data, layer.lut, layer.scale)
    model = state["model"]
    if kind == "prefill":
        with torch.no_grad():
            logits = model.prefill(state["ids"])
        return logits, state["caches"]
    model.position.fill_(state["context"])  # the same step again, not the next one
    state["graph"].replay()
    return state["logits"], state["caches"]


def work(case):
    kind = case["kind"]
    if kind in ("linear", "create", "dequantise"):
        n, k = case["n"], case["k"]
        packed = n * k * case["bits"] / 8 + n * (k // case["block"]) * 2
        if kind == "linear":
            count = case["projections"]
            return {"bytes": count * (packed + case["m"] * (n + k) * 2), "flops": count * 2 * case["m"] * n * k}
        if kind == "create":  # the packed tensors and their tiled copy
            return {"bytes": 2 * n * k + packed + n * k * case["bits"] / 8 + n * (k // 64) * 2, "flops": 0}
        return {"bytes": packed + 2 * n * k, "flops": n * k}
    hidden, heads, ffn = WIDTHS[case["model"]]
    vocab, kv = 128256, 8 * 128
    weights = case["layers"] * (hidden * (heads * 128 + 2 * kv) + heads * 128 * hidden + 3 * hidden * ffn)
    head = vocab * hidden
    per_weight = case["bits"] / 8 + 2 / 64
    packed = weights * per_weight + head * (per_weight if case["quantised_head"] else 2)
    batch = case["batch"]
    if kind == "decode":
        cached = case["layers"] * batch * case["context"] * kv * 2
        return {"bytes": packed + 2 * cached + batch * vocab * 2,
                "flops": 2 * batch * (weights + head) + 4 * case["layers"] * batch * (case["context"] + 1) * heads * 128}
    t = case["tokens"]
    written = case["layers"] * batch * t * kv * 2
    return {"bytes": packed + 2 * written + batch * (vocab * 2 + t * hidden * 2),
            "flops": 2 * batch * (t * weights + head) + 2 * case["layers"] * batch * t * (t + 1) * heads * 128}


def tolerance(case):
    kind = case["kind"]
    if kind == "dequantise":
        return "exact"
    if kind == "create":  # up to 2 bits the scale is a rounded mean, and a tie of its sums moves codes
        return "exact" if case["bits"] > 2 else {"rel": 1e-3, "max": 2e-2, "differ": 1e-3}
    if kind == "linear":  # one rounding of the result, and in the tensor-core form one of each weight
        return {"rel": 1e-2, "max": 6e-2} if case["dtype"] == "bf16" else {"rel": 1.5e-3, "max": 1e-2}
    return {"rel": 3e-2, "max": 0.3}  # bf16 activations: about 1e-2 * sqrt(layers) between correct implementations
