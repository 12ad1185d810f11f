"""The work that users of this package have it do, as measured cases.

Four kinds of call, all through the public entry points:

* ``decode``: one ``attention()`` call of one layer over a compressed cache and its dense window -- what every layer
  of a serving loop issues for every generated token;
* ``pack``: ``compress()`` with a given clustering (both sides packed), for callers that cluster themselves;
* ``layer``: one request batch on one attention layer: a fresh ``ResKVLayerCache`` takes the prompt (clustering and
  packing), then ``steps`` tokens are appended and attended to, decode groups being compressed on the way;
* ``model``: ``ResKVLlama`` with its captured-graph decode: prefill, then ``steps`` tokens.

Sizes are those of this repository's benchmark and tests (32 query / 8 KV heads, contexts up to 65536, batch 1 to 32,
window 32, groups of 64, 32 clusters, 10 or 15 Lloyd iterations) and odd ones around them.
"""

from __future__ import annotations

import math

import torch

from reskv_b200 import ResKVKernelConfig, attention, compress
from reskv_b200.cache import ResKVLayerCache
from reskv_b200.compression import cluster
from reskv_b200.models.llama import LlamaShape, ResKVLlama
from reskv_b200.synthetic import gaussian, mixture
from reskv_b200.tensors import metadata_spec, payload_width

_GROUP, _RECENT = 64, 32
# (token, KV head) pairs of the largest listed decode case: 8 sequences x 8 heads x 65536 tokens
_MOST_PAIRS = 8 * 8 * 65536


def listed():
    return [
        # -- decode ---------------------------------------------------------------------------------------------------
        # the smallest call: a short conversation, one user, default settings
        _decode("decode b1 t192 fp16 s50", 1, 192, recent=40),
        # one user at 8K with the plan that "auto" picks at sparsity 0.75 (4:16 FP16)
        _decode("decode b1 t8128 auto s75", 1, 8128, sparsity=0.75, recent=64),
        # a ragged context, eight query heads per KV head, long-run tables of 64 centroids, 1-of-4 INT4
        _decode("decode b3 t4870 int4 r8", 3, 4870, sparsity=0.75, bits=4, ratio=8, clusters=64, recent=77),
        # default settings at an ordinary batch, three quarters into an 8K context
        _decode("decode b12 t6016 fp16 s50", 12, 6016, recent=50),
        # the benchmark's workload: FP16 bitmap layout at 8K, batch 32
        _decode("decode b32 t8128 fp16 s75", 32, 8128, sparsity=0.75, layout="unstructured", recent=64),
        # quantised residuals at 16K, batch 8
        _decode("decode b8 t16320 int4 s50", 8, 16320, bits=4, theta=1000000.0, recent=32),
        # one GPU's share of the longest context served
        _decode("decode b8 t65536 fp16 s75", 8, 65536, sparsity=0.75, layout="unstructured", recent=95),
        # -- packing alone --------------------------------------------------------------------------------------------
        # both sides of an 8K prompt packed with the "auto" plan at sparsity 0.75, batch 8
        _pack("pack b8 t8128 auto s75", 8, 8128, sparsity=0.75),
        # -- a layer: prompt and generated tokens ---------------------------------------------------------------------
        # one user, a short prompt and an answer that compresses two decode groups
        _layer("layer b1 p1200 +150", 1, 1200, 150),
        # time to first token of an 8K prompt batch: clustering, packing, one step
        _layer("layer b8 p8192 +1 s75", 8, 8192, 1, sparsity=0.75, layout="unstructured"),
        # the benchmark's batch: prompt, then enough steps for one decode group
        _layer("layer b32 p8192 +48 s75", 32, 8192, 48, sparsity=0.75, layout="unstructured"),
        # -- a model --------------------------------------------------------------------------------------------------
        _model("model b4 p1024 +72", 4, 1024, 72),
    ]


def _decode(name, batch, tokens, *, kv_heads=8, ratio=4, sparsity=0.5, bits=16, layout="auto", clusters=32, recent=32,
            theta=500000.0, start=0):
    return _named(name, kind="decode", batch=batch, kv_heads=kv_heads, ratio=ratio, tokens=tokens, sparsity=sparsity,
                  bits=bits, layout=layout, clusters=clusters, recent=recent, theta=theta, start=start)


def _pack(name, batch, tokens, *, kv_heads=8, sparsity=0.5, bits=16, layout="auto", clusters=32):
    return _named(name, kind="pack", batch=batch, kv_heads=kv_heads, tokens=tokens, sparsity=sparsity, bits=bits,
                  layout=layout, clusters=clusters)


def _layer(name, batch, tokens, steps, *, kv_heads=8, ratio=4, sparsity=0.5, bits=16, layout="auto", iterations=10,
           theta=500000.0, sinks=0):
    return _named(name, kind="layer", batch=batch, kv_heads=kv_heads, ratio=ratio, tokens=tokens, steps=steps,
                  sparsity=sparsity, bits=bits, layout=layout, iterations=iterations, theta=theta, sinks=sinks)


def _model(name, batch, tokens, steps, *, sparsity=0.5, bits=16, layers=2):
    return _named(name, kind="model", batch=batch, tokens=tokens, steps=steps, sparsity=sparsity, bits=bits, layers=layers)


def _named(name, **fields):
    return fields if name is None else {"name": name, **fields}


# (sparsity, bits, layout), more often what the settings object picks by itself
_SETTINGS = [
    (0.5, 16, "auto"), (0.75, 16, "auto"), (0.75, 16, "unstructured"), (0.5, 4, "auto"), (0.75, 4, "auto"), (0.5, 2, "auto"),
    (0.75, 2, "auto"), (0.5, 16, "tiled"), (0.5, 4, "compact"), (0.75, 4, "compact"),
]
_WEIGHTS = [4, 4, 4, 3, 2, 1, 1, 1, 1, 1]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    sparsity, bits, layout = rng.choices(_SETTINGS, _WEIGHTS)[0]
    kind = rng.choices(("decode", "pack", "layer", "model"), (10, 3, 6, 1))[0]
    batch = spread(1, 32)
    kv_heads = rng.choice((8, 8, 8, 4, 2))
    ratio = rng.choice((4, 4, 4, 8, 1))
    theta = rng.choice((500000.0, 500000.0, 1000000.0, 10000.0))
    if kind == "decode":
        most = min(65536, _MOST_PAIRS // (batch * kv_heads * max(1, ratio // 4)))
        tokens = spread(96, most)
        if rng.random() < 0.6:  # what a layer cache holds: whole groups
            tokens = max(_GROUP, tokens // _GROUP * _GROUP)
        return _decode(None, batch, tokens, kv_heads=kv_heads, ratio=ratio, sparsity=sparsity, bits=bits, layout=layout,
                       clusters=rng.choice((32, 32, 32, 16, 64)), recent=rng.randint(_RECENT, _RECENT + _GROUP - 1),
                       theta=theta, start=rng.choice((0, 0, 4)))
    if kind == "pack":
        return _pack(None, batch, spread(64, min(16384, 32 * 8 * 8192 // (batch * kv_heads))), kv_heads=kv_heads,
                     sparsity=sparsity, bits=bits, layout=layout, clusters=rng.choice((32, 32, 16, 64)))
    if kind == "layer":
        tokens = spread(200, min(16384, 24 * 8 * 8192 // (batch * kv_heads)))
        steps = rng.choice((1, rng.randint(2, 48), rng.randint(48, 160)))
        if batch * kv_heads * tokens > 4 * 8 * 8192:
            steps = min(steps, 48)
        return _layer(None, batch, tokens, steps, kv_heads=kv_heads, ratio=ratio, sparsity=sparsity, bits=bits,
                      layout=layout, iterations=rng.choice((10, 10, 15)), theta=theta, sinks=rng.choice((0, 0, 4)))
    return _model(None, rng.randint(1, 4), spread(256, 1024), rng.randint(48, 72),
                  sparsity=rng.choice((0.5, 0.75)), bits=rng.choice((16, 4)))


# ---- what a program has in hand before the call ---------------------------------------------------------------------
def _frequencies(theta):
    return (theta ** (-torch.arange(64, device="cuda").float() / 64)).contiguous()


def _rotate(x, first, inv_freq):
    """Half-split RoPE of ``x[..., T, 128]`` at positions ``first, first + 1, ...``, as the model applies it."""
    out = torch.empty_like(x)
    angle = (first + torch.arange(x.shape[-2], device=x.device).float())[:, None] * inv_freq[None, :]
    cos, sin = angle.cos(), angle.sin()
    for i in range(x.shape[0]):  # one sequence at a time: the FP32 temporaries stay small
        lo, hi = x[i, ..., :64].float(), x[i, ..., 64:].float()
        out[i] = torch.cat((lo * cos - hi * sin, hi * cos + lo * sin), -1).to(x.dtype)
    return out


def _settings(case):
    return ResKVKernelConfig(sparsity=case["sparsity"], bits=case["bits"], layout=case.get("layout", "auto"),
                             num_clusters=case.get("clusters", 32), kmeans_iterations=case.get("iterations", 10),
                             recent_size=_RECENT, group_size=_GROUP)


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, 16 * seed)


def _prepare_decode(case, seed):
    b, h, t = case["batch"], case["kv_heads"], case["tokens"]
    inv_freq = _frequencies(case["theta"])
    cache = compress(mixture(b, h, t, seed=seed, device="cuda"), mixture(b, h, t, seed=seed + 1, device="cuda"), _settings(case))
    position = case["start"] + t + case["recent"] - 1
    query = gaussian(b, h * case["ratio"], 1, 128, seed=seed + 2, device="cuda")
    keys = mixture(b, h, case["recent"], seed=seed + 3, device="cuda")
    values = mixture(b, h, case["recent"], seed=seed + 4, device="cuda")
    # the window as a layer cache hands it out: the leading tokens of a longer buffer
    window = torch.zeros(2, b, h, _RECENT + _GROUP, 128, dtype=torch.float16, device="cuda")
    window[0, :, :, : case["recent"]] = _rotate(keys, position - case["recent"] + 1, inv_freq)
    window[1, :, :, : case["recent"]] = values
    recent = (_rotate(query, position, inv_freq), window[0, :, :, : case["recent"]], window[1, :, :, : case["recent"]])
    return {"kind": "decode", "query": query, "cache": cache, "recent": recent, "position": position,
            "start": case["start"], "inv_freq": inv_freq}


def _prepare_pack(case, seed):
    b, h, t = case["batch"], case["kv_heads"], case["tokens"]
    key, value = (mixture(b, h, t, seed=seed + i, device="cuda") for i in (0, 1))
    config = _settings(case)
    clustering = tuple(cluster(x, min(config.num_clusters, t), 3, value=i == 1) for i, x in enumerate((key, value)))
    return {"kind": "pack", "key": key, "value": value, "config": config, "clustering": clustering}


def _prepare_layer(case, seed):
    b, h, t, n = case["batch"], case["kv_heads"], case["tokens"], case["steps"]
    inv_freq = _frequencies(case["theta"])
    raw, value = (mixture(b, h, t + n, seed=seed + i, device="cuda") for i in (0, 1))
    query = gaussian(b, h * case["ratio"], n, 128, seed=seed + 2, device="cuda")
    steps = []
    rotated_query = _rotate(query, t, inv_freq)
    rotated = _rotate(raw, 0, inv_freq)
    for i in range(n):
        steps.append(tuple(x.contiguous() for x in (
            query[:, :, i : i + 1], rotated_query[:, :, i : i + 1], rotated[:, :, t + i : t + i + 1],
            raw[:, :, t + i : t + i + 1], value[:, :, t + i : t + i + 1])))
    prompt = tuple(x[:, :, :t].contiguous() for x in (rotated, raw, value))
    return {"kind": "layer", "config": _settings(case), "sinks": case["sinks"], "prompt": prompt, "steps": steps,
            "inv_freq": inv_freq}


_MODEL_SHAPE = dict(hidden=4096, heads=32, kv_heads=8, ffn=14336, vocab=32000)


def _prepare_model(case, seed):
    model = ResKVLlama(LlamaShape(layers=case["layers"], **_MODEL_SHAPE), _settings(case), seed=seed)
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    ids = torch.randint(128, _MODEL_SHAPE["vocab"], (case["batch"], case["tokens"] + case["steps"]), generator=gen, device="cuda")
    # the continuation is given, as when a known text is scored
    return {"kind": "model", "model": model, "prompt": ids[:, : case["tokens"]].contiguous(),
            "next": list(ids[:, case["tokens"] :].t().contiguous())}


_PREPARE = {"decode": _prepare_decode, "pack": _prepare_pack, "layer": _prepare_layer, "model": _prepare_model}


# ---- one pass -------------------------------------------------------------------------------------------------------
def run(state):
    return _RUN[state["kind"]](state)


def _run_decode(s):
    return attention(s["query"], s["cache"], position=s["position"], start_position=s["start"], inv_freq=s["inv_freq"],
                     recent=s["recent"])


def _run_pack(s):
    packed = compress(s["key"], s["value"], s["config"], clustering=s["clustering"])
    return {side: {name: getattr(tensor, name) for name in ("centroids", "cluster_ids", "payload", "metadata", "scale")}
            for side, tensor in (("key", packed.key), ("value", packed.value))}


def _run_layer(s):
    layer = ResKVLayerCache(s["config"], s["sinks"])
    rotated, raw, value = s["prompt"]
    layer.update(rotated, value, {"raw_keys": raw})
    out = []
    for query, rotated_query, key, raw_key, value in s["steps"]:
        position = layer.length
        keys, values = layer.update(key, value, {"raw_keys": raw_key})
        out.append(attention(query, layer.compressed, position=position, start_position=layer.start_position,
                             inv_freq=s["inv_freq"], recent=(rotated_query, keys, values)))
    # The packed rows are not among the outputs: which of two nearly equal residuals is kept, and with it the place of
    # every later value of the row, hangs on the last bit of a centroid.  What they hold shows in the attention results;
    # "pack" compares the rows themselves, on given centroids.
    return {"attention": torch.cat(out, 2), "key_centroids": layer.compressed.key.centroids,
            "value_centroids": layer.compressed.value.centroids, "window_keys": keys, "window_values": values}


def _run_model(s):
    model = s["model"]
    logits = [model.prefill(s["prompt"], reserve=len(s["next"]))]
    model.begin_graph_decode(s["prompt"].shape[0])
    for token in s["next"]:
        logits.append(model.decode_graph(token).clone())
    return torch.stack(logits, 1)


_RUN = {"decode": _run_decode, "pack": _run_pack, "layer": _run_layer, "model": _run_model}


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def _token_bytes(plan):
    """Bytes of one token and KV head, one side: id, payload row, metadata, scale."""
    spec = metadata_spec(plan)
    meta = 0 if spec is None else spec[0] * (8 if spec[1] == torch.int64 else 4)
    return 1 + payload_width(plan) * (2 if plan.bits == 16 else 4) + meta + (0 if plan.bits == 16 else 2)


def _attention_work(case, tokens, clusters, recent, heads, kv_heads):
    """One attention call: compressed rows, centroid tables, dense window, query (raw and rotated) and result once."""
    plan, b = _settings(case).resolve(case["batch"]), case["batch"]
    rows = b * kv_heads * (2 * tokens * _token_bytes(plan) + 2 * clusters * 256 + 2 * recent * 256)
    return rows + 3 * b * heads * 256, 4 * 128 * b * heads * (tokens + recent)


def _prefill_work(case, tokens, kv_heads):
    """Clustering and packing of a prompt: K and V read once, compressed rows and tables written once."""
    plan, b = _settings(case).resolve(case["batch"]), case["batch"]
    kept = max(0, tokens - _RECENT - case.get("sinks", 0)) // _GROUP * _GROUP
    moved = b * kv_heads * (2 * kept * (256 + _token_bytes(plan)) + 2 * 32 * 256 + 6 * (tokens - kept) * 256)
    # distances to every centre and the sums, each iteration
    return moved, b * kv_heads * 2 * kept * 128 * (2 * 32 + 2) * case.get("iterations", 10)


def _decode_steps_work(case, heads, kv_heads, steps):
    """``steps`` appended tokens after a prompt, each attending to everything before it."""
    t0, sinks = case["tokens"], case.get("sinks", 0)
    compressed = max(0, t0 - _RECENT - sinks) // _GROUP * _GROUP
    live, clusters, nbytes, flops = t0 - compressed, 32, 0, 0
    plan = _settings(case).resolve(case["batch"])
    for _ in range(steps):
        live += 1
        if live == sinks + _RECENT + _GROUP:
            compressed, live, clusters = compressed + _GROUP, live - _GROUP, min(64, clusters + 1)
            nbytes += case["batch"] * kv_heads * 2 * _GROUP * (256 + _token_bytes(plan))
        moved, done = _attention_work(case, compressed, clusters, live, heads, kv_heads)
        nbytes += moved + case["batch"] * kv_heads * 6 * 256
        flops += done
    return nbytes, flops


def work(case):
    kind, h = case["kind"], case.get("kv_heads", 8)
    if kind == "decode":
        nbytes, flops = _attention_work(case, case["tokens"], case["clusters"], case["recent"], h * case["ratio"], h)
    elif kind == "pack":
        plan, pairs = _settings(case).resolve(case["batch"]), case["batch"] * h * case["tokens"]
        nbytes = 2 * pairs * (256 + 4 + _token_bytes(plan)) + 2 * case["batch"] * h * case["clusters"] * 256
        flops = 2 * pairs * 128 * 2
    elif kind == "layer":
        first, steps = _prefill_work(case, case["tokens"], h), _decode_steps_work(case, h * case["ratio"], h, case["steps"])
        nbytes, flops = first[0] + steps[0], first[1] + steps[1]
    else:
        shape = LlamaShape(layers=case["layers"], **_MODEL_SHAPE)
        per_layer = shape.hidden * 128 * (2 * shape.heads + 2 * shape.kv_heads) + 3 * shape.hidden * shape.ffn
        head, prompt = shape.hidden * shape.vocab, case["batch"] * case["tokens"]
        first = _prefill_work(case, case["tokens"], h)
        steps = _decode_steps_work(case, shape.heads, h, case["steps"])
        causal = 2 * 128 * shape.heads * prompt * case["tokens"]
        nbytes = (1 + case["steps"]) * 2 * (shape.layers * per_layer + head) + shape.layers * (first[0] + steps[0])
        flops = (2 * (prompt + case["steps"] * case["batch"]) * shape.layers * per_layer +
                 2 * (1 + case["steps"]) * case["batch"] * head + shape.layers * (causal + first[1] + steps[1]))
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] == "pack":
        return "exact"  # given the centroids, the format fixes every bit
    if case["kind"] == "model":
        # FP16 activations between the layers, rounded at other places by another order of the same sums
        return {"rel": 5e-3, "max": 0.1}
    # FP16 results of FP16 probabilities (each rounded once) and FP32 sums.  A layer's clusters come from FP32 sums whose
    # order is free: a token between two centres may move, and with it what is kept of it.
    return {"rel": 2e-3, "max": 3e-2 if case["kind"] == "decode" else 0.1}
