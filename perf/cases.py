"""Timed cases of the sparse-attention path: what a sampler does with this package, over its range of sizes.

Kinds of work, each through the entry points a host program calls:

* ``layer``   ``B200SparseBackend.prepare`` + ``execute`` on device Q/K/V (the unprojected attention call)
* ``batch``   ``B200SparseBackend.forward`` on a batch
* ``replay``  one layer call recorded by ``B200SparseBackend.capture`` and replayed, as a sampler does step after step
* ``block``   the installed attention forward (``make_forward``): INT8 QKV projection with norm and rotation,
  router, attention, ``out_proj``
* ``mlp``     ``ChunkedFP8MLP`` behind the attention
* ``host``    ``B200SparseBackend.forward_host`` on pinned host activations (offloaded layers)

Geometry: 128-channel heads; ``text`` tokens, then ``video`` tokens, then ``tail`` tokens that are not video.  Only
video x video tiles are routed sparsely at the density ``budget``.
"""

import math
from types import SimpleNamespace

import torch

from h3_optimizations_b200 import B200SparseBackend, ChunkedSparseQKVProjector, HybridSparseConfig, runtime_options, workloads
from h3_optimizations_b200.attention_forward import make_forward
from h3_optimizations_b200.mlp import ChunkedFP8MLP

HEAD_DIM = 128
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
SIZES = {"bf16": 2, "fp16": 2, "fp32": 4}
RANK, GROUP = 8, 64  # of the structure the router finds in Q and K


def _layer(name, kind, heads, text, video, budget, dtype="bf16", tail=0, smooth_k=True, token_major=False, batch=1):
    return {"name": name, "kind": kind, "heads": heads, "text": text, "video": video, "tail": tail, "budget": budget,
            "dtype": dtype, "smooth_k": smooth_k, "token_major": token_major, "batch": batch}


def _block(name, heads, hidden, text, video, budget, tail=0, norm=True, rope="bf16", bias=False, smooth_k=True):
    return {"name": name, "kind": "block", "heads": heads, "hidden": hidden, "text": text, "video": video, "tail": tail,
            "budget": budget, "norm": norm, "rope": rope, "bias": bias, "smooth_k": smooth_k}


def _mlp(name, tokens, hidden, ffn, bias=True):
    return {"name": name, "kind": "mlp", "tokens": tokens, "hidden": hidden, "ffn": ffn, "bias": bias}


def listed():
    return [
        # a preview-size call, four heads: launches and host time are most of it
        _layer("layer_small", "layer", 4, 256, 2048, 0.3, dtype="fp32"),
        # one rank's share of the 24-head layer on eight GPUs, replayed step after step
        _layer("replay_rank", "replay", 3, 512, 32760, 0.3),
        # the benchmark layer: a 21x30x52 latent grid behind 512 text tokens
        _layer("layer_bench", "layer", 24, 512, 32760, 0.3),
        # a short clip with ragged ends, text on both sides of the video, strided views, half precision
        _layer("layer_ragged", "layer", 7, 300, 10007, 0.15, dtype="fp16", tail=77, token_major=True),
        # full density (the first and last steps of a cautious schedule): no router, every tile visited
        _layer("layer_dense", "layer", 24, 512, 9360, 1.0),
        # a long clip: a 21x60x60 latent grid
        _layer("layer_long", "layer", 24, 512, 75600, 0.3),
        # text + reference + audio context in front of the video, two prompts (conditional and not) in one batch
        _layer("batch_mixed", "batch", 24, 3072, 32760, 0.3, batch=2),
        # a whole attention block of a preview: projection, norm, rotation, attention, output projection
        _block("block_small", 24, 3072, 256, 2048, 0.3),
        # the same at the benchmark length
        _block("block_bench", 24, 3072, 512, 32760, 0.3),
        # the MLP of a short sequence (one chunk, ragged)
        _mlp("mlp_small", 1000, 3072, 12288),
        # the MLP of the benchmark length (nine chunks, the last one ragged)
        _mlp("mlp_bench", 33272, 3072, 12288),
        # a layer whose activations are kept in host memory: copies in, kernels and copies out overlapped
        _layer("host_offload", "host", 8, 512, 32760, 0.3),
    ]


def _spread(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """A case of the same ranges: 1 to 24 heads, clips of 700 to 75600 video tokens, densities of 10 to 100 %."""
    kind = rng.choice(["layer", "layer", "layer", "replay", "batch", "block", "block", "mlp", "mlp", "host"])
    if kind == "mlp":
        hidden = rng.choice([1024, 2048, 3072, 3072])
        case = _mlp("", _spread(rng, 64, 72000), hidden, 4 * hidden, bias=rng.random() < 0.5)
        del case["name"]
        return case
    text, tail = rng.randint(64, 1024), rng.choice([0, 0, 0, rng.randint(1, 512)])
    video = _spread(rng, 700, 33000 if kind in ("host", "block") else 75600)
    budget = rng.choice([0.1, 0.15, 0.2, 0.3, 0.3, 0.5, 1.0])
    heads = rng.choice([1, 3, 4, 6, 8, 12, 24, 24])
    smooth_k = rng.random() < 0.8
    if kind == "block":
        hidden = rng.choice([1024, 2048, 3072, 3072])
        norm = rng.random() < 0.8
        case = _block("", heads, hidden, text, video, budget, tail, norm=norm,
                      rope=rng.choice(["bf16", "fp32", "none"]) if norm else "none", bias=rng.random() < 0.3, smooth_k=smooth_k)
    else:
        case = _layer("", kind, heads, text, video, budget, dtype=rng.choice(["bf16", "bf16", "fp16", "fp32"]), tail=tail,
                      smooth_k=smooth_k, token_major=kind == "layer" and rng.random() < 0.5,
                      batch=2 if kind == "batch" else 1)
    # no dearer than half the longest listed layer; host activations stay under 150 MB each
    limit = 0.5 * _pairs(_layer("", "layer", 24, 512, 75600, 0.3))
    while case["heads"] > 1 and (_pairs(case) > limit or (kind == "host" and _elements(case) > 36_000_000)):
        case["heads"] //= 2
    if _pairs(case) > limit:
        case["budget"] = 0.3
    del case["name"]
    return case


# -- inputs ---------------------------------------------------------------------


def _sequence(case):
    return case["text"] + case["video"] + case["tail"]


def _elements(case):
    return case.get("batch", 1) * case["heads"] * _sequence(case) * HEAD_DIM


def _pairs(case):
    """(query, key) pairs the route visits, all heads and batch elements."""
    sequence, start, stop = _sequence(case), case["text"], case["text"] + case["video"]
    last = stop == sequence
    q_tiles, kv_tiles = -(-sequence // 128), -(-sequence // 64)
    q0, q1 = -(-start // 128), q_tiles if last else stop // 128
    k0, k1 = -(-start // 64), kv_tiles if last else stop // 64
    retained = min(k1 - k0, max(1, math.ceil(case["budget"] * (k1 - k0))))
    routed_rows = min(q1 * 128, sequence) - q0 * 128
    keys = min(sequence, (kv_tiles - (k1 - k0) + retained) * 64)
    return case.get("batch", 1) * case["heads"] * ((sequence - routed_rows) * sequence + routed_rows * keys)


def _options(case):
    text, video, tail = case["text"], case["video"], case["tail"]
    segments = [("text", text), ("video", video)] + ([("text", tail)] if tail else [])
    spec = workloads.SequenceSpec("case", case["heads"], workloads._segments(*segments), (1, 1, video))
    return runtime_options(spec.layout(), step_index=5, total_steps=30)


def _qkv(case, gen):
    """Q and K: unit Gaussians plus a rank-8 component per head that is held over 64-token groups, so that tile
    means carry signal; V: unit Gaussian.  ``token_major``: views of (S, H, 128), as a model's own projection hands over."""
    batch, heads, sequence = case["batch"], case["heads"], _sequence(case)
    groups = -(-sequence // GROUP)
    out = []
    for name in "qkv":
        x = torch.randn((batch, heads, sequence, HEAD_DIM), generator=gen, device="cuda")
        if name != "v":
            basis = torch.randn((batch, heads, RANK, HEAD_DIM), generator=gen, device="cuda")
            coeff = torch.randn((batch, heads, groups, RANK), generator=gen, device="cuda") * 0.5
            x += (coeff @ basis).repeat_interleave(GROUP, dim=2)[:, :, :sequence]
        x = x.to(DTYPES[case["dtype"]])
        out.append(x.transpose(1, 2).contiguous().transpose(1, 2) if case["token_major"] else x)
    return out


def _backend(case):
    return B200SparseBackend(HybridSparseConfig(video_budget=case["budget"]), smooth_k=case["smooth_k"])


def _rope(sequence, dtype, gen):
    """(1, S, 1, 48, 2, 2) rotation matrices of positions with a random start."""
    start = torch.randint(0, 1000, (1,), generator=gen, device="cuda")
    position = (start + torch.arange(sequence, device="cuda")).float()
    angle = position[:, None] * torch.exp(torch.arange(48, device="cuda") * (-math.log(10000.0) / 48))
    table = torch.stack([angle.cos(), -angle.sin(), angle.sin(), angle.cos()], dim=-1)
    return table.view(1, sequence, 1, 48, 2, 2).to(DTYPES[dtype]).contiguous()


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    if case["kind"] == "mlp":
        hidden, ffn = case["hidden"], case["ffn"]
        weight = [torch.randn(shape, generator=gen, device="cuda") * 0.02 for shape in ((ffn, hidden), (hidden, ffn))]
        bias = [torch.randn(n, generator=gen, device="cuda") * 0.02 if case["bias"] else None for n in (ffn, hidden)]
        x = torch.randn((case["tokens"], hidden), generator=gen, device="cuda").to(torch.bfloat16)
        return {"kind": "mlp", "mlp": ChunkedFP8MLP(weight[0], bias[0], weight[1], bias[1]), "x": x}
    options = _options(case)
    if case["kind"] == "block":
        heads, hidden, sequence = case["heads"], case["hidden"], _sequence(case)
        rows = 3 * heads * HEAD_DIM
        norm = lambda: SimpleNamespace(
            weight=(1.0 + 0.1 * torch.randn(HEAD_DIM, generator=gen, device="cuda")).to(torch.bfloat16), eps=1e-6)
        out_proj = torch.nn.Linear(heads * HEAD_DIM, hidden, bias=case["bias"], device="cuda", dtype=torch.bfloat16)
        out_proj.weight.data.copy_(torch.randn((hidden, heads * HEAD_DIM), generator=gen, device="cuda") * 0.02)
        if case["bias"]:
            out_proj.bias.data.copy_(torch.randn(hidden, generator=gen, device="cuda") * 0.02)
        module = SimpleNamespace(
            heads=heads, head_dim=HEAD_DIM, out_proj=out_proj,
            qkv_weight_int8=torch.randint(-127, 128, (rows, hidden), generator=gen, device="cuda", dtype=torch.int8),
            qkv_weight_scale=torch.full((rows,), 1.0 / (127.0 * math.sqrt(hidden)), device="cuda"))
        if case["norm"]:
            module.q_norm, module.k_norm = norm(), norm()
        x = torch.randn((sequence, hidden), generator=gen, device="cuda")
        # tokens of one group resemble one another, so that the router has something to find
        x += torch.randn((-(-sequence // GROUP), hidden), generator=gen, device="cuda").repeat_interleave(GROUP, dim=0)[:sequence]
        forward = make_forward(module, 0, backend=_backend(case), projector=ChunkedSparseQKVProjector(smooth_k=case["smooth_k"]))
        rope = None if case["rope"] == "none" else _rope(sequence, case["rope"], gen)
        return {"kind": "block", "forward": forward, "x": x.to(torch.bfloat16), "rope": rope, "options": options}
    q, k, v = _qkv(case, gen)
    backend = _backend(case)
    if case["kind"] == "replay":
        return {"kind": "replay", "call": backend.capture(q, k, v, layer_index=0, transformer_options=options), "qkv": (q, k, v)}
    if case["kind"] == "host":
        q, k, v = (t.cpu().pin_memory() for t in (q, k, v))
        return {"kind": "host", "backend": backend, "qkv": (q, k, v), "out": torch.empty_like(q).pin_memory(), "options": options}
    return {"kind": case["kind"], "backend": backend, "qkv": (q, k, v), "options": options}


def run(state):
    kind = state["kind"]
    if kind == "mlp":
        return state["mlp"](state["x"])
    if kind == "replay":
        return state["call"].replay()
    if kind == "block":
        with torch.no_grad():
            return state["forward"](state["x"], state["rope"], state["options"])
    backend, options = state["backend"], state["options"]
    q, k, v = state["qkv"]
    if kind == "batch":
        return backend.forward(q, k, v, layer_index=0, transformer_options=options)
    if kind == "host":
        return backend.forward_host(q, k, v, state["out"], layer_index=0, transformer_options=options)
    return backend.execute(backend.prepare(q, k, v, layer_index=0, transformer_options=options))


def work(case):
    if case["kind"] == "mlp":
        tokens, hidden, ffn = case["tokens"], case["hidden"], case["ffn"]
        return {"bytes": 2 * 2 * tokens * hidden + 2 * hidden * ffn, "flops": 4 * tokens * hidden * ffn}
    attention = 4 * HEAD_DIM * _pairs(case)
    if case["kind"] != "block":
        return {"bytes": 4 * _elements(case) * SIZES[case["dtype"]], "flops": attention}
    sequence, hidden, inner = _sequence(case), case["hidden"], case["heads"] * HEAD_DIM
    table = 0 if case["rope"] == "none" else sequence * 48 * 4 * SIZES[case["rope"]]
    return {"bytes": 2 * 2 * sequence * hidden + 3 * inner * hidden + 2 * inner * hidden + table,
            "flops": attention + 2 * sequence * hidden * 3 * inner + 2 * sequence * inner * hidden}


def tolerance(case):
    # bf16 results: half a unit in the last place is 2e-3 of a value.  fp16 and fp32 results carry the rounding of the
    # probabilities in front of the 8-bit P.V product, about seven significant bits.
    if case.get("dtype", "bf16") == "bf16":
        return {"rel": 1e-2}
    return {"rel": 5e-3}
