"""The work that a user of this package has it do, as cases that can be timed and compared.

Four kinds, all through the public modules of ``nano_qwen_b200.layers``:

``decode``   one decode step of some decoder layers' linear path from a CUDA graph captured beforehand, as a model
             runner replays it: add + norm -> qkv, o_proj on the attention's output, add + norm -> gate_up ->
             SiLU * up -> down (norms and activation hand the linears FP8, o_proj quantises its input itself)
``prefill``  the same layers called eagerly on the tokens of one or more prompts
``linear``   one replicated linear layer with bias on bf16 activations, called eagerly, ragged sizes
``load``     a bf16 checkpoint's gate and up matrices given to the merged layer's loader, which quantises them

Attention itself is not part of this package: its output is an input here, and qkv is an output.
"""
from __future__ import annotations

import math

import torch
import torch.distributed as dist

# hidden size, query heads, kv heads, MLP width of one layer; head size 128.  The last two are what one rank holds of
# the 8B- and 32B-shaped layers when they are split over 2 and 4 ranks.
MODELS = {
    "0.6b": (1024, 16, 8, 3072),
    "8b": (4096, 32, 8, 12288),
    "32b": (5120, 64, 8, 25600),
    "8b/2": (4096, 16, 4, 6144),
    "32b/4": (5120, 16, 2, 6400),
}
HEAD = 128
MAX_DECODE, MAX_PREFILL = 512, 8192
MAX_FLOPS = 2 * 8192 * 192_937_984          # the largest listed case: 8192 tokens through one 8B-shaped layer
MAX_WEIGHTS = 1_500_000_000                 # weight elements that a case keeps on the GPU


def listed() -> list[dict]:
    return [
        # a short prompt through a small model: nothing but latency, launches and host work
        {"name": "prefill_7_small_model", "kind": "prefill", "model": "0.6b", "layers": 4, "tokens": 7, "gemma": False},
        # one user's chat: the weights stream once per token
        {"name": "decode_1", "kind": "decode", "model": "8b", "layers": 4, "tokens": 1, "gemma": False},
        # a handful of users on one rank's part of a larger model
        {"name": "decode_8_shard", "kind": "decode", "model": "32b/4", "layers": 4, "tokens": 8, "gemma": True},
        # batched serving, from few users to the largest batch that a runner captures
        {"name": "decode_32", "kind": "decode", "model": "8b", "layers": 3, "tokens": 32, "gemma": False},
        {"name": "decode_144", "kind": "decode", "model": "8b", "layers": 3, "tokens": 144, "gemma": False},
        {"name": "decode_256", "kind": "decode", "model": "8b", "layers": 3, "tokens": 256, "gemma": False},
        {"name": "decode_512_shard", "kind": "decode", "model": "8b/2", "layers": 3, "tokens": 512, "gemma": False},
        # an ordinary prompt, its length as it comes
        {"name": "prefill_777", "kind": "prefill", "model": "8b", "layers": 2, "tokens": 777, "gemma": False},
        # several prompts in one batch through the largest layers
        {"name": "prefill_3001_large_model", "kind": "prefill", "model": "32b", "layers": 1, "tokens": 3001, "gemma": True},
        # a full prefill chunk
        {"name": "prefill_8192", "kind": "prefill", "model": "8b", "layers": 1, "tokens": 8192, "gemma": False},
        # a layer outside the big four: sizes that are no multiples of a tile or of a scale group
        {"name": "linear_ragged_bias", "kind": "linear", "tokens": 301, "n": 1320, "k": 1096},
        # loading an unquantised checkpoint
        {"name": "load_bf16", "kind": "load", "n": 12288, "k": 4096},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng) -> dict:
    kind = rng.choices(("decode", "prefill", "linear", "load"), (45, 35, 12, 8))[0]
    if kind == "linear":
        return {"kind": kind, "tokens": _log_int(rng, 1, 4096), "n": 8 * _log_int(rng, 8, 1024), "k": 8 * _log_int(rng, 8, 1024)}
    if kind == "load":
        return {"kind": kind, "n": 128 * _log_int(rng, 8, 200), "k": 16 * _log_int(rng, 64, 512)}
    model = rng.choice(sorted(MODELS))
    tokens = _log_int(rng, 1, MAX_DECODE if kind == "decode" else MAX_PREFILL)
    per_layer = sum(n * k for n, k in _shapes(model).values())
    tokens = min(tokens, MAX_FLOPS // (2 * per_layer))
    layers = max(1, min(rng.randint(1, 4), MAX_WEIGHTS // per_layer, MAX_FLOPS // (2 * per_layer * tokens)))
    return {"kind": kind, "model": model, "layers": layers, "tokens": tokens, "gemma": rng.random() < 0.5}


def _shapes(model: str) -> dict[str, tuple[int, int]]:
    """(N, K) of the four linear layers."""
    hidden, heads, kv, inter = MODELS[model]
    return {"qkv": ((heads + 2 * kv) * HEAD, hidden), "o": (hidden, heads * HEAD), "gate_up": (2 * inter, hidden), "down": (hidden, inter)}


class Layer(torch.nn.Module):
    """A decoder layer without its attention."""

    def __init__(self, model: str, gemma: bool):
        from nano_qwen_b200 import layers as L
        super().__init__()
        hidden, heads, kv, inter = MODELS[model]
        norm = L.GemmaRMSNorm if gemma else L.RMSNorm
        self.input_layernorm = norm(hidden, emit_fp8=True)
        self.qkv_proj = L.QKVParallelLinear(hidden, HEAD, heads, kv)
        self.o_proj = L.RowParallelLinear(heads * HEAD, hidden)
        self.post_attention_layernorm = norm(hidden, emit_fp8=True)
        self.gate_up_proj = L.MergedColumnParallelLinear(hidden, [inter, inter])
        self.act_fn = L.SiluAndMul()
        self.down_proj = L.RowParallelLinear(inter, hidden)

    def forward(self, hidden, residual, attention_output):
        hidden, residual = self.input_layernorm(hidden, residual)
        qkv = self.qkv_proj(hidden)
        hidden = self.o_proj(attention_output)
        hidden, residual = self.post_attention_layernorm(hidden, residual)
        hidden = self.down_proj(self.act_fn(self.gate_up_proj(hidden)))
        return hidden, residual, qkv


def _build(make):
    """Constructs modules as a model runner does: on the GPU, bf16 by default, inside a process group."""
    if not dist.is_initialized():
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)
    old = torch.get_default_dtype()
    torch.set_default_dtype(torch.bfloat16)
    try:
        with torch.device("cuda"):
            return make()
    finally:
        torch.set_default_dtype(old)


def _normal(gen, *shape, scale=1.0):
    return torch.randn(*shape, generator=gen, device="cuda", dtype=torch.bfloat16).mul_(scale)


def _forward(layers, hidden, residual, attention):
    qkvs = []
    for layer, a in zip(layers, attention):
        hidden, residual, qkv = layer(hidden, residual, a)
        qkvs.append(qkv)
    return hidden, residual, qkvs


@torch.inference_mode()
def prepare(case: dict, seed: int) -> dict:
    from nano_qwen_b200 import layers as L
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "linear":
        layer = _build(lambda: L.ReplicatedLinear(case["k"], case["n"], bias=True))
        layer.weight.weight_loader(layer.weight, _normal(gen, case["n"], case["k"], scale=0.02))
        layer.bias.weight_loader(layer.bias, _normal(gen, case["n"], scale=0.02))
        return {"kind": kind, "layer": layer, "x": _normal(gen, case["tokens"], case["k"])}
    if kind == "load":
        layer = _build(lambda: L.MergedColumnParallelLinear(case["k"], [case["n"], case["n"]]))
        return {"kind": kind, "layer": layer, "parts": [_normal(gen, case["n"], case["k"], scale=0.02) for _ in range(2)]}
    hidden, heads, _, _ = MODELS[case["model"]]
    tokens = case["tokens"]
    layers = []
    for _ in range(case["layers"]):
        layer = _build(lambda: Layer(case["model"], case["gemma"]))
        for name, (n, k) in _shapes(case["model"]).items():
            weight = getattr(layer, name + "_proj").weight
            w = _normal(gen, n, k, scale=0.02)
            parts = {"qkv": "qkv", "gate_up": (0, 1)}.get(name)
            if parts is None:
                weight.weight_loader(weight, w)
                continue
            kv = MODELS[case["model"]][2] * HEAD
            rows = (n - 2 * kv, kv, kv) if name == "qkv" else (n // 2, n // 2)
            for part, piece in zip(parts, w.split(rows)):
                weight.weight_loader(weight, piece, part)
        for norm in (layer.input_layernorm, layer.post_attention_layernorm):
            norm.weight.data.add_(_normal(gen, hidden, scale=0.1))
        layers.append(layer)
    args = (layers, _normal(gen, tokens, hidden), _normal(gen, tokens, hidden),
            [_normal(gen, tokens, heads * HEAD) for _ in range(case["layers"])])
    if kind == "prefill":
        return {"kind": kind, "args": args}
    _forward(*args)                                     # what a runner does before it captures
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outputs = _forward(*args)
    return {"kind": kind, "args": args, "graph": graph, "outputs": outputs}


@torch.inference_mode()
def run(state: dict):
    kind = state["kind"]
    if kind == "decode":
        state["graph"].replay()
        return state["outputs"]
    if kind == "prefill":
        return _forward(*state["args"])
    layer = state["layer"]
    if kind == "linear":
        return layer(state["x"])
    for part, w in enumerate(state["parts"]):
        layer.weight.weight_loader(layer.weight, w, part)
    return layer.weight.data.view(torch.uint8), layer.weight_scale_inv.data


def work(case: dict) -> dict:
    """Weights (e4m3 + one fp32 scale per 128 x 128), the path's inputs and its outputs, each once."""
    def stored(n, k):
        return n * k + 4 * (-(-n // 128)) * (-(-k // 128))
    if case["kind"] == "load":
        return {"bytes": 2 * (2 * case["n"] * case["k"] + stored(case["n"], case["k"])), "flops": 0}
    tokens = case["tokens"]
    if case["kind"] == "linear":
        n, k = case["n"], case["k"]
        return {"bytes": stored(n, k) + 2 * n + 2 * tokens * (n + k), "flops": 2 * tokens * n * k}
    hidden = MODELS[case["model"]][0]
    shapes = _shapes(case["model"])
    layer = sum(stored(*s) for s in shapes.values()) + 4 * hidden + 2 * tokens * (shapes["qkv"][0] + shapes["o"][1])
    return {"bytes": case["layers"] * layer + 2 * tokens * hidden * 4, "flops": case["layers"] * 2 * tokens * sum(n * k for n, k in shapes.values())}


def tolerance(case: dict):
    if case["kind"] == "load":
        return "exact"                                  # bytes and scales are fixed by the format's rule
    if case["kind"] == "linear":
        return {"rel": 4e-3}                            # bf16 results (2^-9) of sums in another order
    # an intermediate bf16 that rounds the other way can move an e4m3 value by one step (2^-4) in the next layer
    return {"rel": 1e-2}
