"""The work this engine is measured by: whole steps, layers, token mixers and the sampler, each
through the entry point a program calls.

Kinds of cases (``"kind"``):

* ``step``   - ``ModelRunner.step``: requests that decode one token each, alone or beside a portion
               of a new prompt; logits of every entry's last token.
* ``layer``  - one decoder block (attention, feed-forward, both norms) on a prompt portion, alone or
               beside decoding requests, and the norm that follows it.
* ``delta``, ``gated``, ``latent`` - the token mixer of a layer of another design on prompt portions:
               gated delta rule, gated linear recurrence, attention over cached latents.
* ``routed`` - a routed feed-forward.
* ``sample`` - ``Sampler.sample`` over a step's logits.

Weights, inputs and cached contexts are drawn on the device from the seed.  ``exact`` restates each
path in 64 bits with dense tensors; it uses nothing of the engine.
"""

from __future__ import annotations

import math
import zlib

import torch

from forge_engine_b200.config.registry import read_model_config
from forge_engine_b200.engine import ModelRunner, StepEntry
from forge_engine_b200.engine.batch import build_batch
from forge_engine_b200.sampling.params import SamplingParams
from forge_engine_b200.sampling.sampler import Sampler

PAGE = 16
ROOM = 64                 # tokens a request decodes before it ends and another takes its place
DEVICE = "cuda:0"
EPS = 1e-6
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}


def listed() -> list:
    full = {"width": 2560, "inter": 9728, "heads": 32, "kv_heads": 8, "dim": 128}
    small = {"width": 1024, "inter": 3072, "heads": 16, "kv_heads": 8, "dim": 128}
    return [
        # one user waiting for each token: latency of a step that streams the weights once
        {"name": "decode-1", "kind": "step", "dtype": "bf16", **full, "layers": 12, "vocab": 151936,
         "decoders": 1, "context": 2048, "portion": 0},
        # a busy server between prompts: 48 requests whose contexts differ by a factor of four
        {"name": "decode-48-ragged", "kind": "step", "dtype": "bf16", **full, "layers": 8, "vocab": 151936,
         "decoders": 48, "context": 3001, "portion": 0},
        # the scheduler's everyday step: a prompt portion fills the token budget beside decoding requests
        {"name": "mixed-256", "kind": "step", "dtype": "bf16", **full, "layers": 8, "vocab": 151936,
         "decoders": 8, "context": 2048, "portion": 248},
        # a layer of a whole 2,048-token prompt (the default token budget's largest step)
        {"name": "prompt-2048", "kind": "layer", "dtype": "bf16", **full, "decoders": 0, "context": 0,
         "portion": 2048, "cached": 0},
        # a later portion of a long document: few rows of an odd count, many cached keys
        {"name": "prompt-continued", "kind": "layer", "dtype": "bf16", **full, "decoders": 4, "context": 1500,
         "portion": 1021, "cached": 12288},
        # the true 32-bit engine reading a prompt
        {"name": "f32-prompt", "kind": "layer", "dtype": "f32", **small, "decoders": 0, "context": 0,
         "portion": 500, "cached": 0},
        # the true 32-bit engine decoding, head and all
        {"name": "f32-decode", "kind": "step", "dtype": "f32", **small, "layers": 4, "vocab": 32000,
         "decoders": 4, "context": 700, "portion": 0},
        # a gated delta rule's prompt
        {"name": "delta-prompt", "kind": "delta", "width": 2560, "heads": 32, "kv_heads": 16, "dim": 64, "vdim": 64,
         "conv": 4, "requests": 1, "tokens": 2048},
        # several users' prompts of different lengths through a gated linear recurrence with wide states
        {"name": "gated-prompts", "kind": "gated", "width": 4096, "heads": 32, "dim": 128, "vdim": 128,
         "requests": 3, "tokens": 1000},
        # a prompt over cached latents
        {"name": "latent-prompt", "kind": "latent", "width": 2560, "heads": 32, "dim": 64, "rot_dim": 32, "vdim": 64,
         "q_rank": 768, "kv_rank": 256, "portion": 1500, "cached": 500},
        # a routed feed-forward of a mixed step
        {"name": "routed-700", "kind": "routed", "width": 2560, "ff": 4864, "experts": 16, "top": 2, "rows": 700},
        # sampling for a batch of users with the usual filters
        {"name": "sample-16", "kind": "sample", "rows": 16, "vocab": 151936, "temperature": 0.8, "top_k": 50,
         "top_p": 0.95, "min_p": 0.0},
    ]


SHAPES = (
    {"width": 1024, "inter": 3072, "heads": 16, "kv_heads": 8, "dim": 128},
    {"width": 2560, "inter": 9728, "heads": 32, "kv_heads": 8, "dim": 128},
    {"width": 4096, "inter": 12288, "heads": 32, "kv_heads": 8, "dim": 128},
)


def _spread(rng, low: int, high: int) -> int:
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def _cost(case: dict) -> float:
    need = work(case)
    return max(need["bytes"], need["flops"] / 50)


def draw(rng) -> dict:
    """One more case of the listed ones' ranges that costs no more than the largest of them."""
    most = max(_cost(case) for case in listed())
    while True:
        case = _drawn(rng)
        if _cost(case) <= most:
            return case


def _drawn(rng) -> dict:
    kind = rng.choice(("step", "step", "step", "layer", "layer", "layer", "delta", "gated", "latent", "routed", "sample"))
    if kind == "step":
        if rng.random() < 0.3:
            return {"kind": kind, "dtype": "f32", **SHAPES[0], "layers": rng.randint(2, 6), "vocab": 32000,
                    "decoders": _spread(rng, 1, 16), "context": _spread(rng, 32, 1500),
                    "portion": rng.choice((0, 0, rng.randint(5, 120)))}
        decoders = _spread(rng, 1, 64)
        return {"kind": kind, "dtype": "bf16", **rng.choice(SHAPES), "layers": rng.randint(2, 8), "vocab": 32000,
                "decoders": decoders, "context": _spread(rng, 64, min(16384, 131072 // decoders)),
                "portion": rng.choice((0, rng.randint(20, 440)))}
    if kind == "layer":
        if rng.random() < 0.3:
            return {"kind": kind, "dtype": "f32", **SHAPES[0], "decoders": rng.choice((0, rng.randint(1, 8))),
                    "context": rng.randint(16, 900), "portion": _spread(rng, 33, 700),
                    "cached": rng.choice((0, rng.randint(1, 900)))}
        return {"kind": kind, "dtype": "bf16", **rng.choice(SHAPES), "decoders": rng.choice((0, rng.randint(1, 24))),
                "context": rng.randint(16, 4000), "portion": _spread(rng, 65, 2048),
                "cached": rng.choice((0, rng.randint(1, 12288)))}
    if kind in ("delta", "gated"):
        requests = rng.choice((1, 1, 2, 3, 5))
        size = rng.choice((64, 128))
        case = {"kind": kind, "width": 2560 if size == 64 else 4096, "heads": 32, "dim": size, "vdim": size,
                "requests": requests, "tokens": _spread(rng, 100, 2048 // requests)}
        return dict(case, kv_heads=rng.choice((16, 32)), conv=4) if kind == "delta" else case
    if kind == "latent":
        sizes = rng.choice(((2560, 64, 32, 64, 768, 256), (4096, 128, 64, 128, 1536, 512)))
        names = ("width", "dim", "rot_dim", "vdim", "q_rank", "kv_rank")
        return {"kind": kind, **dict(zip(names, sizes)), "heads": 32, "portion": _spread(rng, 65, 1024),
                "cached": rng.choice((0, rng.randint(1, 2000)))}
    if kind == "routed":
        return {"kind": kind, "width": 2560, "ff": rng.choice((2432, 4864)), "experts": 16, "top": rng.choice((1, 2, 4)),
                "rows": _spread(rng, 4, 1024)}
    return {"kind": kind, "rows": _spread(rng, 1, 64), "vocab": rng.choice((32000, 128256, 151936)),
            "temperature": rng.choice((0.0, 0.7, 1.0)), "top_k": rng.choice((0, 20, 200)), "top_p": rng.choice((1.0, 0.9)),
            "min_p": rng.choice((0.0, 0.05))}


# -- inputs ------------------------------------------------------------------------------------
def _noise(seed: int, name: str, shape, dtype=torch.float32, scale: float = 1.0, shift: float = 0.0) -> torch.Tensor:
    """Normal numbers of this seed and name, rounded once to ``dtype``."""
    gen = torch.Generator(device=DEVICE).manual_seed((seed * 1_000_003 + zlib.crc32(name.encode())) & 0x7FFFFFFFFFFF)
    return torch.randn(tuple(shape), generator=gen, device=DEVICE).mul_(scale).add_(shift).to(dtype)


def _weight(seed: int, name: str, shape, dtype) -> torch.Tensor:
    """A tensor of a checkpoint: matrices keep activations at order one, norm weights lie round one,
    gates, decays and taps spread over their ranges."""
    last = name.rsplit(".", 1)[-1]
    if "norm" in name and len(shape) == 1:
        return _noise(seed, name, shape, dtype, 0.1, 1.0)
    if last == "conv":
        return _noise(seed, name, shape, dtype, 0.5)
    if last == "A_log":
        return _noise(seed, name, shape, dtype, 0.7, -1.0)
    if last == "lower":
        return torch.sigmoid(_noise(seed, name, shape)).mul_(0.9).to(dtype)
    if len(shape) == 1:
        return _noise(seed, name, shape, dtype, 0.5)
    if name in ("model.embed_tokens.weight", "embed"):
        return _noise(seed, name, shape, dtype, 0.02)
    return _noise(seed, name, shape, dtype, shape[-1] ** -0.5)


class _Weights(dict):
    """Checkpoint tensors by name, drawn when the model asks for them and not kept."""

    def __init__(self, expected: dict, seed: int, dtype) -> None:
        super().__init__(expected)
        self.seed, self.dtype = seed, dtype

    def __getitem__(self, name):
        return _weight(self.seed, name, super().__getitem__(name).shape, self.dtype)


def _config(case: dict) -> dict:
    """The config.json of the model a case's part comes from (one layer for parts)."""
    kind = case["kind"]
    if kind in ("step", "layer"):
        return {"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "hidden_act": "silu",
                "vocab_size": case.get("vocab", 64), "hidden_size": case["width"], "intermediate_size": case["inter"],
                "num_hidden_layers": case.get("layers", 1), "num_attention_heads": case["heads"],
                "num_key_value_heads": case["kv_heads"], "head_dim": case["dim"], "max_position_embeddings": 32768,
                "rms_norm_eps": EPS, "rope_theta": 1000000.0, "tie_word_embeddings": True, "attention_bias": False}
    base = {"vocab": 64, "width": case["width"], "norm": {"eps": EPS}}
    mixer = {k: case[k] for k in ("heads", "kv_heads", "dim", "vdim", "conv", "rot_dim", "q_rank", "kv_rank") if k in case}
    if kind == "delta":
        return {"architecture": "Lofuvik", **base, "layers": [{"type": "delta", "mixer": mixer}]}
    if kind == "gated":
        return {"architecture": "Zabutar", **base, "canon": {"taps": 4}, "max_positions": 32768,
                "layers": [{"type": "hgrn2", "mixer": mixer}]}
    if kind == "latent":
        mixer.update(rot={"base": 1e6, "dims": case["rot_dim"]}, scale=(case["dim"] + case["rot_dim"]) ** -0.5)
        return {"architecture": "Zofadra", **base, "layers": [{"type": "latent_attention", "mixer": mixer}]}
    routed = {"kind": "moe", "expert": {"ff": case["ff"]}, "router": {"experts": case["experts"], "top": case["top"]}}
    return {"architecture": "Lofuvik", **base, "layers": [{"type": "delta", "mlp": routed, "mixer": {
        "heads": 2, "dim": 16, "vdim": 16, "conv": 2}}]}


def _contexts(case: dict) -> list:
    """Tokens already cached, per decoding request: from a quarter of ``context`` up to all of it."""
    count, top = case["decoders"], case["context"]
    return [top] * count if count < 2 else [max(1, top * (count - 1 + 3 * i) // (4 * (count - 1))) for i in range(count)]


def _prompts(case: dict) -> list:
    """Lengths of the prompts of a recurrence case: the longest first, each a sixth shorter."""
    return [max(1, case["tokens"] * (6 - i) // 6) for i in range(case["requests"])]


def _cached(case: dict, seed: int, layer: int, side: str, request: int, length: int, shape: tuple) -> torch.Tensor:
    """What layer ``layer`` holds of a request's first ``length`` tokens: [length, *shape]."""
    return _noise(seed, f"cache.{layer}.{side}.{request}", (length, *shape), DTYPES[case.get("dtype", "bf16")])


def _fill(cache, key, case, seed, request, length, shape, layers) -> None:
    """Begin a request whose first ``length`` tokens are already cached."""
    cache.begin_request(key)
    if not length:
        return
    cache.reserve(key, length)
    cache.advance(key, length)
    pages = torch.tensor(cache.request(key).tables[0].pages[: -(-length // PAGE)], device=DEVICE)
    for layer in range(layers):
        for side, store in zip("kv", cache.kv_of_run(layer)):
            if store is None:
                continue
            rows = _cached(case, seed, layer, side, request, length, shape)
            whole = torch.zeros((len(pages) * PAGE, *shape), dtype=rows.dtype, device=DEVICE)
            whole[:length] = rows
            store[pages] = whole.view(len(pages), PAGE, *shape).transpose(1, 2)


def _runner(case: dict, seed: int, pages: int, requests: int) -> ModelRunner:
    arch, _, spec = read_model_config(_config(case))
    dtype = DTYPES[case.get("dtype", "bf16")]
    return ModelRunner.from_tensors(spec, _Weights(arch.expected_tensors(spec), seed, dtype), dtype=dtype, device=DEVICE,
                                    page_size=PAGE, num_pages=pages, max_requests=requests, architecture=arch)


def _tokens(case: dict, seed: int, name: str, count: int) -> list:
    gen = torch.Generator().manual_seed(seed * 7919 + zlib.crc32(name.encode()))
    return torch.randint(0, case["vocab"], (count,), generator=gen).tolist()


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "sample":
        params = SamplingParams(temperature=case["temperature"], top_k=case["top_k"] or None, top_p=case["top_p"],
                                min_p=case["min_p"])
        # logits of a language model: a broad bulk and a few tokens well above it
        logits = _noise(seed, "logits", (case["rows"], case["vocab"]), scale=2.0)
        logits.scatter_add_(1, torch.arange(1, 41, device=DEVICE).repeat(case["rows"], 1) * (case["vocab"] // 41),
                            _noise(seed, "peaks", (case["rows"], 40), scale=2.0, shift=8.0))
        return {"kind": kind, "sampler": Sampler(DEVICE, torch.zeros(1, dtype=torch.int32, device=DEVICE)), "logits": logits,
                "params": [params] * case["rows"], "seeds": [seed * 1009 + i for i in range(case["rows"])],
                "counters": list(range(5, 5 + case["rows"]))}
    if kind == "routed":
        runner = _runner(case, seed, 8, 1)
        return {"kind": kind, "ffn": runner.model.blocks[0].ffn, "x": _noise(seed, "x", (case["rows"], case["width"]), torch.bfloat16)}
    if kind in ("delta", "gated"):
        lengths = _prompts(case)
        runner = _runner(case, seed, 8 + sum(-(-n // PAGE) for n in lengths), len(lengths))
        entries = [StepEntry(f"r{i}", [0] * n) for i, n in enumerate(lengths)]
        for entry in entries:
            runner.begin(entry.key)
        view = runner.cache.view(0)
        return {"kind": kind, "runner": runner, "mixer": runner.model.blocks[0].mixer, "cache": view,
                "batch": build_batch(entries, runner.cache, DEVICE), "x": _noise(seed, "x", (sum(lengths), case["width"]), torch.bfloat16),
                "states": [view.state[runner.cache.request(e.key).slot] for e in entries]}
    contexts = _contexts(case) if "decoders" in case else []
    portion, cached = case["portion"], case.get("cached", 0)
    layers = case.get("layers", 1)
    pages = sum(-(-(c + ROOM) // PAGE) for c in contexts) + -(-(portion + cached) // PAGE) + 8
    runner = _runner(case, seed, pages, len(contexts) + 1)
    shape = (1, case["kv_rank"] + case["rot_dim"]) if kind == "latent" else (case["kv_heads"], case["dim"])
    keys = [f"d{i}" for i in range(len(contexts))]
    for i, (key, length) in enumerate(zip(keys, contexts)):
        _fill(runner.cache, key, case, seed, i, length, shape, layers)
    if kind == "step":
        return {"kind": kind, "runner": runner, "keys": keys, "contexts": contexts, "left": ROOM,
                "tokens": _tokens(case, seed, "decoded", len(keys)), "portion": _tokens(case, seed, "portion", portion)}
    _fill(runner.cache, "prompt", case, seed, len(keys), cached, shape, layers)
    entries = [StepEntry(key, [0]) for key in keys] + [StepEntry("prompt", [0] * portion)]
    for entry in entries:
        runner.cache.reserve(entry.key, runner.cache.request(entry.key).length + len(entry.tokens))
    state = {"kind": kind, "runner": runner, "cache": runner.cache.view(0), "batch": build_batch(entries, runner.cache, DEVICE)}
    rows = len(keys) + portion
    if kind == "latent":
        return dict(state, mixer=runner.model.blocks[0].mixer, x=_noise(seed, "x", (rows, case["width"]), torch.bfloat16))
    return dict(state, block=runner.model.blocks[0], norm=runner.model.final_norm, stream=_noise(seed, "x", (rows, case["width"])))


# -- one pass ------------------------------------------------------------------------------------
def run(state: dict):
    kind = state["kind"]
    if kind == "sample":
        return state["sampler"].sample(state["logits"], state["params"], state["seeds"], state["counters"])
    if kind == "routed":
        return state["ffn"].forward(state["x"])
    if kind == "step":
        return _step(state)
    state["batch"].shared.clear()
    if kind == "layer":
        h = state["stream"].clone()        # the residual stream is updated in place
        pending = state["block"].forward(h, None, state["batch"], state["cache"])
        return {"normed": state["norm"].add_forward(h, pending), "stream": h}
    out = state["mixer"].forward(state["x"], state["batch"], state["cache"])
    # a prompt's next portion starts from the states this one leaves
    return out if kind == "latent" else {"out": out, "states": state["states"]}


def _step(state: dict):
    runner = state["runner"]
    if state["left"] == 0:                 # the requests have ended; as many others take their places
        for key in state["keys"]:
            runner.end(key)
        for key, length in zip(state["keys"], state["contexts"]):
            runner.begin(key)
            runner.cache.reserve(key, length)
            runner.cache.advance(key, length)
        state["left"] = ROOM
    state["left"] -= 1
    entries = [StepEntry(key, [token], [0]) for key, token in zip(state["keys"], state["tokens"])]
    if not state["portion"]:
        return runner.step(entries)
    runner.begin("prompt")
    logits = runner.step(entries + [StepEntry("prompt", state["portion"], [len(state["portion"]) - 1])])
    runner.end("prompt")
    return logits


# -- what a pass cannot do without -----------------------------------------------------------------
def work(case: dict) -> dict:
    kind, size = case["kind"], 4 if case.get("dtype") == "f32" else 2
    if kind == "sample":
        return {"bytes": case["rows"] * case["vocab"] * 4, "flops": case["rows"] * case["vocab"] * 4}
    width = case["width"]
    if kind == "routed":
        pairs = case["rows"] * case["top"]
        used = case["experts"] * (1 - (1 - case["top"] / case["experts"]) ** case["rows"])
        return {"bytes": int(used * 3 * width * case["ff"] * 2) + case["rows"] * width * (2 + 4),
                "flops": pairs * 6 * width * case["ff"]}
    if kind in ("delta", "gated"):
        tokens, h, dk, dv = sum(_prompts(case)), case["heads"], case["dim"], case["vdim"]
        if kind == "delta":
            rows, per = 2 * case["kv_heads"] * dk + 2 * h * dv + 2 * h, 8
        else:
            rows, per = 2 * h * dk + h * dv, 4
        weights = width * (rows + h * dv)
        return {"bytes": weights * 2 + tokens * width * (2 + 4) + 2 * case["requests"] * h * dk * dv * 4,
                "flops": tokens * (2 * weights + per * h * dk * dv)}
    portion, cached = case["portion"], case.get("cached", 0)
    if kind == "latent":
        h, rank, rot, d, dv = case["heads"], case["kv_rank"], case["rot_dim"], case["dim"], case["vdim"]
        weights = width * (case["q_rank"] + rank + rot) + case["q_rank"] * h * (d + rot) + h * (d + dv) * rank + width * h * dv
        pairs = portion * cached + portion * (portion + 1) // 2
        # keys and values are expanded once per token, or the queries and sums are taken through the
        # expansions: the cheaper of the two
        expanded = 2 * pairs * h * (d + rot + dv) + 2 * cached * h * (d + dv) * rank
        absorbed = 2 * pairs * h * (2 * rank + rot)
        return {"bytes": weights * 2 + portion * width * 4 + (cached + portion) * (rank + rot) * 2,
                "flops": 2 * portion * weights + min(expanded, absorbed)}
    contexts, layers = _contexts(case), case.get("layers", 1)
    q, kv = case["heads"] * case["dim"], case["kv_heads"] * case["dim"]
    weights = width * (q + 2 * kv) + q * width + 3 * width * case["inter"]
    rows = len(contexts) + portion
    pairs = sum(c + 1 for c in contexts) + portion * cached + portion * (portion + 1) // 2
    total = {"bytes": layers * (weights * size + (sum(contexts) + cached + rows) * 2 * kv * size),
             "flops": layers * (2 * rows * weights + 4 * q * pairs)}
    if kind == "layer":
        total["bytes"] += rows * width * (4 + 4 + size)
        return total
    wanted = len(contexts) + (1 if portion else 0)
    total["bytes"] += case["vocab"] * (width * size + wanted * 4)
    total["flops"] += 2 * wanted * case["vocab"] * width
    return total


def tolerance(case: dict):
    if case["kind"] == "sample":
        return "exact"
    # a whole model's logits carry the rounding of all its layers; in 32 bits that of the rotation's
    # angles too (7e-7 of a layer, 9e-6 of four layers and the head against 64 bits)
    if case.get("dtype") == "f32":
        return {"rel": 4e-5} if case["kind"] == "step" else {"rel": 1e-5}
    return {"rel": 0.03} if case["kind"] == "step" else {"rel": 0.015}


# -- the same in 64 bits ---------------------------------------------------------------------------
def _rms(x, weight=None):
    y = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + EPS)
    return y if weight is None else y * weight


def _silu(x):
    return x * torch.sigmoid(x)


def _rotate(x, positions, base, pairs: bool):
    """x [N, heads, D] turned by position * base^(-2i / D); element i goes with i + D / 2, or with its
    neighbour (``pairs``)."""
    d = x.shape[-1]
    angle = positions.double()[:, None] * base ** (-torch.arange(0, d, 2, dtype=torch.float64, device=x.device) / d)
    cos, sin = torch.cos(angle)[:, None], torch.sin(angle)[:, None]
    if pairs:
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack((u * cos - v * sin, v * cos + u * sin), dim=-1).flatten(-2)
    u, v = x[..., : d // 2], x[..., d // 2 :]
    return torch.cat((u * cos - v * sin, v * cos + u * sin), dim=-1)


def _attend(q, k, v, first: int, scale: float):
    """q [n, heads, D] at positions first.. over k, v [L, kv_heads, D], causal."""
    n, heads, _ = q.shape
    per = heads // k.shape[1]
    hidden = torch.arange(k.shape[0], device=q.device)[None, :] > first + torch.arange(n, device=q.device)[:, None]
    out = torch.empty((n, heads, v.shape[-1]), dtype=q.dtype, device=q.device)
    for head in range(heads):
        scores = (q[:, head] @ k[:, head // per].T).mul_(scale).masked_fill_(hidden, -math.inf)
        out[:, head] = torch.softmax(scores, dim=-1) @ v[:, head // per]
    return out


def _qwen_layer(case, seed, layer, h, spans):
    """``spans``: (request, first row, rows, tokens cached) of every entry."""
    dtype = DTYPES[case["dtype"]]
    heads, kv, d = case["heads"], case["kv_heads"], case["dim"]
    width, inter = case["width"], case["inter"]

    def w(name, *shape):
        return _weight(seed, f"model.layers.{layer}.{name}.weight", shape, dtype).double()

    x = _rms(h, w("input_layernorm", width))
    positions = torch.cat([torch.arange(done, done + rows) for _, _, rows, done in spans]).to(DEVICE)
    q = _rms((x @ w("self_attn.q_proj", heads * d, width).T).view(-1, heads, d), w("self_attn.q_norm", d))
    k = _rms((x @ w("self_attn.k_proj", kv * d, width).T).view(-1, kv, d), w("self_attn.k_norm", d))
    v = (x @ w("self_attn.v_proj", kv * d, width).T).view(-1, kv, d)
    q, k = _rotate(q, positions, 1e6, False), _rotate(k, positions, 1e6, False)
    out = torch.empty_like(q)
    for request, at, rows, done in spans:
        seen = [_cached(case, seed, layer, side, request, done, (kv, d)).double() for side in "kv"] if done else [k[:0], v[:0]]
        out[at : at + rows] = _attend(q[at : at + rows], torch.cat((seen[0], k[at : at + rows])),
                                      torch.cat((seen[1], v[at : at + rows])), done, d ** -0.5)
    h = h + out.flatten(1) @ w("self_attn.o_proj", width, heads * d).T
    x = _rms(h, w("post_attention_layernorm", width))
    gate, up = x @ w("mlp.gate_proj", inter, width).T, x @ w("mlp.up_proj", inter, width).T
    return h + (_silu(gate) * up) @ w("mlp.down_proj", width, inter).T


def _exact_qwen(case, seed):
    contexts, portion = _contexts(case), case["portion"]
    spans = [(i, i, 1, length) for i, length in enumerate(contexts)]
    if portion:
        spans.append((len(contexts), len(contexts), portion, case.get("cached", 0)))
    dtype, width = DTYPES[case["dtype"]], case["width"]
    final = _weight(seed, "model.norm.weight", (width,), dtype).double()
    if case["kind"] == "layer":
        h = _qwen_layer(case, seed, 0, _noise(seed, "x", (len(contexts) + portion, width)).double(), spans)
        return {"normed": _rms(h, final), "stream": h}
    embed = _weight(seed, "model.embed_tokens.weight", (case["vocab"], width), dtype)
    ids = _tokens(case, seed, "decoded", len(contexts)) + _tokens(case, seed, "portion", portion)
    h = embed[torch.tensor(ids, device=DEVICE)].double()
    for layer in range(case["layers"]):
        h = _qwen_layer(case, seed, layer, h, spans)
    last = torch.tensor([at + rows - 1 for _, at, rows, _ in spans], device=DEVICE)
    x = _rms(h[last], final)
    return torch.cat([x @ piece.double().T for piece in embed.split(16384)], dim=1)


def _exact_recurrence(case, seed):
    width, h, dk, dv = case["width"], case["heads"], case["dim"], case["vdim"]
    lengths = _prompts(case)
    x = _noise(seed, "x", (sum(lengths), width), torch.bfloat16).double()

    def w(name, *shape):
        return _weight(seed, ("l0.mix." if name else "") + name, shape, torch.bfloat16).double()

    delta = case["kind"] == "delta"
    if delta:
        g = case["kv_heads"]
        raw = {"q": x @ w("q", g * dk, width).T, "k": x @ w("k", g * dk, width).T, "v": x @ w("v", h * dv, width).T}
        taps = {s: w(f"{s}.conv", raw[s].shape[1], case["conv"]) for s in "qkv"}
        beta = torch.sigmoid(x @ w("b", h, width).T)
        decay = torch.exp(-torch.exp(w("A_log", h)) * torch.nn.functional.softplus(x @ w("a", h, width).T + w("dt_bias", h)))
        gate = _silu(x @ w("g", h * dv, width).T).view(-1, h, dv)
    else:
        q_all = _silu(x @ w("q", h * dk, width).T).view(-1, h, dk)
        v_all = (x @ w("v", h * dv, width).T).view(-1, h, dv)
        low = w("lower", h * dk).view(h, dk)
        f_all = low + (1 - low) * torch.sigmoid(x @ w("f", h * dk, width).T + w("f.b", h * dk)).view(-1, h, dk)
    out, states, at = [], [], 0
    for length in lengths:
        rows = slice(at, at + length)
        at += length
        if delta:
            def convolved(s):
                padded = torch.nn.functional.pad(raw[s][rows].T, (case["conv"] - 1, 0))
                return _silu((padded.unfold(1, case["conv"], 1) * taps[s][:, None]).sum(-1).T)

            def unit(y):
                y = y.view(length, case["kv_heads"], dk)
                return (y * torch.rsqrt((y * y).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(h // case["kv_heads"], 1)

            q, k, v = unit(convolved("q")) * dk ** -0.5, unit(convolved("k")), convolved("v").view(length, h, dv)
            b, f = beta[rows], decay[rows]
        else:
            q, v, f = q_all[rows], v_all[rows], f_all[rows]
        state = torch.zeros((h, dk, dv), dtype=torch.float64, device=x.device)
        o = torch.empty((length, h, dv), dtype=torch.float64, device=x.device)
        for t in range(length):
            if delta:
                state = f[t, :, None, None] * state
                u = b[t, :, None] * (v[t] - (k[t, :, None] @ state).squeeze(1))
                state = torch.baddbmm(state, k[t, :, :, None], u[:, None])
            else:
                state = f[t, :, :, None] * state + (1 - f[t])[:, :, None] * v[t, :, None]
            o[t] = (q[t, :, None] @ state).squeeze(1)
        o = _rms(o, w("norm", dv))
        out.append((o * gate[rows] if delta else o).flatten(1))
        states.append(state)
    return {"out": torch.cat(out) @ w("o", width, h * dv).T, "states": states}


def _exact_latent(case, seed):
    width, h, d, r, dv, rank = (case[k] for k in ("width", "heads", "dim", "rot_dim", "vdim", "kv_rank"))
    portion, done = case["portion"], case["cached"]
    x = _noise(seed, "x", (portion, width), torch.bfloat16).double()

    def w(name, *shape):
        return _weight(seed, "l0.mix." + name, shape, torch.bfloat16).double()

    positions = torch.arange(done, done + portion, device=DEVICE)
    q = _rms(x @ w("dq", case["q_rank"], width).T, w("dq.norm", case["q_rank"])) @ w("uq", h * (d + r), case["q_rank"]).T
    q = q.view(portion, h, d + r)
    q = torch.cat((q[:, :, :d], _rotate(q[:, :, d:], positions, 1e6, True)), dim=-1)
    both = x @ w("dkv", rank + r, width).T
    shared = _rotate(both[:, None, rank:], positions, 1e6, True)[:, 0]
    cached = torch.cat((_rms(both[:, :rank], w("dkv.norm", rank)), shared), dim=-1)
    if done:
        cached = torch.cat((_cached(case, seed, 0, "k", 0, done, (1, rank + r))[:, 0].double(), cached))
    latent, shared = cached[:, :rank], cached[:, rank:]
    keys = torch.cat(((latent @ w("uk", h * d, rank).T).view(-1, h, d), shared[:, None].expand(-1, h, -1)), dim=-1)
    values = (latent @ w("uv", h * dv, rank).T).view(-1, h, dv)
    return _attend(q, keys, values, done, (d + r) ** -0.5).flatten(1) @ w("o", width, h * dv).T


def _exact_routed(case, seed):
    width, ff = case["width"], case["ff"]
    x = _noise(seed, "x", (case["rows"], width), torch.bfloat16).double()

    def w(name, *shape):
        return _weight(seed, "l0.mlp." + name, shape, torch.bfloat16).double()

    logits = x @ w("router", case["experts"], width).T + w("router.b", case["experts"])
    best, chosen = torch.topk(logits, case["top"], dim=-1)
    share = torch.softmax(best, dim=-1)
    out = torch.zeros_like(x)
    for e in range(case["experts"]):
        rows, place = (chosen == e).nonzero(as_tuple=True)
        y = _silu(x[rows] @ w(f"e{e}.gate", ff, width).T) * (x[rows] @ w(f"e{e}.up", ff, width).T)
        out.index_add_(0, rows, share[rows, place, None] * (y @ w(f"e{e}.down", width, ff).T))
    return out


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "sample":
        return None                        # whole numbers
    if kind in ("step", "layer"):
        return _exact_qwen(case, seed)
    if kind == "latent":
        return _exact_latent(case, seed)
    return _exact_routed(case, seed) if kind == "routed" else _exact_recurrence(case, seed)
