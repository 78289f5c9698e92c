"""What the engine's speed is judged by: the calls that programs make of it, at real Llama shapes.

The engine's work is to take token ids through a Llama decoder over a paged cache.  Programs do that in four ways, and every case
is one of them:

* ``generate``  requests run their prompts (``ModelRunner.step``), then decode together one token per step through a
  ``DecodeSession``, token ids from host memory in and sampled ids back to the host every step: one request at the lowest latency, a
  few, a full batch; greedy or with temperature and top-p.  The continuation's ids are given (the sampled ids are returned but not fed
  back), so that two runs whose last bits differ still run the same tokens.
* ``prompt``    prompts run as one step, the logits of their last places wanted and a token chosen from them: the time to a first token.
* ``score``     prompts run as one step, the logits of every place wanted and the likeliest token at each: how well given texts are predicted.
* ``serve``     ``Engine.generate`` over more requests of mixed lengths than one step takes, by the scheduler (prompts cut into
  portions and mixed with other requests' decode steps), then one pass over the generated texts for the logits at their ends.

Models: the three shapes of ``bench.py`` with as many layers as it runs by default.  Their weights are random but peaked as trained
ones are: the embedding's rows outweigh what random layers add, and the head's row of a token is the embedding's row of
the token that it follows, so that the likeliest token has a probability near 0.9 and greedy text does not hang on the last bits of
16-bit products.  Data types: bfloat16, and float32 (the engine's true 32-bit path) at smaller sizes.

Other architectures of this package share these products, norms, cache, scheduler and sampling; their own mixers are timed by
``bench.py --designs``.
"""
from __future__ import annotations

import json
import math
import os
import tempfile
from pathlib import Path

import numpy as np
import torch

from tinyllama_inference_engine_b200 import EngineConfig
from tinyllama_inference_engine_b200.engine.api import Engine
from tinyllama_inference_engine_b200.engine.batch import StepEntry
from tinyllama_inference_engine_b200.engine.decode_session import DecodeSession
from tinyllama_inference_engine_b200.engine.request import SamplingParams
from tinyllama_inference_engine_b200.weights import write_safetensors

MODELS = {
    "tinyllama": dict(hidden_size=2048, intermediate_size=5632, num_hidden_layers=22, num_attention_heads=32, num_key_value_heads=4,
                      max_position_embeddings=2048, vocab_size=32000, rms_norm_eps=1e-5, rope_theta=10000.0),
    "llama2-7b": dict(hidden_size=4096, intermediate_size=11008, num_hidden_layers=8, num_attention_heads=32, num_key_value_heads=32,
                      max_position_embeddings=4096, vocab_size=32000, rms_norm_eps=1e-5, rope_theta=10000.0),
    "llama3-8b": dict(hidden_size=4096, intermediate_size=14336, num_hidden_layers=8, num_attention_heads=32, num_key_value_heads=8,
                      max_position_embeddings=8192, vocab_size=128256, rms_norm_eps=1e-5, rope_theta=500000.0),
}
# tokens of cache and tokens of one step that a program of this model's would ask for
CAPACITY = {"tinyllama": (98304, 2048), "llama2-7b": (32768, 2048), "llama3-8b": (65536, 8192)}
MAX_REQUESTS = 64


# --- the cases ----------------------------------------------------------------------------------------------------------------
def listed() -> list[dict]:
    return [
        # A chat turn for one user: a short prompt, an answer token by token.  Latency and launches are all there is.
        _case("chat", "generate", "tinyllama", requests=1, shortest=57, longest=57, new=32),
        # The benchmark's headline: eight requests of 1,024 tokens each decode together.
        _case("eight requests", "generate", "tinyllama", requests=8, shortest=1024, longest=1024, new=64),
        # A full batch of short dialogues, sampled with the usual temperature and top-p.
        _case("full batch sampled", "generate", "tinyllama", requests=64, shortest=90, longest=310, new=32, temperature=0.8, top_p=0.95),
        # A wider model with a cache entry per head, two users.
        _case("two requests at 7B", "generate", "llama2-7b", requests=2, shortest=333, longest=500, new=32),
        # A server's middling batch on the widest model, texts of different lengths.
        _case("batch of 24 at 8B", "generate", "llama3-8b", requests=24, shortest=150, longest=1100, new=24),
        # Questions over long documents: the cache is a large part of what a decode step reads.
        _case("long documents at 8B", "generate", "llama3-8b", requests=4, shortest=3500, longest=4001, new=48, temperature=0.7, top_p=0.9),
        # The first token of a short question: the smallest call, mostly launches.
        _case("short prompt", "prompt", "tinyllama", requests=1, shortest=150, longest=150),
        # The first token after a whole context of prompt.
        _case("prompt of 2048", "prompt", "tinyllama", requests=1, shortest=2048, longest=2048),
        # A whole context of prompt on the widest model: the largest call.
        _case("prompt of 8192 at 8B", "prompt", "llama3-8b", requests=1, shortest=8192, longest=8192),
        # How well a few texts are predicted: logits at every place.
        _case("scored texts", "score", "tinyllama", requests=3, shortest=201, longest=420),
        # A serving run through the engine's own scheduler.
        _case("served requests", "serve", "tinyllama", requests=24, shortest=60, longest=1000, new=32),
        # The 32-bit path, as used to check a checkpoint's conversion: a few prompts and some tokens of each.
        _case("32-bit check", "generate", "tinyllama", dtype="float32", requests=4, shortest=120, longest=260, new=8),
    ]


def _case(name, kind, model, *, dtype="bfloat16", requests, shortest, longest, new=0, temperature=0.0, top_p=1.0) -> dict:
    case = {"kind": kind, "model": model, "dtype": dtype, "requests": requests, "shortest": shortest, "longest": longest, "new": new,
            "temperature": temperature, "top_p": top_p}
    return {"name": name, **case} if name else case


def _log_int(rng, low: int, high: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng) -> dict:
    """A case of the same ranges: any of the four kinds, any of the models, sizes spread over their logarithm, odd ones as likely as even ones."""
    most = max(_seconds(case) for case in listed())
    while True:
        kind = rng.choices(["generate", "prompt", "score", "serve"], [10, 6, 2, 3])[0]
        model = rng.choices(list(MODELS), [6, 2, 2])[0]
        tokens, budget = CAPACITY[model]
        context = MODELS[model]["max_position_embeddings"]
        dtype = "float32" if model == "tinyllama" and kind != "serve" and rng.random() < 0.15 else "bfloat16"
        spread = rng.choice([1.0, rng.uniform(0.1, 1.0)])
        if kind == "generate":
            small = dtype == "float32"
            requests, new = _log_int(rng, 1, 8 if small else 64), _log_int(rng, 8, 16 if small else 64)
            longest = _log_int(rng, 16, 512 if small else min(4096, context) - new)
            sampled = {"temperature": round(rng.uniform(0.5, 1.2), 2), "top_p": rng.choice([0.8, 0.9, 0.95, 1.0])} if rng.random() < 0.4 else {}
        elif kind == "prompt":
            requests, new, sampled = rng.choice([1, 1, 1, rng.randint(2, 8)]), 0, {}
            longest = _log_int(rng, 16, 512 if dtype == "float32" else budget // requests)
        elif kind == "score":
            requests, new, sampled = _log_int(rng, 1, 8), 0, {}
            longest = _log_int(rng, 16, min(1024, budget // requests))
        else:
            model, tokens, context = "tinyllama", CAPACITY["tinyllama"][0], MODELS["tinyllama"]["max_position_embeddings"]
            requests, new, sampled = _log_int(rng, 8, 48), _log_int(rng, 8, 48), {}
            longest = _log_int(rng, 64, 1500)
        case = _case(None, kind, model, dtype=dtype, requests=requests, shortest=max(8, int(longest * spread)), longest=max(8, longest), new=new, **sampled)
        total = sum(-(-(n + new + 1) // 64) * 64 for n in _lengths(case))
        if total <= tokens and _seconds(case) <= most:
            return case


def _lengths(case: dict) -> list[int]:
    """The requests' prompt lengths, spread from the shortest to the longest, in an order that is not sorted."""
    n, low, high = case["requests"], case["shortest"], case["longest"]
    spread = [high if n == 1 else low + (high - low) * i // (n - 1) for i in range(n)]
    return [spread[(i * 7 + 3) % n] for i in range(n)] if n % 7 else spread[::-1]


def _portions(lengths: list[int], budget: int) -> list[list[int]]:
    """Which requests run their prompts in one step: in order, as many as the step's budget takes."""
    steps: list[list[int]] = []
    room = 0
    for index, length in enumerate(lengths):
        if length > room or not steps:
            steps.append([])
            room = budget
        steps[-1].append(index)
        room -= length
    return steps


# --- what a program has in hand -------------------------------------------------------------------------------------------------
class _Handle:
    """An engine with its weights, and its decode sessions by batch size, as a program keeps them."""

    def __init__(self, model: str, dtype: str):
        tokens, self.budget = CAPACITY[model]
        tokens = tokens if dtype == "bfloat16" else 16384
        self.engine = Engine(_folder(model), EngineConfig(dtype=dtype, page_size=64, max_cache_tokens=tokens, max_requests=MAX_REQUESTS, max_batch_tokens=self.budget))
        self.runner = self.engine.runner
        self.sessions: dict[int, DecodeSession] = {}

    def session(self, count: int) -> DecodeSession:
        if count not in self.sessions:
            self.sessions[count] = DecodeSession(self.runner, count)
        return self.sessions[count]


_HANDLES: dict[tuple, _Handle] = {}


def _handle(model: str, dtype: str) -> _Handle:
    if (model, dtype) not in _HANDLES:
        _HANDLES[model, dtype] = _Handle(model, dtype)
    return _HANDLES[model, dtype]


def _weights(model: str) -> dict[str, torch.Tensor]:
    """The model's tensors (bfloat16, on the GPU), the same every time."""
    shapes = MODELS[model]
    hidden, inner, vocab = shapes["hidden_size"], shapes["intermediate_size"], shapes["vocab_size"]
    kv = hidden // shapes["num_attention_heads"] * shapes["num_key_value_heads"]
    generator = torch.Generator(device="cuda").manual_seed(20)

    def normal(*size, std=0.02, mean=0.0):
        return torch.empty(size, dtype=torch.bfloat16, device="cuda").normal_(mean, std, generator=generator)

    tensors = {"model.embed_tokens.weight": normal(vocab, hidden, std=1.0)}
    for layer in range(shapes["num_hidden_layers"]):
        prefix = f"model.layers.{layer}."
        tensors[prefix + "input_layernorm.weight"] = normal(hidden, mean=1.0)
        tensors[prefix + "self_attn.q_proj.weight"] = normal(hidden, hidden)
        tensors[prefix + "self_attn.k_proj.weight"] = normal(kv, hidden)
        tensors[prefix + "self_attn.v_proj.weight"] = normal(kv, hidden)
        tensors[prefix + "self_attn.o_proj.weight"] = normal(hidden, hidden)
        tensors[prefix + "post_attention_layernorm.weight"] = normal(hidden, mean=1.0)
        tensors[prefix + "mlp.gate_proj.weight"] = normal(inner, hidden)
        tensors[prefix + "mlp.up_proj.weight"] = normal(inner, hidden)
        tensors[prefix + "mlp.down_proj.weight"] = normal(hidden, inner)
    tensors["model.norm.weight"] = normal(hidden, mean=1.0)
    follows = torch.randperm(vocab, generator=generator, device="cuda")   # the token that each token follows
    tensors["lm_head.weight"] = (tensors["model.embed_tokens.weight"][follows].float() * 0.02).bfloat16()
    return tensors


def _folder(model: str) -> Path:
    """The model's folder, written once and kept in the temporary folder."""
    folder = Path(tempfile.gettempdir()) / f"tlie_b200_cases_{os.getuid()}_{model}"
    if not folder.exists():
        staging = Path(tempfile.mkdtemp(prefix="tlie_b200_cases_", dir=tempfile.gettempdir()))
        config = dict(MODELS[model], architectures=["LlamaForCausalLM"], model_type="llama", bos_token_id=1, eos_token_id=2)
        (staging / "config.json").write_text(json.dumps(config))
        write_safetensors(staging / "model.safetensors", _weights(model))
        try:
            os.replace(staging, folder)
        except OSError:   # another process was first
            return folder if folder.exists() else staging
    return folder


def _tokens(case: dict, seed: int) -> tuple[list[list[int]], np.ndarray]:
    """Prompts (uniform token ids) and the ids of the continuations, [new, requests]."""
    rng = np.random.default_rng(seed)
    vocab = MODELS[case["model"]]["vocab_size"]
    prompts = [rng.integers(3, vocab, size=n).tolist() for n in _lengths(case)]
    return prompts, rng.integers(3, vocab, size=(case["new"], case["requests"]))


_SERIAL = iter(range(1 << 62))


def prepare(case: dict, seed: int) -> dict:
    handle = _handle(case["model"], case["dtype"])
    prompts, following = _tokens(case, seed)
    serial = next(_SERIAL)
    state = {"kind": case["kind"], "handle": handle, "prompts": prompts, "ids": [f"case{serial}-{i}" for i in range(len(prompts))],
             "portions": _portions([len(p) for p in prompts], handle.budget),
             "params": [SamplingParams(max_tokens=max(1, case["new"]), temperature=case["temperature"], top_p=case["top_p"], seed=seed * 1000 + i) for i in range(len(prompts))]}
    if case["kind"] == "generate":
        state["following"] = following.tolist()
        state["session"] = handle.session(len(prompts))
        state["logits"] = torch.empty(case["new"], len(prompts), MODELS[case["model"]]["vocab_size"], dtype=torch.float32, device="cuda")
    return state


# --- one pass -------------------------------------------------------------------------------------------------------------------
def run(state: dict) -> dict:
    return {"generate": _generate, "prompt": _prompt, "score": _score, "serve": _serve}[state["kind"]](state)


def _run_prompts(state: dict, texts: list[list[int]], portions: list[list[int]], params: list, every_place: bool = False) -> tuple[torch.Tensor, np.ndarray]:
    """The texts step by step: the logits at their last places (or at every place) and the tokens chosen there, read by the host after every step."""
    engine, ids = state["handle"].engine, state["ids"]
    logits, chosen = [], []
    for portion in portions:
        entries = [StepEntry(ids[i], texts[i], list(range(len(texts[i]))) if every_place else [len(texts[i]) - 1]) for i in portion]
        logits.append(engine.runner.step(entries))
        choice = [params[i] for i in portion for _ in (texts[i] if every_place else [0])]
        chosen += engine.sampler.select(logits[-1], choice, [0] * len(choice))
    return torch.cat(logits) if len(logits) > 1 else logits[0], np.array(chosen)


def _finish(state: dict) -> None:
    for request in state["ids"]:
        state["handle"].runner.finish(request)


def _generate(state: dict) -> dict:
    session, ids = state["session"], state["ids"]
    first, chosen = _run_prompts(state, state["prompts"], state["portions"], state["params"])
    following, logits, sampled = state["following"], state["logits"], []
    session.load(ids, following[0], state["params"], [1] * len(ids))
    for index, tokens in enumerate(following):
        session.set_tokens(tokens)
        session.step()
        logits[index].copy_(session.logits)
        sampled.append(session.read_tokens())
    _finish(state)
    return {"first": first, "chosen": chosen, "logits": logits, "sampled": np.array(sampled)}


def _prompt(state: dict) -> dict:
    logits, chosen = _run_prompts(state, state["prompts"], state["portions"], state["params"])
    _finish(state)
    return {"logits": logits, "chosen": chosen}


def _score(state: dict) -> dict:
    logits, chosen = _run_prompts(state, state["prompts"], state["portions"], state["params"], every_place=True)
    _finish(state)
    return {"logits": logits, "likeliest": chosen}


def _serve(state: dict) -> dict:
    results = state["handle"].engine.generate(state["prompts"], state["params"])
    texts = [r.prompt_tokens + r.generated_tokens for r in results]
    logits, chosen = _run_prompts(state, texts, _portions([len(t) for t in texts], state["handle"].budget), state["params"])
    _finish(state)
    return {"generated": np.array([r.generated_tokens for r in results]), "logits": logits, "next": chosen}


# --- what a pass cannot do without ----------------------------------------------------------------------------------------------
def work(case: dict) -> dict:
    """Weights once per step, keys and values written once and read once per step, logits written; 2 flops per weight and row, 4 per query, key and channel."""
    shapes = MODELS[case["model"]]
    hidden, inner, layers, vocab = shapes["hidden_size"], shapes["intermediate_size"], shapes["num_hidden_layers"], shapes["vocab_size"]
    kv = hidden // shapes["num_attention_heads"] * shapes["num_key_value_heads"]
    size = 2 if case["dtype"] == "bfloat16" else 4
    layer_weights = layers * (2 * hidden * hidden + 2 * hidden * kv + 3 * hidden * inner)
    head = vocab * hidden
    budget = CAPACITY[case["model"]][1]
    total = {"bytes": 0.0, "flops": 0.0}

    def step(rows: int, pairs: int, read: int, wanted: int) -> None:
        """``rows`` tokens run, ``pairs`` of a query and a key that it sees, ``read`` cached tokens read, ``wanted`` rows of logits."""
        total["bytes"] += size * (layer_weights + head) + size * layers * 2 * kv * (rows + read) + 2 * size * rows * hidden + 4 * wanted * vocab
        total["flops"] += 2.0 * rows * layer_weights + 2.0 * wanted * head + 4.0 * pairs * hidden * layers

    def prompts(lengths: list[int], every_place: bool = False) -> None:
        for portion in _portions(lengths, budget):
            ns = [lengths[i] for i in portion]
            step(sum(ns), sum(n * (n + 1) // 2 for n in ns), 0, sum(ns) if every_place else len(ns))

    lengths = _lengths(case)
    prompts(lengths, every_place=case["kind"] == "score")
    for index in range(case["new"]):
        held = sum(n + index + 1 for n in lengths)
        step(len(lengths), held, held, len(lengths))
    if case["kind"] == "serve":
        prompts([n + case["new"] for n in lengths])
    return total


def _seconds(case: dict) -> float:
    """A pass's time on a B200, roughly: for the choice of cases that cost no more than the listed ones."""
    need = work(case)
    return need["bytes"] / 3e12 + need["flops"] / (6e14 if case["dtype"] == "bfloat16" else 3e13)


def tolerance(case: dict) -> dict:
    """Relative error of the logits, and the share of sampled ids that may fall the other way (a draw at the edge of a probability, a near tie)."""
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 2e-4, "differ": 0.02}
    return {"rel": 4e-2, "max": 3e-1, "differ": 0.05}


# --- the same in 64 bits, plainly -----------------------------------------------------------------------------------------------
def _norm64(x: torch.Tensor, weight: torch.Tensor, eps: float) -> torch.Tensor:
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * weight.double()


def _rotate64(x: torch.Tensor, theta: float) -> torch.Tensor:
    """x [length, heads, dim]: pairs (d, d + dim / 2) turned by position * theta ** (-2 d / dim)."""
    half = x.shape[-1] // 2
    angle = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None] * theta ** (-torch.arange(half, dtype=torch.float64, device=x.device) / half)
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)


def _attend64(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor) -> torch.Tensor:
    """Causal attention of one text, [length, heads, dim], a block of queries at a time."""
    length, heads, dim = q.shape
    groups = heads // k.shape[1]
    q = q.view(length, k.shape[1], groups, dim)
    out = torch.empty_like(q)
    block = max(1, (1 << 28) // (heads * length))
    for begin in range(0, length, block):
        end = min(length, begin + block)
        scores = torch.einsum("qhgd,khd->hgqk", q[begin:end], k[:end]) / math.sqrt(dim)
        later = torch.arange(end, device=q.device)[None, :] > torch.arange(begin, end, device=q.device)[:, None]
        out[begin:end] = torch.einsum("hgqk,khd->qhgd", scores.masked_fill_(later, -math.inf).softmax(-1), v[:end])
    return out.reshape(length, heads * dim)


def _logits64(shapes: dict, weights: dict, texts: list[list[int]], places: list[list[int]]) -> torch.Tensor:
    """Logits at the wanted places of every text, text after text."""
    heads, kv_heads, eps = shapes["num_attention_heads"], shapes["num_key_value_heads"], shapes["rms_norm_eps"]
    ids = torch.tensor([t for text in texts for t in text], device="cuda")
    starts = np.cumsum([0] + [len(t) for t in texts]).tolist()
    x = weights["model.embed_tokens.weight"][ids].double()
    for layer in range(shapes["num_hidden_layers"]):
        w = {name.removeprefix(f"model.layers.{layer}."): t for name, t in weights.items() if name.startswith(f"model.layers.{layer}.")}
        linear = lambda name, y: y @ w[name].double().T  # noqa: E731
        y = _norm64(x, w["input_layernorm.weight"], eps)
        q, k, v = (linear(f"self_attn.{c}_proj.weight", y).view(len(ids), n, -1) for c, n in (("q", heads), ("k", kv_heads), ("v", kv_heads)))
        mixed = [_attend64(_rotate64(q[a:b], shapes["rope_theta"]), _rotate64(k[a:b], shapes["rope_theta"]), v[a:b]) for a, b in zip(starts, starts[1:])]
        x = x + linear("self_attn.o_proj.weight", torch.cat(mixed))
        y = _norm64(x, w["post_attention_layernorm.weight"], eps)
        x = x + linear("mlp.down_proj.weight", torch.nn.functional.silu(linear("mlp.gate_proj.weight", y)) * linear("mlp.up_proj.weight", y))
    rows = torch.tensor([start + p for start, wanted in zip(starts, places) for p in wanted], device="cuda")
    return _norm64(x[rows], weights["model.norm.weight"], eps) @ weights["lm_head.weight"].double().T


_WEIGHTS: dict[str, dict] = {}


def exact(case: dict, seed: int) -> dict:
    """What ``run`` returns, in 64 bits; sampled ids have no such value (the likeliest ones do, where nothing is sampled at random)."""
    shapes = MODELS[case["model"]]
    if case["model"] not in _WEIGHTS:
        _WEIGHTS.clear()
        _WEIGHTS[case["model"]] = _weights(case["model"])
    weights = _WEIGHTS[case["model"]]
    prompts, following = _tokens(case, seed)
    new, count = case["new"], len(prompts)
    at_random = case["temperature"] > 0
    if case["kind"] == "prompt":
        logits = _logits64(shapes, weights, prompts, [[len(p) - 1] for p in prompts])
        return {"logits": logits, "chosen": logits.argmax(-1)}
    if case["kind"] == "score":
        logits = _logits64(shapes, weights, prompts, [list(range(len(p))) for p in prompts])
        return {"logits": logits, "likeliest": logits.argmax(-1)}
    if case["kind"] == "generate":
        texts = [p + following[:, i].tolist() for i, p in enumerate(prompts)]
        logits = _logits64(shapes, weights, texts, [list(range(len(p) - 1, len(p) + new)) for p in prompts]).view(count, new + 1, -1)
        likeliest = logits.argmax(-1).T.contiguous()
        return {"first": logits[:, 0], "chosen": None if at_random else likeliest[0], "logits": logits[:, 1:].transpose(0, 1).contiguous(),
                "sampled": None if at_random else likeliest[1:]}
    # greedy text: every token is guessed to be the likeliest one after the token before it, then the guesses are checked and mended until they hold
    follower = torch.empty(shapes["vocab_size"], dtype=torch.int64, device="cuda")
    norms = weights["model.embed_tokens.weight"].float()
    for begin in range(0, shapes["vocab_size"], 4000):
        follower[begin : begin + 4000] = (norms[begin : begin + 4000] @ weights["lm_head.weight"].float().T).argmax(-1)
    follower = follower.tolist()
    texts = [list(p) for p in prompts]
    for text in texts:
        for _ in range(new):
            text.append(follower[text[-1]])
    for _ in range(new):
        likeliest = _logits64(shapes, weights, texts, [list(range(len(p) - 1, len(p) + new - 1)) for p in prompts]).argmax(-1).view(count, new).tolist()
        right = True
        for text, prompt, best in zip(texts, prompts, likeliest):
            for index, token in enumerate(best):
                if text[len(prompt) + index] != token:
                    right = False
                    text[len(prompt) + index] = token
                    for later in range(index + 1, new):
                        text[len(prompt) + later] = follower[text[len(prompt) + later - 1]]
                    break
        if right:
            break
    logits = _logits64(shapes, weights, texts, [[len(t) - 1] for t in texts])
    return {"generated": torch.tensor([text[-new:] for text in texts], device="cuda"), "logits": logits, "next": logits.argmax(-1)}
