"""The engine's work in cases that can be timed and compared: what ``prepare`` makes is what a program that uses the engine
keeps (weights on the device, a page pool, captured decode graphs, the requests' token ids on the host), ``run`` is one pass
of such a program through ``ModelRunner.step``, and ``exact`` says in 64 bits what the pass computes.

A pass replays given token ids (as ``bin/trace_run`` does): every step's batch is fixed by the case, so that the logits of
two runs can be compared value by value; sampled tokens could not be, since a rounding decides between near-equal logits
and everything after that differs.  The sampler has a case of its own, on given logits.  For the same reason no case has
routed experts: a rounding turns the choice of an expert.

A case names a model (``model``: a Qwen2.5 shape of the benchmark or one of its hybrid designs at a benchmark size), its
``dtype``, how many ``requests`` run, the longest ``prompt`` among them (``ragged``: the others are spread evenly between a
quarter of it and all of it), ``budget``, the tokens of a step that go to prompts and decoding together, dealt out in order
of arrival, and ``outputs``, the tokens fed one by one after a prompt.  With ``cached`` the prompts are in the cache before
the pass and shared by its requests, so that a pass is decode steps only.
"""
from __future__ import annotations

import hashlib
import math

import torch

from flexengine_b200.bench.hybrid import SIZES, bebulorn_config, fuvuvik_config, ribozen_config
from flexengine_b200.bench.shapes import PAGE, SHAPES
from flexengine_b200.cache import CacheManager
from flexengine_b200.config import resolve
from flexengine_b200.engine import ModelRunner, StepEntry
from flexengine_b200.sampling import Sampler
from flexengine_b200.weights import random_model

DEV = "cuda:0"
TORCH_DTYPE = {"bfloat16": torch.bfloat16, "float32": torch.float32}


# ---- the cases --------------------------------------------------------------------------------------------------------
def _case(model, requests, prompt, budget, outputs, ragged=False, cached=False, dtype="bfloat16"):
    return {"kind": "model", "model": model, "dtype": dtype, "requests": requests, "prompt": prompt, "ragged": ragged,
            "cached": cached, "budget": budget, "outputs": outputs}


def listed():
    return [
        # one short question to a small model, answered alone: every step is all latency
        dict(_case("qwen2-1.5b", 1, 61, 2048, 32), name="answer-1.5b-b1"),
        # the headline workload of the benchmark: batch 8 after 2,048-token prompts
        dict(_case("qwen2-7b", 8, 2048, 2048, 16, cached=True), name="decode-7b-b8"),
        # a loaded server: 64 conversations of different length
        dict(_case("qwen2-7b", 64, 2048, 2048, 4, ragged=True, cached=True), name="decode-7b-b64"),
        # long documents on the largest shape, 16 of them
        dict(_case("qwen2-14b", 16, 8192, 8192, 4, ragged=True, cached=True), name="decode-14b-b16-8k"),
        # the benchmark's prompt in one step
        dict(_case("qwen2-7b", 1, 2048, 2048, 0), name="prefill-7b-2k"),
        # a long document in one step: the largest
        dict(_case("qwen2-14b", 1, 8192, 8192, 0), name="prefill-14b-8k"),
        # a small model serves: prompts of odd lengths in portions beside decoded tokens, under the benchmark's budget
        dict(_case("qwen2-1.5b", 32, 1021, 2048, 8, ragged=True), name="serve-1.5b"),
        # the 32-bit path, in which results are checked: the same model, portions of prompts beside decoded tokens
        dict(_case("qwen2-1.5b", 4, 509, 256, 4, ragged=True, dtype="float32"), name="check-1.5b-fp32"),
        # the hybrid designs: prompts of odd lengths under the benchmark's budget, then decoding
        dict(_case("fuvuvik-2k", 4, 2039, 2048, 16, ragged=True), name="fuvuvik-2k"),
        dict(_case("bebulorn-2k", 4, 2039, 2048, 16, ragged=True), name="bebulorn-2k"),
        dict(_case("ribozen-2k", 4, 2039, 2048, 16, ragged=True), name="ribozen-2k"),
        # the next tokens of 64 requests, greedy, with a temperature, and with the largest logits only
        {"kind": "sample", "rows": 64, "vocab": 152064, "name": "sample-b64"},
    ]


def _spread(rng, low, high):
    """A whole number between the two, uniform over its logarithm."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prefill", "prefill", "serve", "check", "hybrid", "hybrid", "sample"])
    if kind == "sample":
        return {"kind": "sample", "rows": _spread(rng, 1, 64), "vocab": rng.choice([32000, 151936, 152064])}
    if kind == "hybrid":
        model = rng.choice(["fuvuvik", "bebulorn", "ribozen"]) + "-" + rng.choice(["1k", "2k"])
        return _case(model, _spread(rng, 1, 8), _spread(rng, 33, 2048), rng.choice([512, 1024, 2048]), rng.randint(8, 16), ragged=True)
    if kind == "check":
        return _case("qwen2-1.5b", _spread(rng, 1, 4), _spread(rng, 17, 500), rng.choice([128, 256]), rng.randint(2, 4), ragged=True, dtype="float32")
    shape = rng.choice(["1.5b", "7b", "14b"])
    if kind == "decode":
        requests = _spread(rng, 1, 64)
        prompt = _spread(rng, 64, min(8192, 65536 // requests)) // PAGE * PAGE
        return _case("qwen2-" + shape, requests, prompt, 8192, rng.randint(3, 8), ragged=rng.random() < 0.7, cached=True)
    if kind == "prefill":
        return _case("qwen2-" + shape, rng.randint(1, 2), _spread(rng, 17, 4096), rng.choice([2048, 8192]), 0, ragged=True)
    return _case("qwen2-" + shape, _spread(rng, 4, 32 if shape == "1.5b" else 12), _spread(rng, 64, 1024), rng.choice([512, 2048]),
                 rng.randint(4, 8), ragged=True)


# ---- what a case means ------------------------------------------------------------------------------------------------
# Layers of the Qwen2.5 shapes.  The widths, heads and vocabularies are the shapes' own, but random weights make roundings grow
# with depth: two runs that round bfloat16 at other places differ by 2.6 % in the logits of the whole 7B shape and by over 3 %
# in those of the 14B shape (1.8 % at 28 layers of the 1.5B shape, 14 of the 7B shape and 12 of the 14B shape).
LAYERS = {"1.5b": 28, "7b": 14, "14b": 12}


def _config(model):
    design, size = model.split("-", 1)
    if design == "qwen2":
        return dict(SHAPES[size], num_hidden_layers=LAYERS[size])
    width, layers, vocab, heads = SIZES[size]
    if design == "fuvuvik":
        return fuvuvik_config(width, layers, vocab, heads)
    if design == "bebulorn":       # with a dense feed-forward in every layer
        config = bebulorn_config(width, layers, vocab, heads)
        for layer in config["layers"]:
            layer["mlp"] = {"kind": "dense", "ff": width * 5 // 2}
        return config
    config = ribozen_config(width, layers, vocab, heads)      # a stack of mixers alone
    for layer in config["layers"]:
        del layer["mlp"]
    return config


def _prompt_lengths(case):
    n, longest = case["requests"], case["prompt"]
    lengths = [longest] * n
    if case["ragged"] and n > 1:
        lengths = [longest - (longest * 3 // 4) * (n - 1 - i) // (n - 1) for i in range(n)]
    return [max(PAGE, length // PAGE * PAGE) for length in lengths] if case["cached"] else lengths


def _schedule(case, lengths):
    """[[(request, first position, tokens)]]: the steps of a pass, the budget dealt out in order of arrival."""
    done = list(lengths) if case["cached"] else [0] * len(lengths)
    total = [length + case["outputs"] for length in lengths]
    steps = []
    while any(d < t for d, t in zip(done, total)):
        budget, step = case["budget"], []
        for r, (d, t) in enumerate(zip(done, total)):
            count = min(budget, lengths[r] - d) if d < lengths[r] else min(budget, t - d, 1)
            if count > 0:
                step.append((r, d, count))
                done[r] += count
                budget -= count
        steps.append(step)
    return steps


def _wants_logits(lengths, r, first, count):
    return first + count >= lengths[r]


def _arrival(case, seed):
    """The requests' lengths in the order they arrive, and their token ids: prompt and what is fed after it."""
    lengths = _prompt_lengths(case)
    gen = torch.Generator().manual_seed(seed)
    lengths = [lengths[i] for i in torch.randperm(len(lengths), generator=gen).tolist()]
    config = _config(case["model"])
    vocab = config["vocab_size"] if "vocab_size" in config else config["vocab"]
    return lengths, [torch.randint(0, vocab, (n + case["outputs"],), generator=gen).tolist() for n in lengths]


class _State:
    pass


def prepare(case, seed):
    if case["kind"] == "sample":
        return _prepare_sample(case, seed)
    lengths, ids = _arrival(case, seed)
    n, outputs = len(lengths), case["outputs"]
    state = _State()
    _typed, plan, model = random_model(_config(case["model"]), seed=seed, dtype=case["dtype"], device=DEV)
    pages = sum(-(-(length + outputs) // PAGE) + (1 if case["cached"] else 0) for length in lengths)
    seats = 2 * n if case["cached"] else n
    state.cache = CacheManager(plan.cache_groups, pages, PAGE, seats, TORCH_DTYPE[case["dtype"]], DEV)
    state.runner = ModelRunner(model, state.cache)
    if outputs:
        limit = max(2048, -(-(max(lengths) + outputs) // 1024) * 1024)
        state.runner.enable_decode_graphs(n, limit)
        state.runner.capture_decode_graphs()
    state.shared = []
    if case["cached"]:
        for r, length in enumerate(lengths):
            for first in range(0, length, case["budget"]):
                state.runner.step([StepEntry(f"prompt{r}", ids[r][first:min(first + case["budget"], length)], [])])
            state.shared.append((f"prompt{r}", f"r{r}", length))
    state.steps, rows = [], 0
    for step in _schedule(case, lengths):
        entries = [(f"r{r}", ids[r][a:a + k], [k - 1] if _wants_logits(lengths, r, a, k) else []) for r, a, k in step]
        wanted = sum(len(want) for _, _, want in entries)
        state.steps.append((entries, rows, wanted))
        rows += wanted
    state.names = [f"r{r}" for r in range(n)]
    state.logits = torch.empty((rows, plan.vocab_size), dtype=torch.float32, device=DEV)
    # the cache of a pass that fills all of it belongs to what the pass computes
    state.storages = [] if case["cached"] else [g.storage for g in state.cache.groups if g.storage.numel()]
    return state


def _prepare_sample(case, seed):
    """Logits as a model of this kind gives them (spread 1 to 2), parameters as requests bring them, in turns."""
    gen = torch.Generator(DEV).manual_seed(seed)
    state = _State()
    rows = case["rows"]
    spread = 1.0 + torch.rand((rows, 1), generator=gen, device=DEV)
    state.given = torch.randn((rows, case["vocab"]), generator=gen, device=DEV) * spread
    state.temperatures = [(0.0, 0.8, 1.0, 0.7)[i % 4] for i in range(rows)]
    state.top_ks = [(0, 40, 0, 50)[i % 4] for i in range(rows)]
    state.seeds = [seed + i for i in range(rows)]
    state.draws = [(seed + 7 * i) % 256 for i in range(rows)]
    state.sampler = Sampler()
    return state


def run(state):
    if hasattr(state, "sampler"):
        return {"tokens": state.sampler.sample_on_device(state.given, state.temperatures, state.top_ks, state.seeds, state.draws)}
    runner = state.runner
    for donor, name, tokens in state.shared:
        state.cache.share_prefix(donor, name, tokens)
    for entries, at, wanted in state.steps:
        logits = runner.step([StepEntry(name, tokens, want) for name, tokens, want in entries])
        if wanted:           # a decode step's logits are overwritten by the next one's
            state.logits[at:at + wanted].copy_(logits)
    for name in state.names:
        runner.finish(name)
    return {"logits": state.logits, "cache": state.storages}


# ---- what a pass cannot do without ------------------------------------------------------------------------------------
def work(case):
    if case["kind"] == "sample":
        return {"bytes": 4.0 * case["rows"] * (case["vocab"] + 1), "flops": 0.0}
    config = _config(case["model"])
    _typed, plan = resolve(config)
    width = 2 if case["dtype"] == "bfloat16" else 4
    hidden, vocab = plan.hidden_size, plan.vocab_size
    runs = [entry.layer for entry in plan.run]
    in_layer = {}
    for b in plan.bindings:
        if b.target[0] == "layer":
            in_layer[b.target[1]] = in_layer.get(b.target[1], 0) + sum(math.prod(s.shape) for s in b.sources if len(s.shape) > 1)
    body, passed = sum(in_layer.values()), sum(in_layer[i] for i in runs)
    # attention as (query heads x (query + value size), elements a token keeps, window), one per layer that runs
    if "layers" in config:
        sights = []
        for i in runs:
            m = config["layers"][i]["mixer"]
            m = m.get("left", m)
            if config["layers"][i]["type"] in ("attention", "attention_2", "parallel"):
                sights.append((m["heads"] * (m["dim"] + m["vdim"]), m["kv_heads"] * (m["dim"] + m["vdim"]), (m.get("mask") or {}).get("size", 0)))
    else:
        d = config["head_dim"]
        sights = [(config["num_attention_heads"] * 2 * d, config["num_key_value_heads"] * 2 * d, 0)] * len(runs)
    states = sum(g.slots * math.prod(g.state_shape) for g in plan.cache_groups if g.kind == "state")
    lengths = _prompt_lengths(case)
    steps = _schedule(case, lengths)
    total_bytes = total_flops = 0.0
    for step in steps:
        tokens = sum(k for _, _, k in step)
        rows = sum(1 for r, a, k in step if _wants_logits(lengths, r, a, k))
        total_bytes += width * (body + tokens * hidden) + (width * hidden * vocab if rows else 0) + 4.0 * rows * vocab
        total_bytes += 2 * 4.0 * states * len(step)
        total_flops += 2.0 * passed * tokens + 2.0 * hidden * vocab * rows + 4.0 * states * tokens
        for per_key, kept, window in sights:
            for _, a, k in step:
                earlier = min(a, window) if window else a
                pairs = sum(min(a + i + 1, window) for i in range(k)) if window else k * a + k * (k + 1) / 2
                total_bytes += width * kept * (earlier + k)
                total_flops += 2.0 * per_key * pairs
    return {"bytes": total_bytes, "flops": total_flops}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    if case["dtype"] == "float32":          # 1e-5 off the 64-bit result, where roundings grow as they do in bfloat16
        return {"rel": 4e-5, "max": 2e-3}
    if case["model"].startswith("qwen2"):   # the same prompts in portions of another length: 1.3 to 1.8 %, a value by up to 0.12
        return {"rel": 0.03, "max": 0.5}
    return {"rel": 0.02, "max": 0.5}        # 0.4 % off the 64-bit result


# ---- in 64 bits -------------------------------------------------------------------------------------------------------
class _Weights:
    """The tensors of the random checkpoint of a seed, each drawn by itself in 32 bits, kept in bfloat16, given in 64 bits."""

    def __init__(self, seed):
        self.seed = seed

    def stored(self, name, *shape, mean=0.0, std=None):
        std = 1.0 / math.sqrt(shape[-1]) if std is None else std
        digest = hashlib.sha256(f"{int(self.seed)}:{name}".encode("utf8")).digest()
        gen = torch.Generator(DEV).manual_seed(int.from_bytes(digest[:8], "little") & ((1 << 63) - 1))
        slab = max(1, (1 << 26) // (math.prod(shape) // shape[0]))
        if len(shape) < 2:
            slab = shape[0]
        parts = []
        for first in range(0, shape[0], slab):
            part = (min(slab, shape[0] - first),) + shape[1:]
            parts.append((torch.randn(part, generator=gen, device=DEV) * std + mean).to(torch.bfloat16))
        return torch.cat(parts)

    def __call__(self, name, *shape, mean=0.0, std=None):
        return self.stored(name, *shape, mean=mean, std=std).double()


def _product(x, w):
    """x W^T, a few thousand rows at a time."""
    rows = x.reshape(-1, x.shape[-1])
    return torch.cat([part @ w.T for part in rows.split(8192)]).reshape(*x.shape[:-1], w.shape[0])


def _unit_rms(x, eps):
    return x * torch.rsqrt(x.square().mean(dim=-1, keepdim=True) + eps)


def _layer_norm(x, eps):
    x = x - x.mean(dim=-1, keepdim=True)
    return x * torch.rsqrt(x.square().mean(dim=-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _softplus(x):
    return torch.clamp(x, min=0.0) + torch.log1p(torch.exp(-x.abs()))


def _turn(x, freq, gain=1.0):
    """x [B, T, heads, dim]: entry i and entry i + len(freq) of a head turn by position * freq[i]; the others stay."""
    half = freq.numel()
    angle = (torch.arange(x.shape[1], dtype=torch.float64, device=DEV)[:, None] * freq)[:, None, :]
    c, s = torch.cos(angle) * gain, torch.sin(angle) * gain
    a, b = x[..., :half], x[..., half:2 * half]
    return torch.cat([a * c - b * s, b * c + a * s, x[..., 2 * half:]], dim=-1)


def _frequencies(base, dims):
    return base ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device=DEV) / dims)


def _attend(q, k, v, scale, seen=None, squash=None, sink=False):
    """q [B, T, heads, d], k and v [B, T, kv heads, d]: softmax attention over the keys before, ``seen(i, j)`` of them."""
    T, heads = q.shape[1], q.shape[2]
    group = heads // k.shape[2]
    out = torch.empty(q.shape[:3] + v.shape[-1:], dtype=q.dtype, device=DEV)
    j = torch.arange(T, device=DEV)[None, :]
    for b in range(q.shape[0]):
        for h in range(heads):
            for first in range(0, T, 2048):
                i = torch.arange(first, min(first + 2048, T), device=DEV)[:, None]
                scores = q[b, i[:, 0], h] @ k[b, :, h // group].T * scale
                if squash is not None:
                    cap, factor = squash
                    scores = cap * torch.tanh(scores * (1.0 if factor is None else factor[h]) / cap)
                visible = j <= i
                if seen is not None:
                    visible = visible & seen(i, j)
                scores = scores.masked_fill(~visible, float("-inf"))
                top = scores.amax(dim=-1, keepdim=True)
                if sink:
                    top = top.clamp(min=0.0)
                e = torch.exp(scores - top)
                below = e.sum(dim=-1, keepdim=True) + (torch.exp(-top) if sink else 0.0)
                out[b, i[:, 0], h] = (e / below) @ v[b, :, h // group]
    return out.flatten(2)


def _convolve(x, table, bias=None):
    """x [B, T, channels], table [channels, taps]: every channel's last ``taps`` rows weighed, zeros before the start."""
    taps = table.shape[1]
    padded = torch.nn.functional.pad(x, (0, 0, taps - 1, 0))
    y = sum(padded[:, t:t + x.shape[1]] * table[:, t] for t in range(taps))
    return y if bias is None else y + bias


def _qwen2(config, w, ids):
    hidden, inner, vocab = config["hidden_size"], config["intermediate_size"], config["vocab_size"]
    heads, kv, d, eps = config["num_attention_heads"], config["num_key_value_heads"], config["head_dim"], config["rms_norm_eps"]
    freq = _frequencies(config["rope_theta"], d)
    x = w.stored("model.embed_tokens.weight", vocab, hidden, std=0.02)[ids].double()
    for i in range(config["num_hidden_layers"]):
        p = f"model.layers.{i}."

        def linear(h, name, rows, columns, bias=False):
            y = _product(h, w(p + name + ".weight", rows, columns, std=0.02))
            return y + w(p + name + ".bias", rows, std=0.02) if bias else y

        h = _unit_rms(x, eps) * w(p + "input_layernorm.weight", hidden, mean=1.0, std=0.01)
        q, k, v = (linear(h, f"self_attn.{n}_proj", m * d, hidden, True).unflatten(-1, (m, d)) for n, m in (("q", heads), ("k", kv), ("v", kv)))
        x = x + linear(_attend(_turn(q, freq), _turn(k, freq), v, d ** -0.5), "self_attn.o_proj", hidden, heads * d)
        h = _unit_rms(x, eps) * w(p + "post_attention_layernorm.weight", hidden, mean=1.0, std=0.01)
        x = x + linear(_silu(linear(h, "mlp.gate_proj", inner, hidden)) * linear(h, "mlp.up_proj", inner, hidden), "mlp.down_proj", hidden, inner)
    x = _unit_rms(x, eps) * w("model.norm.weight", hidden, mean=1.0, std=0.01)
    head = "model.embed_tokens.weight" if config["tie_word_embeddings"] else "lm_head.weight"
    return x, w(head, vocab, hidden, std=0.02)


def _fuvuvik(config, w, ids):
    D, vocab, eps, S = config["width"], config["vocab"], config["norm"]["eps"], config["streams"]
    x = w.stored("embed", vocab, D, std=1.0)[ids].double() * config["embedding"]["scale"]
    streams = torch.stack([x] * S)
    for i, layer in enumerate(config["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        mp = p + "mix."

        def mixer(h):
            before = torch.nn.functional.pad(h, (0, 0, 1, 0))[:, :-1]
            h = h + (before - h) * w(p + "shift", D, mean=0.5, std=0.2)
            if layer["type"] == "mingru":
                W = m["width"]
                z = torch.sigmoid(_product(h, w(mp + "z", W, D)) + w(mp + "z.b", W, std=0.5))
                u = _product(h, w(mp + "x", W, D)) + w(mp + "x.b", W, std=0.5)
                u = torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
                state, rows = torch.zeros_like(z[:, 0]), []
                for t in range(z.shape[1]):
                    state = torch.lerp(state, u[:, t], z[:, t])
                    rows.append(state)
                return _product(torch.stack(rows, 1) * _silu(_product(h, w(mp + "g", W, D))), w(mp + "o", D, W))
            H, G, d, dv, chunk = m["heads"], m["kv_heads"], m["dim"], m["vdim"], (m.get("mask") or {}).get("size", 0)
            made = []
            for name, heads, size in (("q", H, d), ("k", G, d), ("v", G, dv)):
                y = _product(h, w(mp + name, heads * size, D))
                if not chunk:
                    taps = m["conv"]
                    y = _convolve(y, w(mp + name + ".conv", heads * size, taps, mean=1.0 / taps, std=0.5 / taps))
                y = y.unflatten(-1, (heads, size))
                if name != "v":
                    y = _turn(y, _frequencies(m["rot"]["base"], m["rot"]["dims"]))
                    y = y if chunk else _unit_rms(y, eps)
                made.append(y)
            out = _attend(*made, m["scale"], seen=(lambda a, b: a // chunk == b // chunk) if chunk else None, sink=bool(chunk))
            out = out.unflatten(-1, (H, dv)) * torch.sigmoid(_product(h, w(mp + "g", H, D)))[..., None]
            return _product(out.flatten(2), w(mp + "o", D, H * dv))

        def feed_forward(h):
            f = layer["mlp"]["ff"]
            g = torch.nn.functional.gelu(_product(h, w(p + "mlp.gate", f, D)), approximate="tanh")
            return _product(g * _product(h, w(p + "mlp.up", f, D)), w(p + "mlp.down", D, f))

        for q, branch in (("1", mixer), ("2", feed_forward)):
            h = torch.einsum("s,sbtd->btd", w(p + f"hc{q}.in", S, mean=1.0 / S, std=0.3 / S), streams)
            h = _unit_rms(h, eps) * w(p + "norm" + q, D, mean=1.0, std=0.1)
            y = branch(h) * torch.sigmoid(_product(h, w(p + "rg" + q, D, D)) + w(p + f"rg{q}.b", D, mean=0.5, std=0.5))
            mixed = torch.einsum("st,sbxd->tbxd", w(p + f"hc{q}.mix", S, S, mean=1.0 / S, std=0.3 / S), streams)
            streams = mixed + w(p + f"hc{q}.out", S, mean=1.0, std=0.2)[:, None, None, None] * y
    x = _unit_rms(streams.sum(0), eps) * w("final.norm", D, mean=1.0, std=0.1)
    return x, w("head", vocab, D)


def _bebulorn(config, w, ids):
    D, vocab, eps = config["width"], config["vocab"], config["norm"]["eps"]

    def norm(x, name):
        return _layer_norm(x, eps) * w(name, D, mean=1.0, std=0.1) + w(name + ".b", D, std=0.1)

    def attention(h, p, m):
        H, G, d, dv, window = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["mask"]["size"]
        q = _product(h, w(p + "q", H * d, D)).unflatten(-1, (H, d))
        k = _product(h, w(p + "k", G * d, D)).unflatten(-1, (G, d))
        v = _unit_rms(_product(h, w(p + "v", G * dv, D)).unflatten(-1, (G, dv)), eps)
        out = _attend(q, k, v, m["scale"], seen=lambda a, b: a - b < window, squash=(m["softcap"], w(p + "temp", H, mean=1.0, std=0.1)))
        return _product(out, w(p + "o", D, H * dv))

    def lightning(h, p, m):
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        q, k, v = (_silu(_product(h, w(p + n, H * s, D))).unflatten(-1, (H, s)) for n, s in (("q", d), ("k", d), ("v", dv)))
        decay = torch.tensor(m["decay"], dtype=torch.float64, device=DEV)[:, None, None]
        state, rows = torch.zeros(h.shape[0], H, d, dv, dtype=torch.float64, device=DEV), []
        for t in range(h.shape[1]):
            state = decay * state + k[:, t, :, :, None] * v[:, t, :, None, :]
            rows.append((q[:, t, :, None, :] @ state)[:, :, 0])
        out = _unit_rms(torch.stack(rows, 1).flatten(2), eps) * w(p + "norm", H * dv, mean=1.0, std=0.1)
        return _product(out * torch.sigmoid(_product(h, w(p + "g", H * dv, D))), w(p + "o", D, H * dv))

    def delta(h, p, m):
        H, G, d, dv, taps = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["conv"]

        def stream(name, heads, size):
            return _silu(_convolve(_product(h, w(p + name, heads * size, D)), w(p + name + ".conv", heads * size, taps))).unflatten(-1, (heads, size))

        def unit(x):
            return (x * torch.rsqrt(x.square().sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, dim=2)

        q, k, v = unit(stream("q", G, d)) * d ** -0.5, unit(stream("k", G, d)), stream("v", H, dv)
        rate = torch.exp(w(p + "A_log", H, mean=-1.0, std=1.0))
        keep = torch.exp(-rate * _softplus(_product(h, w(p + "a", H, D)) + w(p + "dt_bias", H, mean=-2.0, std=1.0)))
        step = torch.sigmoid(_product(h, w(p + "b", H, D)))
        state, rows = torch.zeros(h.shape[0], H, d, dv, dtype=torch.float64, device=DEV), []
        for t in range(h.shape[1]):
            state = keep[:, t, :, None, None] * state
            off = step[:, t, :, None, None] * (v[:, t, :, None, :] - k[:, t, :, None, :] @ state)
            state = state + k[:, t, :, :, None] * off
            rows.append((q[:, t, :, None, :] @ state)[:, :, 0])
        out = _unit_rms(torch.stack(rows, 1), eps) * w(p + "norm", dv, mean=1.0, std=0.1)
        return _product(out.flatten(2) * _silu(_product(h, w(p + "g", H * dv, D))), w(p + "o", D, H * dv))

    first = x = w.stored("embed", vocab, D, std=1.0)[ids].double()
    loop = config["loop"]
    order = [(i, turn > 0 and i == loop["start"]) for turn in range(loop["times"]) for i in range(loop["start"], loop["stop"])]
    order = [(i, False) for i in range(loop["start"])] + order + [(i, False) for i in range(loop["stop"], len(config["layers"]))]
    for i, again in order:
        p, layer = f"l{i}.", config["layers"][i]
        x = x + first if again else x
        mixer = {"attention": attention, "lightning": lightning, "delta": delta}[layer["type"]]
        x = x + config["residual_mult"] * norm(mixer(norm(x, p + "norm1"), p + "mix.", layer["mixer"]), p + "norm1b")
        f, h = layer["mlp"]["ff"], norm(x, p + "norm2")
        y = torch.relu(_product(h, w(p + "mlp.gate", f, D))) * _product(h, w(p + "mlp.up", f, D))
        x = x + config["residual_mult"] * norm(_product(y, w(p + "mlp.down", D, f)), p + "norm2b")
    return norm(x, "final.norm"), w("head", vocab, D)


def _ribozen(config, w, ids):
    D, vocab, eps = config["width"], config["vocab"], config["norm"]["eps"]

    def scan(q, k, v, decay, weight):
        """State of [N, dv] a head: S <- decay S + weight k v^T, read by q."""
        state, rows = torch.zeros(q.shape[0], q.shape[2], q.shape[3], v.shape[3], dtype=torch.float64, device=DEV), []
        for t in range(q.shape[1]):
            state = decay[:, t, :, None, None] * state + (weight[:, t, :, None] * k[:, t])[..., None] * v[:, t, :, None, :]
            rows.append((q[:, t, :, None, :] @ state)[:, :, 0])
        return torch.stack(rows, 1)

    def memory(h, p, m):
        H, d, dv, cap = m["heads"], m["dim"], m["vdim"], m["gate_cap"]
        q, k, v = (_product(h, w(p + n, H * s, D)).unflatten(-1, (H, s)) for n, s in (("q", d), ("k", d), ("v", dv)))
        q = q * d ** -0.5

        def gate(name, mean):
            return cap * torch.tanh((_product(h, w(p + name, H, D)) + w(p + name + ".b", H, mean=mean, std=1.0)) / cap)

        taken, kept = gate("i", -1.0), -_softplus(-gate("f", 3.0))
        top, tops, keep, add = torch.zeros_like(taken[:, 0]), [], [], []
        for t in range(h.shape[1]):
            new = torch.maximum(kept[:, t] + top, taken[:, t])
            keep.append(torch.exp(kept[:, t] + top - new))
            add.append(torch.exp(taken[:, t] - new))
            tops.append(new)
            top = new
        ones = torch.ones(v.shape[:3] + (1,), dtype=torch.float64, device=DEV)
        o = scan(q, k, torch.cat([v, ones], -1), torch.stack(keep, 1), torch.stack(add, 1))
        o = o[..., :dv] / (torch.maximum(o[..., dv:].abs(), torch.exp(-torch.stack(tops, 1))[..., None]) + 1e-6)
        out = _unit_rms(o, eps).flatten(2) * w(p + "norm", H * dv, mean=1.0, std=0.1)
        return _product(out * torch.sigmoid(_product(h, w(p + "g", H * dv, D))), w(p + "o", D, H * dv))

    def head_space(h, p, m):
        H, dv, N, G, taps = m["heads"], m["vdim"], m["state"], m["groups"], m["conv"]
        inner, channels = H * dv, H * dv + 2 * G * N
        z, x, dt = _product(h, w(p + "in", inner + channels + H, D)).split([inner, channels, H], dim=-1)
        x = _silu(_convolve(x, w(p + "conv", channels, taps, std=1.0 / math.sqrt(taps)), w(p + "conv.b", channels, std=0.1)))
        x, B, C = x.split([inner, G * N, G * N], dim=-1)
        x = x.unflatten(-1, (H, dv))
        B, C = (t.unflatten(-1, (G, N)).repeat_interleave(H // G, dim=2) for t in (B, C))
        dt = _softplus(dt + w(p + "dt_bias", H, mean=-2.0, std=1.0))
        y = scan(C, B, x, torch.exp(-torch.exp(w(p + "A_log", H, mean=-1.0, std=1.0)) * dt), dt) + w(p + "D", H, mean=1.0, std=0.1)[:, None] * x
        y = (y.flatten(2) * _silu(z)).unflatten(-1, (m["norm_groups"], -1))
        return _product(_unit_rms(y, eps).flatten(2) * w(p + "norm", inner, mean=1.0, std=0.1), w(p + "o", D, inner))

    def window_attention(h, p, m):
        H, G, d, dv, rot = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["rot"]
        size, first = m["mask"]["size"], m["mask"]["keep_first"]
        plain, scaling = _frequencies(rot["base"], rot["dims"]), rot["scaling"]

        def pair(times):
            return rot["dims"] * math.log(scaling["original"] / (2 * math.pi * times)) / (2 * math.log(rot["base"]))

        low, high = max(math.floor(pair(scaling["fast"])), 0), min(math.ceil(pair(scaling["slow"])), rot["dims"] - 1)
        slow = ((torch.arange(plain.numel(), dtype=torch.float64, device=DEV) - low) / max(high - low, 0.001)).clamp(0.0, 1.0)
        freq, gain = plain / scaling["factor"] * slow + plain * (1.0 - slow), 0.1 * math.log(scaling["factor"]) + 1.0
        made = []
        for name, heads, s in (("q", H, d), ("k", G, d), ("v", G, dv)):
            y = _product(h, w(p + name, heads * s, D)) + w(p + name + ".b", heads * s, std=0.1)
            if name != "v":
                y = _unit_rms(y, eps) * w(p + name + ".norm", heads * s, mean=1.0, std=0.1)
            y = y.unflatten(-1, (heads, s))
            made.append(y if name == "v" else _turn(y, freq, gain))
        out = _attend(*made, m["scale"], seen=lambda a, b: (a - b < size) | (b < first), squash=(m["softcap"], None))
        return _product(out * torch.sigmoid(_product(h, w(p + "g", H * dv, D))), w(p + "o", D, H * dv))

    def selective(h, p, m):
        inner, N, rank, taps = m["inner"], m["state"], m["dt_rank"], m["conv"]
        x, z = _product(h, w(p + "in", 2 * inner, D)).split([inner, inner], dim=-1)
        x = _silu(_convolve(x, w(p + "conv", inner, taps, std=1.0 / math.sqrt(taps)), w(p + "conv.b", inner, std=0.1)))
        low, B, C = _product(x, w(p + "x", rank + 2 * N, inner)).split([rank, N, N], dim=-1)
        dt = _softplus(_product(low, w(p + "dt", inner, rank)) + w(p + "dt.b", inner, mean=-2.0, std=1.0))
        A = -torch.exp(w(p + "A_log", inner, N, mean=0.5, std=0.7))
        state, rows = torch.zeros(h.shape[0], inner, N, dtype=torch.float64, device=DEV), []
        for t in range(h.shape[1]):
            state = torch.exp(dt[:, t, :, None] * A) * state + (dt[:, t] * x[:, t])[..., None] * B[:, t, None, :]
            rows.append((state @ C[:, t, :, None])[..., 0])
        y = torch.stack(rows, 1) + w(p + "D", inner, mean=1.0, std=0.1) * x
        return _product(y * _silu(z), w(p + "o", D, inner))

    def side_by_side(h, p, m):
        return m["left_scale"] * window_attention(h, p + "left.", m["left"]) + m["right_scale"] * selective(h, p + "right.", m["right"])

    x = w.stored("embed", vocab, D)[ids].double() * config["embedding"]["scale"]
    for i, layer in enumerate(config["layers"]):
        p = f"l{i}."
        h = _unit_rms(x, eps) * w(p + "norm1", D, mean=1.0, std=0.1)
        mixer = {"mlstm": memory, "mamba2": head_space, "parallel": side_by_side}[layer["type"]]
        x = x + w(p + "ls1", D, mean=0.5, std=0.2) * mixer(h, p + "mix.", layer["mixer"])
    return _unit_rms(x, eps) * w("final.norm", D, mean=1.0, std=0.1), w("head", vocab, D)


EXACT_AT_MOST = 3.5e14          # flops of whole sequences in 64 bits: about ten seconds


@torch.inference_mode()
def exact(case, seed):
    if case["kind"] == "sample":
        return None
    lengths, ids = _arrival(case, seed)
    longest = max(len(i) for i in ids)
    if work(dict(case, cached=False))["flops"] * longest * len(ids) / sum(len(i) for i in ids) > EXACT_AT_MOST:
        return None
    design = case["model"].split("-")[0]
    forward = {"qwen2": _qwen2, "fuvuvik": _fuvuvik, "bebulorn": _bebulorn, "ribozen": _ribozen}[design]
    config = _config(case["model"])
    # every request as a row; what follows a request's end is not seen by what comes before it
    padded = torch.tensor([i + [0] * (longest - len(i)) for i in ids], device=DEV)
    x, head = forward(config, _Weights(seed), padded)
    rows = [x[r, lengths[r] - 1:len(ids[r])] @ head.T for r in range(len(ids))]
    out = []
    for step in _schedule(case, lengths):
        out += [rows[r][a + k - lengths[r]] for r, a, k in step if _wants_logits(lengths, r, a, k)]
    _typed, plan = resolve(config)
    storages = 0 if case["cached"] else sum(1 for g in plan.cache_groups if g.kind != "state" or math.prod(g.state_shape))
    return {"logits": torch.stack(out), "cache": [None] * storages}
