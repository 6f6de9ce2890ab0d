"""What the engine's speed is measured on: the calls that serving a model makes, each through the entry point a program
uses for it, over the sizes of this repository's presets.

Kinds of case (``kind``):

* ``engine_decode``, ``engine_prompt``: a whole model through ``StepRunner.run`` (metadata, captured graph, logits);
* ``attention``: an attention layer (projections, rotation, cache store, paged attention, output product) over a flat
  batch of prompt portions (``portions``: "new+cached" tokens of each) and single decoded tokens;
* ``feed_forward``: the gated feed-forward; ``experts``: routed experts with a shared one;
* ``delta_rule``, ``state_space``: the two recurrent mixers whose state is a matrix per head, over new prompts;
* ``sample``: temperature, top-k and top-p over the logits of a step.

All tensors are drawn on the GPU from (seed, name), so that ``exact`` draws the same ones again.
"""

from __future__ import annotations

import math
import zlib
from types import SimpleNamespace

import numpy as np
import torch

from gllm_b200 import ops
from gllm_b200.cache.manager import CacheManager
from gllm_b200.config.llama_config import LlamaConfig
from gllm_b200.config.presets import load_preset
from gllm_b200.engine.step import StepEntry, StepRunner
from gllm_b200.models.decoder import DecoderModel
from gllm_b200.models.llama import build_llama_spec
from gllm_b200.models.spec import PartSpec
from gllm_b200.parts import FEED_FORWARDS, MIXERS, build_part

DEV = "cuda:0"
BLOCK = 16
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}
BYTES = {"bf16": 2, "f32": 4}
ROPE_SCALING = {"rope_type": "llama3", "factor": 32.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
                "original_max_position_embeddings": 8192}
THETA = 500000.0
STD = 0.02


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # one step of a small chat server: eight requests with about 2,000 tokens each (the benchmark's headline)
        dict(name="decode step 1B batch 8", kind="engine_decode", preset="llama-3.2-1b", batch=8, context=2048),
        # the time to a first token: one prompt of 2,048 tokens through the same model (the benchmark's prefill)
        dict(name="prompt step 1B 2048", kind="engine_prompt", preset="llama-3.2-1b", tokens=2048),
        # a busy server's attention layer: 64 requests decode over contexts of very different lengths
        dict(name="attention 64 decodes", kind="attention", dtype="bf16", hidden=2048, heads=32, kv_heads=8, dim=64,
             portions="", singles=64, context=4096),
        # a mixed step at the 8B sizes: a prompt, the second portion of another, and 30 requests that decode
        dict(name="attention mixed 8B", kind="attention", dtype="bf16", hidden=4096, heads=32, kv_heads=8, dim=128,
             portions="1531+0 517+1200", singles=30, context=3000),
        # the true 32-bit mode (trace replays): portions of two prompts beside a few single tokens
        dict(name="attention float32", kind="attention", dtype="f32", hidden=2048, heads=32, kv_heads=8, dim=64,
             portions="512+0 200+300", singles=8, context=1024),
        # the feed-forward of a decode step, where the weights' bytes are the work
        dict(name="feed-forward 8 tokens", kind="feed_forward", dtype="bf16", hidden=2048, inter=8192, tokens=8),
        # the feed-forward of a prompt portion of an odd length at the 8B sizes
        dict(name="feed-forward 1999 8B", kind="feed_forward", dtype="bf16", hidden=4096, inter=14336, tokens=1999),
        # the feed-forward of a portion in the 32-bit mode
        dict(name="feed-forward float32", kind="feed_forward", dtype="f32", hidden=2048, inter=8192, tokens=700),
        # routed experts over a portion of a prompt
        dict(name="experts 777 tokens", kind="experts", hidden=2048, inter=1024, experts=16, top=4, groups=4, kept=3,
             shared=4096, tokens=777),
        # the delta rule over two prompts and two one-token prompts
        dict(name="delta rule prompts", kind="delta_rule", hidden=2048, heads=16, dk=64, dv=128, taps=4, rank=64,
             head_decay=False, portions="1500 517 1 1"),
        # state-space duality over one whole prompt
        dict(name="state space 2048", kind="state_space", hidden=2048, heads=64, dim=64, states=128, groups=1, taps=4,
             norm_groups=1, portions="2048"),
        # the sampler behind a step of 64 requests, with the request defaults
        dict(name="sample 64 rows", kind="sample", rows=64, vocab=128256, temperature=0.7, top_k=40, top_p=0.9),
    ]


def _spread(rng, low, high):
    """A whole number of [low, high], spread over its logarithm, odd ones among them."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high + 1)))))))


def _portions(rng, most, cached):
    left, out = _spread(rng, max(16, most // 16), most), []
    for _ in range(rng.randint(1, 3)):
        if left < 2:
            break
        n = left if rng.random() < 0.4 else rng.randint(2, left)
        out.append(f"{n}+{_spread(rng, 1, cached) if rng.random() < 0.5 else 0}" if cached else str(n))
        left -= n
    return " ".join(out)


def draw(rng):
    kind = rng.choice(["engine_decode", "engine_prompt", "attention", "attention", "attention", "feed_forward",
                       "feed_forward", "experts", "delta_rule", "state_space", "sample"])
    if kind == "engine_decode":
        return dict(kind=kind, preset="llama-3.2-1b", batch=_spread(rng, 1, 32), context=_spread(rng, 64, 3000))
    if kind == "engine_prompt":
        return dict(kind=kind, preset="llama-3.2-1b", tokens=_spread(rng, 16, 2040))
    if kind == "attention":
        f32 = rng.random() < 0.25
        hidden, dim = (2048, 64) if f32 or rng.random() < 0.5 else (4096, 128)
        portions = _portions(rng, 500 if f32 else 2000, 512 if f32 else 2048) if rng.random() < 0.7 else ""
        singles = 0 if portions and rng.random() < 0.3 else _spread(rng, 1, 64)
        return dict(kind=kind, dtype="f32" if f32 else "bf16", hidden=hidden, heads=32, kv_heads=8, dim=dim,
                    portions=portions, singles=singles, context=_spread(rng, 64, 1024 if f32 else 4096))
    if kind == "feed_forward":
        f32 = rng.random() < 0.3
        hidden, inter = (2048, 8192) if f32 else rng.choice([(2048, 8192), (3072, 8192), (4096, 14336)])
        return dict(kind=kind, dtype="f32" if f32 else "bf16", hidden=hidden, inter=inter,
                    tokens=_spread(rng, 1, 700 if f32 else 2000))
    if kind == "experts":
        return dict(kind=kind, hidden=2048, inter=rng.choice([1024, 2048]), experts=16, top=4, groups=4, kept=3,
                    shared=4096, tokens=_spread(rng, 1, 2048))
    if kind == "delta_rule":
        heads = rng.choice([8, 16])
        return dict(kind=kind, hidden=128 * heads, heads=heads, dk=64, dv=128, taps=4, rank=64,
                    head_decay=rng.random() < 0.5, portions=_portions(rng, 2040, 0))
    if kind == "state_space":
        heads = rng.choice([32, 64])
        return dict(kind=kind, hidden=32 * heads, heads=heads, dim=64, states=128, groups=1, taps=4, norm_groups=1,
                    portions=_portions(rng, 2040, 0))
    return dict(kind=kind, rows=_spread(rng, 1, 128), vocab=rng.choice([32000, 128256]), temperature=rng.choice([0.7, 1.0]),
                top_k=rng.choice([0, 40, 50]), top_p=rng.choice([0.9, 0.95, 1.0]))


# ------------------------------------------------------------------ what is drawn
def _randn(seed, name, shape, std=1.0, dtype=torch.float32):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + zlib.crc32(name.encode())) % (1 << 62))
    return torch.randn(shape, generator=g, device=DEV, dtype=torch.float32).mul_(std).to(dtype)


def _uniform(seed, name, shape, low, high):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + zlib.crc32(name.encode())) % (1 << 62))
    return torch.rand(shape, generator=g, device=DEV, dtype=torch.float32) * (high - low) + low


def _weight(seed, name, shape, role, dtype):
    """A checkpoint tensor: matrices N(0, 0.02), norm weights about one, and the recurrent mixers' own tensors as such
    models start out: decay rates log U(1, 16), step-size biases the inverse softplus of 0.001 .. 0.1."""
    if name.endswith("A_log"):
        return torch.log(_uniform(seed, name, shape, 1.0, 16.0))
    if name.endswith("dt_bias"):
        dt = torch.exp(_uniform(seed, name, shape, math.log(1e-3), math.log(1e-1)))
        return dt + torch.log(-torch.expm1(-dt))
    if name.endswith("conv") or name.endswith("conv_bias"):
        return _randn(seed, name, shape, 0.3)
    if name == "D" or role == "vector":
        return 1.0 + _randn(seed, name, shape, 0.1)
    return _randn(seed, name, shape, STD, dtype if role == "matrix" else torch.float32)


class _Drawn:
    """Stands in for a checkpoint: every tensor the model expects, drawn when it is asked for."""

    def __init__(self, seed, expected):
        self.seed, self.expected = seed, expected

    def validate(self, expected, ignorable=()):
        pass

    def getter(self, dtype, device):
        def get(name, role="matrix"):
            return _weight(self.seed, name, tuple(self.expected[name].shape), role, dtype).contiguous()

        return get


def _rope_frequencies(dim):
    """fp64 rotary frequencies with the llama3 scaling of the 1B and 8B presets' kind."""
    out = []
    low, high = ROPE_SCALING["low_freq_factor"], ROPE_SCALING["high_freq_factor"]
    original, factor = ROPE_SCALING["original_max_position_embeddings"], ROPE_SCALING["factor"]
    for m in range(dim // 2):
        f = THETA ** (-2.0 * m / dim)
        wave = 2.0 * math.pi / f
        if wave < original / high:
            out.append(f)
        elif wave > original / low:
            out.append(f / factor)
        else:
            s = (original / wave - low) / (high - low)
            out.append((1.0 - s) * f / factor + s * f)
    return torch.tensor(out, dtype=torch.float64).to(torch.float32).to(DEV).double()


def _single_contexts(case):
    """The cached lengths of the single tokens: between an eighth of ``context`` and all of it."""
    n, top = case["singles"], case["context"]
    return [max(1, top - (top - top // 8) * ((i * 37) % max(n, 1)) // max(n, 1)) for i in range(n)]


def _batch_of(case):
    """(new tokens, cached tokens) of every request of an attention case, portions first."""
    parts = [tuple(int(v) for v in p.split("+")) for p in case["portions"].split()]
    return parts + [(1, c) for c in _single_contexts(case)]


def _decode_contexts(case):
    n, top = case["batch"], case["context"]
    return [top - (i * 13) % max(1, top // 8) for i in range(n)]


# ------------------------------------------------------------------ prepare
def _cached(seed, layer, r, n, kv_heads, dim, dtype):
    """Keys and values that a request already has in a layer's cache: ``[2, tokens, kv_heads, dim]``."""
    return _randn(seed, f"cache{layer}.{r}", (2, n, kv_heads, dim), 0.9, dtype)


def _fill(cache, lengths, seed, layers, kv_heads, dim, dtype):
    """Requests 0, 1, .. with ``lengths`` cached tokens each; their pages lie between one another's, as a server's do."""
    slots = [[] for _ in lengths]
    done = [0] * len(lengths)
    for r in range(len(lengths)):
        cache.add_request(r)
    while any(d < n for d, n in zip(done, lengths)):
        for r, n in enumerate(lengths):
            step = min(128, n - done[r])
            if step:
                slots[r].append(cache.append(r, step)[0])
                cache.commit(r, step)
                done[r] += step
    pool = cache.groups[0].pool
    for layer in range(layers):
        pages = pool[layer].view(pool.shape[1], 2, kv_heads, BLOCK, dim)
        for r, n in enumerate(lengths):
            if n:
                at = torch.from_numpy(np.concatenate(slots[r]).astype(np.int64)).to(DEV)
                both = _cached(seed, layer, r, n, kv_heads, dim, dtype)
                for which in range(2):
                    pages[at // BLOCK, which, :, at % BLOCK] = both[which]


def _llama(case, seed):
    raw = load_preset(case["preset"])
    config = LlamaConfig.from_dict(raw)
    model = DecoderModel(build_llama_spec(config), torch.bfloat16, torch.device(DEV))
    needs = model.kernel_needs()
    ops.prepare(model.dtype, needs.get("attention_head_dims", ()), modules=sorted(needs.get("modules", ())))
    model.load(_Drawn(seed, model.expected_tensors()))
    return config, model


def _tokens(seed, name, n, vocab):
    return _uniform(seed, name, (n,), 0.0, float(vocab) - 0.5).long().clamp(0, vocab - 1).tolist()


def _prepare_engine(case, seed):
    config, model = _llama(case, seed)
    decode = case["kind"] == "engine_decode"
    lengths = _decode_contexts(case) if decode else []
    most = max(lengths, default=0) + case.get("tokens", 0) + 64
    batch = max(8, len(lengths))
    cache = CacheManager(model.cache_requirements(), block_size=BLOCK, num_blocks=sum(-(-(n + 64) // BLOCK) for n in lengths)
                         + -(-most // BLOCK) + 8, max_batch_size=batch, max_seq_len=max(4096, most), dtype=model.dtype,
                         device=DEV)
    runner = StepRunner(model, cache, 4096, cuda_graphs=True, prefill_graph_tokens=(2048,))
    state = SimpleNamespace(case=case, kind=case["kind"], cache=cache, runner=runner, lengths=lengths)
    if decode:
        _fill(cache, lengths, seed, config.num_hidden_layers, config.num_key_value_heads, config.head_dim, model.dtype)
        state.entries = [StepEntry(r, [t], [0]) for r, t in
                         enumerate(_tokens(seed, "tokens", len(lengths), config.vocab_size))]
    else:
        state.prompt = _tokens(seed, "tokens", case["tokens"], config.vocab_size)
    run(state)                  # a server's graphs are captured by its first steps
    return state


def _one_layer(seed, table, spec, dtype):
    part = build_part(table, spec)
    needs = part.kernel_needs()
    ops.prepare(dtype, needs.get("attention_head_dims", ()), modules=sorted(needs.get("modules", ())))
    part.load(_Drawn(seed, part.expected_tensors()).getter(dtype, torch.device(DEV)), dtype, torch.device(DEV))
    return part


def _runner_for(mixer, requests, dtype):
    """The cache and the step runner that feed one mixer a batch of (new, cached) tokens per request."""
    most = max(n + c for n, c in requests)
    cache = CacheManager([(mixer.kv_requirement(), mixer.state_requirement(), None)], block_size=BLOCK,
                         num_blocks=sum(-(-(n + c) // BLOCK) for n, c in requests) + 8, max_batch_size=len(requests),
                         max_seq_len=max(4096, most), dtype=dtype, device=DEV)
    return cache, StepRunner(SimpleNamespace(device=torch.device(DEV), dtype=dtype), cache,
                             sum(n for n, _ in requests) + 64, cuda_graphs=False)


def _mixer_spec(case):
    if case["kind"] == "attention":
        rope = PartSpec("rotary", dict(head_dim=case["dim"], rotary_dim=case["dim"], theta=THETA, scaling=ROPE_SCALING))
        return PartSpec("attention", dict(hidden_size=case["hidden"], num_heads=case["heads"],
                                          num_kv_heads=case["kv_heads"], head_dim=case["dim"], position=rope),
                        {n: n for n in "qkvo"})
    if case["kind"] == "delta_rule":
        names = ("q", "k", "v", "b", "o", "q_conv", "k_conv", "v_conv", "A_log", "norm", "dt_bias") + (
            ("a", "g") if case["head_decay"] else ("a1", "a2", "g1", "g2"))
        ranks = {} if case["head_decay"] else dict(decay_rank=case["rank"], gate_rank=case["rank"])
        return PartSpec("gated_delta_rule", dict(hidden_size=case["hidden"], heads=case["heads"], kv_heads=case["heads"],
                                                 dk=case["dk"], dv=case["dv"], taps=case["taps"], eps=1e-5,
                                                 head_decay=case["head_decay"], **ranks), {n: n for n in names})
    return PartSpec("state_space_duality", dict(hidden_size=case["hidden"], heads=case["heads"], head_dim=case["dim"],
                                                states=case["states"], groups=case["groups"], taps=case["taps"],
                                                norm_groups=case["norm_groups"], eps=1e-5),
                    {n: n for n in ("in", "conv", "conv_bias", "dt_bias", "A_log", "D", "norm", "o")})


def _prepare_mixer(case, seed):
    dtype = DTYPES[case.get("dtype", "bf16")]
    mixer = _one_layer(seed, MIXERS, _mixer_spec(case), dtype)
    attention = case["kind"] == "attention"
    requests = _batch_of(case) if attention else [(int(p), 0) for p in case["portions"].split()]
    cache, runner = _runner_for(mixer, requests, dtype)
    if attention:
        _fill(cache, [c for _, c in requests], seed, 1, case["kv_heads"], case["dim"], dtype)
    _, ctx, _ = runner.build([StepEntry(r, [0] * n, []) for r, (n, _) in enumerate(requests)])
    x = _randn(seed, "x", (ctx.num_tokens, case["hidden"]), 1.0, dtype)
    return SimpleNamespace(kind=case["kind"], part=mixer, ctx=ctx, cache=cache.mixer_caches()[0], x=x, runner=runner)


def _feed_forward_spec(case):
    if case["kind"] == "feed_forward":
        return PartSpec("swiglu", dict(hidden_size=case["hidden"], intermediate_size=case["inter"]),
                        {n: n for n in ("gate", "up", "down")})
    return PartSpec("routed_experts", dict(
        hidden_size=case["hidden"], intermediate_size=case["inter"], experts=case["experts"], top=case["top"],
        groups=case["groups"], groups_kept=case["kept"], score="sigmoid", renormalize=True, correction=True,
        shared=PartSpec("swiglu", dict(hidden_size=case["hidden"], intermediate_size=case["shared"]),
                        {n: f"shared.{n}" for n in ("gate", "up", "down")})),
        {"router": "router", "correction": "correction", "expert": "e{index}.{part}"})


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("engine_decode", "engine_prompt"):
        return _prepare_engine(case, seed)
    if kind in ("attention", "delta_rule", "state_space"):
        return _prepare_mixer(case, seed)
    if kind == "sample":
        rows = case["rows"]
        full = lambda v, t: torch.full((rows,), v, dtype=t, device=DEV)  # noqa: E731
        return SimpleNamespace(
            kind=kind, logits=_randn(seed, "logits", (rows, case["vocab"]), 2.0),
            temperature=full(case["temperature"], torch.float32), top_k=full(case["top_k"], torch.int32),
            top_p=full(case["top_p"], torch.float32), counter=torch.arange(rows, dtype=torch.int32, device=DEV),
            seed=torch.arange(rows, dtype=torch.int64, device=DEV) + int(seed))
    dtype = DTYPES[case.get("dtype", "bf16")]
    part = _one_layer(seed, FEED_FORWARDS, _feed_forward_spec(case), dtype)
    ctx = SimpleNamespace(residual_sink=None)
    return SimpleNamespace(kind=kind, part=part, ctx=ctx, x=_randn(seed, "x", (case["tokens"], case["hidden"]), 1.0, dtype))


# ------------------------------------------------------------------ run
def run(state):
    if state.kind == "engine_decode":
        logits = state.runner.run(state.entries, check=False, greedy=True)
        for r, n in enumerate(state.lengths):       # the decoded tokens are dropped again
            state.cache.requests[r].num_tokens = n
        return {"logits": logits}
    if state.kind == "engine_prompt":
        logits = state.runner.run([StepEntry(0, state.prompt, [len(state.prompt) - 1])], check=False, greedy=True)
        state.runner.finish(0)
        return {"logits": logits}
    if state.kind == "sample":
        out = ops.sample(state.logits, state.temperature, state.top_k, state.top_p, state.seed, state.counter)
        return {k: out[k] for k in ("tokens", "logprobs", "num_candidates")}
    if state.kind in ("feed_forward", "experts"):
        return {"out": ops.as_tensor(state.part.forward(state.x, state.ctx))}
    if state.kind == "attention":
        out = ops.as_tensor(state.part.forward(state.x, state.ctx, state.cache))
        return {"out": out, "cache": state.cache.pages}
    for s in state.cache.states:                    # the requests are new ones
        s.zero_()
    out = ops.as_tensor(state.part.forward(state.x, state.ctx, state.cache))
    return {"out": out, "state": state.cache.states[0], "inputs": state.cache.states[1]}


# ------------------------------------------------------------------ what a pass cannot do without
def _visible(requests):
    return sum(n * c + n * (n + 1) / 2 for n, c in requests)


def work(case):
    kind, size = case["kind"], BYTES[case.get("dtype", "bf16")]
    if kind in ("engine_decode", "engine_prompt"):
        raw = load_preset(case["preset"])
        h, i, layers, vocab = raw["hidden_size"], raw["intermediate_size"], raw["num_hidden_layers"], raw["vocab_size"]
        d, hq, hkv = raw["head_dim"], raw["num_attention_heads"], raw["num_key_value_heads"]
        per_layer = h * (2 * hq + 2 * hkv) * d + 3 * h * i
        requests = [(1, n) for n in _decode_contexts(case)] if kind == "engine_decode" else [(case["tokens"], 0)]
        tokens, wanted = sum(n for n, _ in requests), len(requests)
        cached = sum(n + c for n, c in requests) * 2 * hkv * d * layers * 2
        return {"bytes": (layers * per_layer + vocab * h) * 2 + cached + wanted * vocab * 4,
                "flops": 2.0 * tokens * layers * per_layer + 2.0 * wanted * vocab * h
                + 4.0 * layers * hq * d * _visible(requests)}
    if kind == "attention":
        requests = _batch_of(case)
        tokens, h, qd, kd = sum(n for n, _ in requests), case["hidden"], case["heads"] * case["dim"], case["kv_heads"] * case["dim"]
        weights = h * (2 * qd + 2 * kd)
        return {"bytes": size * (weights + 2 * tokens * h + 2 * kd * sum(n + c for n, c in requests)),
                "flops": 2.0 * tokens * weights + 4.0 * qd * _visible(requests)}
    if kind == "feed_forward":
        weights = 3 * case["hidden"] * case["inter"]
        return {"bytes": size * (weights + 2 * case["tokens"] * case["hidden"]), "flops": 2.0 * case["tokens"] * weights}
    if kind == "experts":
        one, shared = 3 * case["hidden"] * case["inter"], 3 * case["hidden"] * case["shared"]
        used = min(case["experts"], case["tokens"] * case["top"])
        return {"bytes": 2 * (used * one + shared + 2 * case["tokens"] * case["hidden"] + case["experts"] * case["hidden"]),
                "flops": 2.0 * case["tokens"] * (case["top"] * one + shared + case["experts"] * case["hidden"])}
    if kind == "sample":
        return {"bytes": case["rows"] * (4 * case["vocab"] + 40), "flops": 0.0}
    requests = [int(p) for p in case["portions"].split()]
    tokens, h = sum(requests), case["hidden"]
    if kind == "delta_rule":
        qk, hv = case["heads"] * case["dk"], case["heads"] * case["dv"]
        low = (h * case["heads"] + h * hv) if case["head_decay"] else case["rank"] * (2 * h + qk + hv)
        weights = h * (2 * qk + 2 * hv + case["heads"]) + low
        state = case["heads"] * case["dk"] * case["dv"] + (case["taps"] - 1) * (2 * qk + hv)
        steps = 7.0 * case["heads"] * case["dk"] * case["dv"]
    else:
        inner, gn = case["heads"] * case["dim"], case["groups"] * case["states"]
        weights = h * (3 * inner + 2 * gn + case["heads"])
        state = inner * case["states"] + (case["taps"] - 1) * (inner + 2 * gn)
        steps = 5.0 * inner * case["states"]
    return {"bytes": 2 * (weights + 2 * tokens * h) + 2 * 4 * state * len(requests),
            "flops": 2.0 * tokens * weights + tokens * steps}


def tolerance(case):
    """Largest relative error between two right implementations at the same precision."""
    kind = case["kind"]
    if kind in ("engine_decode", "engine_prompt"):
        return {"rel": 0.03, "max": 0.3}
    if kind == "sample":
        return {"rel": 1e-4, "differ": 0.01}
    if case.get("dtype") == "f32":
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 0.01, "max": 0.2}


# ------------------------------------------------------------------ the same in 64 bits
def _rms(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _silu(x):
    return x * torch.sigmoid(x)


def _rotate(x, positions):
    """Rotation of ``x [n, heads, dim]`` in halves."""
    half = x.shape[-1] // 2
    angle = positions.double()[:, None] * _rope_frequencies(x.shape[-1])
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)


def _attend(x, weight, requests, seed, layer, heads, kv_heads, dim, dtype):
    """Attention of the flat batch ``x`` over cached and new keys, up to and with the output product."""
    q = (x @ weight("q").T).view(-1, heads, dim)
    k = (x @ weight("k").T).view(-1, kv_heads, dim)
    v = (x @ weight("v").T).view(-1, kv_heads, dim)
    out, at = torch.empty_like(q), 0
    for r, (n, c) in enumerate(requests):
        rows = slice(at, at + n)
        pos = torch.arange(c, c + n, device=DEV)
        qr, kr, vr = _rotate(q[rows], pos), _rotate(k[rows], pos), v[rows]
        if c:
            both = _cached(seed, layer, r, c, kv_heads, dim, dtype).double()
            kr, vr = torch.cat([both[0], kr]), torch.cat([both[1], vr])
        s = torch.einsum("nkgd,tkd->kgnt", qr.view(n, kv_heads, heads // kv_heads, dim), kr) / math.sqrt(dim)
        s.masked_fill_(torch.arange(c + n, device=DEV) > pos[:, None], -math.inf)
        out[rows] = torch.einsum("kgnt,tkd->nkgd", torch.softmax(s, -1), vr).reshape(n, heads, dim)
        at += n
    return out.reshape(x.shape[0], heads * dim) @ weight("o").T


def _exact_engine(case, seed):
    config = LlamaConfig.from_dict(load_preset(case["preset"]))
    h, d, hq, hkv = config.hidden_size, config.head_dim, config.num_attention_heads, config.num_key_value_heads
    w = lambda name, *shape: _weight(seed, name, shape, "matrix", torch.bfloat16).double()  # noqa: E731
    norm = lambda name: _weight(seed, name, (h,), "vector", None).double()  # noqa: E731
    if case["kind"] == "engine_decode":
        requests = [(1, n) for n in _decode_contexts(case)]
    else:
        requests = [(case["tokens"], 0)]
    table = _weight(seed, "model.embed_tokens.weight", (config.vocab_size, h), "matrix", torch.bfloat16)
    ids = torch.tensor(_tokens(seed, "tokens", sum(n for n, _ in requests), config.vocab_size), device=DEV)
    x = table[ids].double()
    shapes = {"q": (hq * d, h), "k": (hkv * d, h), "v": (hkv * d, h), "o": (h, hq * d)}
    for i in range(config.num_hidden_layers):
        p = f"model.layers.{i}"
        y = _rms(x, norm(f"{p}.input_layernorm.weight"), config.rms_norm_eps)
        x = x + _attend(y, lambda n: w(f"{p}.self_attn.{n}_proj.weight", *shapes[n]), requests, seed, i, hq, hkv, d,
                        torch.bfloat16)
        y = _rms(x, norm(f"{p}.post_attention_layernorm.weight"), config.rms_norm_eps)
        inter = config.intermediate_size
        gate, up = (y @ w(f"{p}.mlp.{n}_proj.weight", inter, h).T for n in ("gate", "up"))
        x = x + (_silu(gate) * up) @ w(f"{p}.mlp.down_proj.weight", h, inter).T
    rows = torch.tensor(np.cumsum([n for n, _ in requests]) - 1, device=DEV)
    y = _rms(x[rows], norm("model.norm.weight"), config.rms_norm_eps)
    return {"logits": torch.cat([y @ part.double().T for part in table.split(16384)], 1)}


def _exact_feed_forward(case, seed, x):
    dtype = DTYPES[case.get("dtype", "bf16")]
    h = case["hidden"]

    def glu(y, prefix, inter):
        gate, up = (y @ _weight(seed, prefix + n, (inter, h), "matrix", dtype).double().T for n in ("gate", "up"))
        return (_silu(gate) * up) @ _weight(seed, prefix + "down", (h, inter), "matrix", dtype).double().T

    if case["kind"] == "feed_forward":
        return {"out": glu(x, "", case["inter"])}
    experts, groups = case["experts"], case["groups"]
    score = torch.sigmoid(x @ _weight(seed, "router", (experts, h), "matrix", dtype).double().T)
    choice = score + _weight(seed, "correction", (experts,), "bias", None).double()
    by_group = choice.view(-1, groups, experts // groups)
    kept = by_group.topk(2, -1).values.sum(-1).topk(case["kept"], -1).indices
    open_ = torch.zeros(by_group.shape[:2], dtype=torch.bool, device=DEV).scatter_(1, kept, True)
    choice = by_group.masked_fill(~open_[..., None], -math.inf).reshape(-1, experts)
    picked = torch.zeros_like(score).scatter_(1, choice.topk(case["top"], -1).indices, 1.0)
    weights = score * picked
    weights = weights / weights.sum(-1, keepdim=True)
    out = glu(x, "shared.", case["shared"])
    for e in range(experts):
        rows = picked[:, e].nonzero()[:, 0]
        if rows.numel():
            out[rows] += weights[rows, e, None] * glu(x[rows], f"e{e}.", case["inter"])
    return {"out": out}


def _convolve(x, w, bias, taps):
    """Causal convolution per channel over one request's rows (zeros before them), then SiLU; and the last inputs."""
    padded = torch.cat([torch.zeros(taps - 1, x.shape[1], dtype=torch.float64, device=DEV), x])
    y = sum(padded[j:j + x.shape[0]] * w[:, j] for j in range(taps))
    return _silu(y if bias is None else y + bias), padded[padded.shape[0] - (taps - 1):]


def _exact_delta(case, seed, x):
    heads, dk, dv, h = case["heads"], case["dk"], case["dv"], case["hidden"]
    qk, hv = heads * dk, heads * dv
    w = lambda name, *shape: _weight(seed, name, shape, "matrix", torch.bfloat16).double()  # noqa: E731
    own = lambda name, *shape: _weight(seed, name, shape, "bias", None).double()  # noqa: E731
    raw = torch.cat([x @ w("q", qk, h).T, x @ w("k", qk, h).T, x @ w("v", hv, h).T], 1)
    conv = torch.cat([own("q_conv", qk, case["taps"]), own("k_conv", qk, case["taps"]), own("v_conv", hv, case["taps"])])
    beta = torch.sigmoid(x @ w("b", heads, h).T)
    rate = torch.exp(own("A_log", heads))
    if case["head_decay"]:
        step = torch.nn.functional.softplus(x @ w("a", heads, h).T + own("dt_bias", heads))
        decay = torch.exp(-rate * step)[..., None].expand(-1, -1, dk)
        gate = _silu(x @ w("g", hv, h).T)
    else:
        rank = case["rank"]
        step = torch.nn.functional.softplus((x @ w("a1", rank, h).T) @ w("a2", qk, rank).T + own("dt_bias", qk))
        decay = torch.exp(-rate[:, None] * step.view(-1, heads, dk))
        gate = torch.sigmoid((x @ w("g1", rank, h).T) @ w("g2", hv, rank).T)
    lengths = [int(p) for p in case["portions"].split()]
    state = torch.zeros(len(lengths) + 1, heads, dv, dk, dtype=torch.float64, device=DEV)
    inputs = torch.zeros(len(lengths) + 1, case["taps"] - 1, raw.shape[1], dtype=torch.float64, device=DEV)
    out, at = torch.empty(x.shape[0], heads, dv, dtype=torch.float64, device=DEV), 0
    order = sorted(range(len(lengths)), key=lambda r: lengths[r] == 1)     # single tokens lie behind the portions
    for slot, r in enumerate(order):
        n = lengths[r]
        rows = slice(at, at + n)
        y, inputs[slot] = _convolve(raw[rows], conv, None, case["taps"])
        unit = lambda t: t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6)  # noqa: E731
        q, k = unit(y[:, :qk].view(n, heads, dk)) * dk ** -0.5, unit(y[:, qk:2 * qk].view(n, heads, dk))
        v, b, g, s = y[:, 2 * qk:].view(n, heads, dv), beta[rows], decay[rows], state[slot]
        for t in range(n):
            s = s * g[t][:, None]
            u = b[t][:, None] * (v[t] - (s @ k[t][..., None])[..., 0])
            s = torch.baddbmm(s, u[..., None], k[t][:, None])
            out[at + t] = (s @ q[t][..., None])[..., 0]
        state[slot] = s
        at += n
    normed = _rms(out, _weight(seed, "norm", (dv,), "vector", None).double(), 1e-5).reshape(-1, hv) * gate
    return {"out": normed @ w("o", h, hv).T, "state": state, "inputs": inputs}


def _exact_state_space(case, seed, x):
    heads, dim, ns, groups, h = case["heads"], case["dim"], case["states"], case["groups"], case["hidden"]
    inner, gn, taps = heads * dim, groups * ns, case["taps"]
    own = lambda name, role, *shape: _weight(seed, name, shape, role, None).double()  # noqa: E731
    w_in = _weight(seed, "in", (2 * inner + 2 * gn + heads, h), "matrix", torch.bfloat16).double()
    proj = x @ w_in.T
    z, raw = proj[:, :inner], proj[:, inner:2 * inner + 2 * gn]
    step = torch.nn.functional.softplus(proj[:, 2 * inner + 2 * gn:] + own("dt_bias", "bias", heads))
    decay = torch.exp(-torch.exp(own("A_log", "vector", heads)) * step)
    conv, bias = own("conv", "vector", inner + 2 * gn, taps), own("conv_bias", "bias", inner + 2 * gn)
    lengths = [int(p) for p in case["portions"].split()]
    state = torch.zeros(len(lengths) + 1, heads, dim, ns, dtype=torch.float64, device=DEV)
    inputs = torch.zeros(len(lengths) + 1, taps - 1, inner + 2 * gn, dtype=torch.float64, device=DEV)
    out, at = torch.empty(x.shape[0], heads, dim, dtype=torch.float64, device=DEV), 0
    order = sorted(range(len(lengths)), key=lambda r: lengths[r] == 1)
    for slot, r in enumerate(order):
        n = lengths[r]
        rows = slice(at, at + n)
        y, inputs[slot] = _convolve(raw[rows], conv, bias, taps)
        xs = y[:, :inner].view(n, heads, dim)
        expand = lambda t: t.view(n, groups, 1, ns).expand(-1, -1, heads // groups, -1).reshape(n, heads, ns)  # noqa: E731
        b, c, s = expand(y[:, inner:inner + gn]), expand(y[:, inner + gn:]), state[slot]
        fed = xs * step[rows][..., None]
        for t in range(n):
            s = torch.baddbmm(s * decay[at + t][:, None, None], fed[t][..., None], b[t][:, None])
            out[at + t] = (s @ c[t][..., None])[..., 0]
        out[rows] += own("D", "vector", heads)[:, None] * xs
        state[slot] = s
        at += n
    y = (out.reshape(-1, inner) * _silu(z)).view(-1, case["norm_groups"], inner // case["norm_groups"])
    y = _rms(y, 1.0, 1e-5).reshape(-1, inner) * own("norm", "vector", inner)
    return {"out": y @ _weight(seed, "o", (h, inner), "matrix", torch.bfloat16).double().T, "state": state, "inputs": inputs}


def exact(case, seed):
    kind = case["kind"]
    if kind == "sample":            # which token is drawn hangs on the generator: nothing to state in 64 bits
        return None
    if kind in ("engine_decode", "engine_prompt"):
        return _exact_engine(case, seed)
    dtype = DTYPES[case.get("dtype", "bf16")]
    if kind in ("feed_forward", "experts"):
        x = _randn(seed, "x", (case["tokens"], case["hidden"]), 1.0, dtype).double()
        return _exact_feed_forward(case, seed, x)
    requests = _batch_of(case) if kind == "attention" else [(int(p), 0) for p in case["portions"].split()]
    x = _randn(seed, "x", (sum(n for n, _ in requests), case["hidden"]), 1.0, dtype).double()
    if kind == "delta_rule":
        return _exact_delta(case, seed, x)
    if kind == "state_space":
        return _exact_state_space(case, seed, x)
    h, qd, kd = case["hidden"], case["heads"] * case["dim"], case["kv_heads"] * case["dim"]
    shapes = {"q": (qd, h), "k": (kd, h), "v": (kd, h), "o": (h, qd)}
    out = _attend(x, lambda n: _weight(seed, n, shapes[n], "matrix", dtype).double(), requests, seed, 0, case["heads"],
                  case["kv_heads"], case["dim"], dtype)
    return {"out": out, "cache": None}
