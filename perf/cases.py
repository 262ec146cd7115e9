"""The work that this engine is timed on: steps of a served model, through the step function that the
engine, the command line and the trace replayer all run, and the sampling of a step's logits.

A case is one call of `ModelRunner.step` on a batch a server meets (single decoded tokens, whole prompts, a
portion of a prompt beside decoded tokens) or one call of `Sampler.sample`. Weights, caches and token ids
are random, made from the seed: gains 1 + N(0, 0.1), matrices N(0, 0.02), the embedding N(0, 1) and the last
matrix of a feed-forward smaller by the root of twice the depth, which leave projections, scores and logits
with the spread that a trained model's have and let a layer add to the stream rather than replace it; the
keys and values of earlier tokens N(0, 1), as the per-head norm leaves the keys. The models are Qwen3, the architecture that has checkpoints to
serve: the layer sizes of its 8B, 14B and 32B models (14B and 32B with fewer layers, all alike, so that
several fit one device) and the tests' small one.

`exact` computes a case again in float64 with plain tensor operations.
"""

from __future__ import annotations

import math
import zlib

import numpy as np
import torch

DEVICE = "cuda"

QWEN3 = {  # hidden, heads, kv heads, head size, feed-forward, vocabulary, all layers, page size
    "8b": (4096, 32, 8, 128, 12288, 151936, 36, 16),
    "14b": (5120, 40, 8, 128, 17408, 151936, 40, 16),
    "32b": (5120, 64, 8, 128, 25600, 151936, 64, 16),
    "tiny": (96, 6, 3, 32, 224, 512, 3, 8),
}
# (temperature, top-k, top-p): the engine's default, nucleus sampling over the whole vocabulary, greedy
SETTINGS = {"default": (0.6, 20, 0.95), "nucleus": (0.8, 0, 0.95), "greedy": (0.0, 0, 1.0)}


def listed():
    def case(name, **rest):
        return dict(name=name, **rest)

    return [
        # the smallest step there is: three tiny layers in float32, bound by launches and latency
        case("tiny decode 4", kind="qwen3", model="tiny", layers=3, dtype="float32", decodes=4, low=17, high=40, prompts=0, tokens=0, start=0),
        # one person's chat: one request decoding on the whole 8B model
        case("8B decode 1", kind="qwen3", model="8b", layers=36, dtype="bfloat16", decodes=1, low=2048, high=2048, prompts=0, tokens=0, start=0),
        # the engine's headline: eight requests at one context
        case("8B decode 8", kind="qwen3", model="8b", layers=36, dtype="bfloat16", decodes=8, low=2048, high=2048, prompts=0, tokens=0, start=0),
        # a full server: 64 requests of all lengths
        case("8B decode 64", kind="qwen3", model="8b", layers=36, dtype="bfloat16", decodes=64, low=300, high=3000, prompts=0, tokens=0, start=0),
        # long conversations on the largest shape: eight query heads a kv head, the cache as large as the weights
        case("32B decode long", kind="qwen3", model="32b", layers=6, dtype="bfloat16", decodes=13, low=6000, high=12000, prompts=0, tokens=0, start=0),
        # a whole prompt in one step
        case("8B prompt 2048", kind="qwen3", model="8b", layers=36, dtype="bfloat16", decodes=0, low=0, high=0, prompts=1, tokens=2048, start=0),
        # short questions arriving together
        case("8B short prompts", kind="qwen3", model="8b", layers=36, dtype="bfloat16", decodes=0, low=0, high=0, prompts=3, tokens=117, start=0),
        # chunked prefill: a portion of a long prompt beside 32 decoding requests, the budget of 512 full
        case("14B portion and decodes", kind="qwen3", model="14b", layers=12, dtype="bfloat16", decodes=32, low=400, high=1800, prompts=1, tokens=480, start=960),
        # a portion deep in a long prompt, at the default budget, with nothing beside it
        case("8B portion at 7000", kind="qwen3", model="8b", layers=36, dtype="bfloat16", decodes=0, low=0, high=0, prompts=1, tokens=512, start=7000),
        # the float32 path that checks the other one, at full width
        case("8B float32", kind="qwen3", model="8b", layers=2, dtype="float32", decodes=0, low=0, high=0, prompts=1, tokens=300, start=0),
        # drawing the next token of 48 requests whose clients ask for different settings
        case("sampling 48", kind="sample", vocab=151936, rows=48, settings="default nucleus greedy"),
    ]


def draw(rng):
    """One more case: sizes by their logarithm over what a server of these models meets, up to the listed largest."""

    def spread(low, high):
        return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high + 0.49)))))))

    def qwen3(model, layers, dtype="bfloat16", decodes=0, low=0, high=0, prompts=0, tokens=0, start=0):
        return dict(kind="qwen3", model=model, layers=layers, dtype=dtype, decodes=decodes, low=low, high=high, prompts=prompts, tokens=tokens, start=start)

    what = rng.choice(["decode", "decode", "decode", "decode", "prompt", "prompt", "mixed", "mixed", "tiny", "float32", "sample"])
    if what == "decode":
        model, layers = rng.choice([("8b", 36), ("8b", 36), ("14b", 12), ("32b", 6)])
        batch = spread(1, 64)
        high = spread(64, min(12000, 90000 // batch))
        return qwen3(model, layers, decodes=batch, low=rng.randint(max(1, high // 8), high), high=high)
    if what == "prompt":
        prompts = rng.choice([1, 1, 2, 3, 5])
        return qwen3("8b", 36, prompts=prompts, tokens=spread(9, 2048 // prompts))
    if what == "mixed":  # a portion of a longer prompt, alone or beside decoding requests
        model, layers = rng.choice([("8b", 36), ("14b", 12)])
        high = spread(100, 2000)
        return qwen3(model, layers, decodes=rng.choice([0, spread(1, 32)]), low=rng.randint(high // 4, high), high=high, prompts=1,
                     tokens=spread(16, 512), start=spread(1, 7000))  # fmt: skip
    if what == "tiny":
        high = rng.randint(2, 120)
        return qwen3("tiny", 3, dtype=rng.choice(["float32", "bfloat16"]), decodes=spread(1, 24), low=rng.randint(1, high), high=high)
    if what == "float32":
        if rng.random() < 0.5:
            return qwen3("8b", 2, dtype="float32", prompts=1, tokens=spread(9, 300))
        return qwen3("8b", 2, dtype="float32", decodes=spread(1, 16), low=100, high=rng.randint(100, 1500))
    return dict(kind="sample", vocab=rng.choice([32000, 151936]), rows=spread(1, 64), settings=rng.choice(["default", "nucleus", "default nucleus", "default greedy"]))


# ---- what is made from the seed, for the engine and for `exact` alike ------------------------------


def _lengths(count, low, high):
    """`count` contexts spread over [low, high], in no order of size."""
    return [int(round(low + (high - low) * ((i * 0.6180339887 + 0.5) % 1.0))) for i in range(count)]


def _generator(seed, name):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(zlib.crc32(f"{seed}:{name}".encode()) + (int(seed) << 33))
    return g


def _normal(seed, name, shape, dtype):
    return torch.randn(shape, generator=_generator(seed, name), device=DEVICE, dtype=dtype)


def _weight(case, seed, name, shape):
    """A matrix (values that bfloat16 holds) or a vector of gains (float32)."""
    if len(shape) == 1:
        return 1.0 + 0.1 * _normal(seed, name, shape, torch.float32)
    t = _normal(seed, name, shape, torch.bfloat16)
    if "embed_tokens" in name:
        return t
    std = 0.1 if case["model"] == "tiny" else 0.02
    return t.mul_(std / math.sqrt(2 * case["layers"]) if "down_proj" in name else std)


class _Weights:
    """The model's tensors by name, each made when it is asked for."""

    def __init__(self, specs, case, seed):
        self.specs, self.case, self.seed = {s.name: s for s in specs}, case, seed

    def __getitem__(self, name):
        spec = self.specs[name]
        t = _weight(self.case, self.seed, name, tuple(spec.shape))
        return t.to(getattr(torch, self.case["dtype"]) if spec.kind == "matrix" else torch.float32)


def _tokens(seed, name, count, vocab):
    return torch.randint(0, vocab, (count,), generator=_generator(seed, name), device=DEVICE).tolist()


def _pieces(case):
    """The rows of a step: (name, position it starts at, new tokens), decodes first."""
    rows = [(f"decode{i}", n, 1) for i, n in enumerate(_lengths(case["decodes"], case["low"], case["high"]))]
    sizes = [case["tokens"] - (i * case["tokens"]) // 7 for i in range(case["prompts"])]  # prompts of several lengths
    return rows + [(f"prompt{i}", case["start"], n) for i, n in enumerate(sizes)]


def _past(case, seed, layer, which, count):
    """Keys or values of all earlier tokens of all rows of one layer, [count, kv heads, head size]."""
    _, _, kv, hd, *_ = QWEN3[case["model"]]
    dtype = getattr(torch, case["dtype"])
    return _normal(seed, f"past {which} {layer}", (count, kv, hd), dtype)


def _qwen3_config(case):
    hidden, heads, kv, hd, ff, vocab, _, _ = QWEN3[case["model"]]
    return dict(architectures=["Qwen3ForCausalLM"], vocab_size=vocab, hidden_size=hidden, intermediate_size=ff, num_hidden_layers=case["layers"],
                num_attention_heads=heads, num_key_value_heads=kv, head_dim=hd, rms_norm_eps=1e-6, rope_theta=1000000.0,
                tie_word_embeddings=False, max_position_embeddings=40960)  # fmt: skip


# ---- the engine ------------------------------------------------------------------------------------


def _engine(case, seed, tokens, requests):
    from atomserve_b200.config import EngineConfig
    from atomserve_b200.config.registry import config_from_dict
    from atomserve_b200.engine.engine import create_engine
    from atomserve_b200.parts.model import build_model

    arch, config = config_from_dict(_qwen3_config(case))
    model = build_model(arch.build_spec(config))
    model.load(_Weights(model.tensor_specs(), case, seed))
    block_size = QWEN3[case["model"]][7]
    blocks = tokens // block_size + requests + 1
    limits = EngineConfig(block_size=block_size, num_blocks=blocks, max_num_seqs=requests, max_num_batched_tokens=4096,
                          max_model_len=blocks * block_size, enable_prefix_caching=False)  # fmt: skip
    return create_engine(model, limits, sampler_seed=0)


def _new_request(cache, tokens):
    rc = cache.new_request()
    if not (cache.admit(rc) and cache.reserve(rc, 0, tokens)):
        raise RuntimeError("the cache was made too small for the case")
    return rc


def prepare(case, seed):
    if case["kind"] == "sample":
        return _prepare_sampling(case, seed)
    from atomserve_b200.engine.runner import Row

    block_size = QWEN3[case["model"]][7]
    pieces = _pieces(case)
    engine = _engine(case, seed, sum(s + n for _, s, n in pieces), len(pieces))
    runner, cache = engine.runner, engine.runner.cache
    rows, fresh, blocks, offsets = [], [], [], []
    for name, start, n in pieces:
        tokens = _tokens(seed, name, n, QWEN3[case["model"]][5])
        if start == 0:  # a whole prompt: it comes as a new request each time
            fresh.append(tokens)
            continue
        rc = _new_request(cache, start + n)
        rows.append(Row(tokens, start, rc, [n - 1]))
        at = torch.arange(start)
        blocks.append(torch.tensor(rc.block_table)[at // block_size])
        offsets.append(at % block_size)
    if blocks:  # the keys and values of the tokens before the step
        block, offset = torch.cat(blocks).to(DEVICE), torch.cat(offsets).to(DEVICE)
        for layer in range(case["layers"]):
            pages = runner.views[layer].pages
            for which in ("k", "v"):
                pages[which][block, :, offset] = _past(case, seed, layer, which, len(block))
    return dict(case=case, runner=runner, cache=cache, rows=rows, fresh=fresh)


def _prepare_sampling(case, seed):
    from atomserve_b200.engine.sequence import SamplingParams, Sequence
    from atomserve_b200.sampling.sampler import Sampler

    kinds = case["settings"].split()
    seqs = []
    for i in range(case["rows"]):
        temperature, top_k, top_p = SETTINGS[kinds[i % len(kinds)]]
        seqs.append(Sequence(i, [1] * (4 + i), SamplingParams(temperature=temperature, top_k=top_k, top_p=top_p, seed=1000 * int(seed) + i), 3))
    logits = _normal(seed, "logits", (case["rows"], case["vocab"]), torch.float32) * 3.0
    return dict(case=case, sampler=Sampler(DEVICE, 0), logits=logits, seqs=seqs)


def run(state):
    """The step's logits, and what it left in the last layer's cache; or the sampled token ids."""
    case = state["case"]
    if case["kind"] == "sample":
        return np.asarray(state["sampler"].sample(state["logits"], state["seqs"]))
    runner, cache = state["runner"], state["cache"]
    rows, new = state["rows"], []
    if state["fresh"]:
        from atomserve_b200.engine.runner import Row

        new = [Row(tokens, 0, _new_request(cache, len(tokens)), [len(tokens) - 1]) for tokens in state["fresh"]]
        rows = rows + new
    logits = runner.step(rows)
    for row in new:  # the request has ended
        cache.free(row.cache)
    last = runner.views[case["layers"] - 1]
    return dict(logits=logits, pages=dict(last.pages))


# ---- what a pass cannot do without -----------------------------------------------------------------


def work(case):
    if case["kind"] == "sample":
        return {"bytes": 4.0 * case["rows"] * case["vocab"] + 4.0 * case["rows"], "flops": 0.0}
    hidden, heads, kv, hd, ff, vocab, _, _ = QWEN3[case["model"]]
    size = 2 if case["dtype"] == "bfloat16" else 4
    per_layer = hidden * (heads + 2 * kv) * hd + heads * hd * hidden + 3 * hidden * ff
    pieces = _pieces(case)
    new = sum(n for _, _, n in pieces)
    pairs = sum(n * s + n * (n + 1) // 2 for _, s, n in pieces)
    cache = 2 * kv * hd * case["layers"] * sum(s + n for _, s, n in pieces)
    weights = case["layers"] * per_layer
    return {
        "bytes": size * (weights + hidden * vocab + cache + new * hidden) + 4.0 * vocab * len(pieces),
        "flops": 2.0 * weights * new + 2.0 * hidden * vocab * len(pieces) + 4.0 * heads * hd * pairs * case["layers"],
    }


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    if case["dtype"] == "bfloat16":
        return {"rel": 0.03, "max": 0.5}
    return {"rel": 2e-5, "max": 4e-4}


# ---- the same in float64 ---------------------------------------------------------------------------

F64 = torch.float64


def exact(case, seed):
    if case["kind"] == "sample":
        return None  # the rows' draws are whole numbers
    with torch.inference_mode():
        return dict(logits=_exact_qwen3(case, seed), pages=dict.fromkeys(("k", "v")))


def _rms(x, eps=1e-6):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _turn_halves(x, positions, base):
    """x [T, heads, dim]: entry i is paired with entry i + dim / 2 and the pair turned by position * base^(-2 i / dim)."""
    half = x.shape[-1] // 2
    freq = base ** (-2.0 * torch.arange(half, dtype=F64, device=x.device) / x.shape[-1])
    angle = positions.to(F64)[:, None, None] * freq
    c, s = torch.cos(angle), torch.sin(angle)
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _attend(q, k, v, positions, scale):
    """q [n, H, d] at `positions`, k and v [S, KV, d] of positions 0 .. S - 1; [n, H, d]. 256 queries at a time."""
    group = q.shape[1] // k.shape[1]
    key_at = torch.arange(k.shape[0], device=q.device)
    out = []
    for qs, ps in zip(q.split(256), positions.split(256)):
        s = torch.einsum("tgud,sgd->guts", qs.unflatten(1, (-1, group)), k) * scale
        seen = key_at[None] <= ps[:, None]
        s = s.masked_fill_(~seen, -math.inf)
        p = torch.softmax(s, -1)
        out.append(torch.einsum("guts,sgd->tgud", p, v).flatten(1, 2))
    return torch.cat(out)


def _exact_qwen3(case, seed):
    hidden, heads, kv, hd, ff, vocab, _, _ = QWEN3[case["model"]]
    pieces = _pieces(case)

    def w(name, *shape):
        return _weight(case, seed, name, shape).to(F64)

    tokens = [t for name, _, n in pieces for t in _tokens(seed, name, n, vocab)]
    positions = torch.cat([torch.arange(s, s + n, device=DEVICE) for _, s, n in pieces])
    x = _weight(case, seed, "model.embed_tokens.weight", (vocab, hidden))[torch.tensor(tokens, device=DEVICE)].to(F64)
    earlier = sum(s for _, s, _ in pieces)
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        h = _rms(x) * w(p + "input_layernorm.weight", hidden)
        q = (h @ w(p + "self_attn.q_proj.weight", heads * hd, hidden).T).view(-1, heads, hd)
        k = (h @ w(p + "self_attn.k_proj.weight", kv * hd, hidden).T).view(-1, kv, hd)
        v = (h @ w(p + "self_attn.v_proj.weight", kv * hd, hidden).T).view(-1, kv, hd)
        q = _turn_halves(_rms(q) * w(p + "self_attn.q_norm.weight", hd), positions, 1e6)
        k = _turn_halves(_rms(k) * w(p + "self_attn.k_norm.weight", hd), positions, 1e6)
        past_k, past_v = (_past(case, seed, i, which, earlier) for which in ("k", "v")) if earlier else (k[:0], v[:0])
        out, at, behind = [], 0, 0
        for _, s, n in pieces:
            ks, vs = (torch.cat([past[behind : behind + s].to(F64), t[at : at + n]]) for past, t in ((past_k, k), (past_v, v)))
            out.append(_attend(q[at : at + n], ks, vs, positions[at : at + n], hd**-0.5))
            at, behind = at + n, behind + s
        x = x + torch.cat(out).flatten(1) @ w(p + "self_attn.o_proj.weight", hidden, heads * hd).T
        h = _rms(x) * w(p + "post_attention_layernorm.weight", hidden)
        gate, up = h @ w(p + "mlp.gate_proj.weight", ff, hidden).T, h @ w(p + "mlp.up_proj.weight", ff, hidden).T
        x = x + (gate * torch.sigmoid(gate) * up) @ w(p + "mlp.down_proj.weight", hidden, ff).T
    ends = torch.tensor([n for _, _, n in pieces], device=DEVICE).cumsum(0) - 1
    h = _rms(x[ends]) * w("model.norm.weight", hidden)
    head = _weight(case, seed, "lm_head.weight", (vocab, hidden))
    return torch.cat([h @ part.to(F64).T for part in head.split(16384)], 1)
