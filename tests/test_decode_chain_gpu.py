"""The projections from one layer's attention to the next one's as one kernel, against plain products with the same
roundings."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(tokens, hidden, attn_k, ff, next_rows, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, std=1.0):
        return (torch.randn(*shape, generator=g, device="cuda") * std).bfloat16()

    gains = [1 + 0.1 * torch.randn(hidden, generator=g, device="cuda") for _ in range(2)]
    return dict(attn=normal(tokens, attn_k), o=normal(hidden, attn_k, std=attn_k**-0.5), x=normal(tokens, hidden), gains=gains,
                gate=normal(ff, hidden, std=hidden**-0.5), up=normal(ff, hidden, std=hidden**-0.5),
                down=normal(hidden, ff, std=ff**-0.5), proj=normal(next_rows, hidden, std=hidden**-0.5) if next_rows else None)  # fmt: skip


def _normed_product(x, gain, eps, *matrices):
    """N(x) . w^T in float64: the operand is x times the gain rounded to bfloat16, the norm's factor multiplies the sums."""
    d = torch.float64
    factor = torch.rsqrt((x.to(d) ** 2).mean(-1, keepdim=True) + eps)
    operand = (x.float() * gain).bfloat16().to(d)
    return [factor * (operand @ w.to(d).T) for w in matrices]


def _plain(v, eps):
    """Every stored value rounded to bfloat16 once, all else in float64."""
    d = torch.float64
    x1 = (v["attn"].to(d) @ v["o"].to(d).T + v["x"].to(d)).bfloat16()
    gate, up = _normed_product(x1, v["gains"][0], eps, v["gate"], v["up"])
    act = (torch.nn.functional.silu(gate) * up).bfloat16()
    x2 = (act.to(d) @ v["down"].to(d).T + x1.to(d)).bfloat16()
    return x2, (_normed_product(x2, v["gains"][1], eps, v["proj"])[0].bfloat16() if v["proj"] is not None else None)


def _close(got, want):
    # A stored value may be the neighbour of the plain one where the sum lies at a rounding boundary (float32 sums against
    # float64: one element in a few thousand); each such step of 2^-8 in x1 or the gated values moves the products behind it
    # by far less than their own rounding, 2^-9 of a value at most: 4e-3 of the norm holds both, with room for neither wrong
    # rows, nor wrong tokens, nor a product left out.
    got, want = got.double(), want.double()
    assert torch.isfinite(got).all()
    assert (got - want).norm() <= 4e-3 * want.norm()
    assert (got - want).abs().max() <= 2**-6 * want.abs().max()


# rows a block: fewer than blocks, a part of a row tile, one tile and a part, several passes; K of one step and of several
@pytest.mark.parametrize("hidden,attn_k,ff,next_rows", [
    (512, 512, 512, 130), (1024, 2048, 1536, 1536), (4096, 4096, 12288, 6144), (5120, 8192, 25600, 10240), (2048, 512, 6144, 0),
])  # fmt: skip
@pytest.mark.parametrize("tokens", [1, 2, 3, 7, 8])
def test_against_plain_products(hidden, attn_k, ff, next_rows, tokens):
    from atomserve_b200 import ops
    from atomserve_b200.ops.linear import check_gemm_status

    v = _inputs(tokens, hidden, attn_k, ff, next_rows, seed=tokens)
    gate_up = ops.interleave_gate_up(v["gate"], v["up"])
    assert ops.decode_chain_takes(v["x"], v["o"], gate_up, v["down"])
    want = _plain(v, 1e-6)
    for _ in range(2):  # (what a call leaves behind is not met by the next)
        got = ops.decode_chain(v["attn"], v["o"], v["x"], v["gains"][0], 1e-6, gate_up, v["down"], torch.zeros(4, dtype=torch.int32, device="cuda"),
                               next_gain=v["gains"][1], next_eps=1e-6, next_proj=v["proj"])  # fmt: skip
        check_gemm_status()
        _close(got[0], want[0])
        assert (got[1] is None) == (next_rows == 0)
        if next_rows:
            _close(got[1], want[1])


# 2 to 18 pairs of rows a block in the sums of squares: one thread a pair, several threads and several warps of a token. (The
# sums are read too: a factor that differs in its last bit changes one bfloat16 value in some ten thousand.)
@pytest.mark.parametrize("hidden", [512, 1024, 4096, 5120])
def test_a_row_does_not_depend_on_the_others(hidden):
    from atomserve_b200.ops.library import check, lib, ptr, stream
    from atomserve_b200.ops.linear import check_gemm_status, gemm_status
    from atomserve_b200 import ops

    attn_k, ff, next_rows = 2048, 1536, 1536
    v = _inputs(8, hidden, attn_k, ff, next_rows)
    gate_up = ops.interleave_gate_up(v["gate"], v["up"])
    blocks = lib().asb_decode_chain_blocks()

    def run(rows):
        attn, x = v["attn"][rows].contiguous(), v["x"][rows].contiguous()
        T = x.shape[0]
        x1, x2, act, out = (torch.empty(T, n, device="cuda", dtype=torch.bfloat16) for n in (hidden, hidden, ff, next_rows))
        squares, arrived = torch.empty(2, T, blocks, device="cuda"), torch.zeros(4, dtype=torch.int32, device="cuda")
        check(lib().asb_decode_chain(
            ptr(attn), ptr(v["o"]), ptr(x), ptr(x1), ptr(v["gains"][0]), 1e-6, ptr(gate_up), ptr(act), ptr(v["down"]), ptr(x2),
            ptr(v["gains"][1]), 1e-6, ptr(v["proj"]), ptr(out), ptr(squares), ptr(arrived), T, hidden, attn_k, ff, next_rows,
            ptr(gemm_status(x.device)), stream()))  # fmt: skip
        check_gemm_status()
        return x1, act, x2, out, squares[0], squares[1]

    whole = run(slice(0, 8))
    for rows in (slice(0, 1), slice(7, 8), slice(2, 4), slice(2, 5), slice(1, 5), slice(3, 8)):
        for part, all_rows in zip(run(rows), whole):
            assert torch.equal(part, all_rows[rows])


def test_what_lies_between_16_byte_boundaries_goes_to_the_separate_kernels():
    """A stream or a gain that does not begin on one, as a slice of a longer tensor may, in a block wide enough that the
    separate kernels take it."""
    from atomserve_b200 import ops
    from atomserve_b200.ops.linear import check_gemm_status
    from atomserve_b200.parts.attention import GQAttention
    from atomserve_b200.parts.base import StepContext
    from atomserve_b200.parts.block import PreNormBlock
    from atomserve_b200.parts.mlp import SwiGLU
    from atomserve_b200.parts.norms import RMSNorm

    tokens, hidden, heads, hd, ff = 3, 8704, 4, 128, 512
    v = _inputs(tokens, hidden, heads * hd, ff, 0)

    def shifted(t):  # the same values one element further on
        return torch.cat([t.new_zeros(1), t.flatten()])[1:].view(t.shape)

    attention = GQAttention(hidden, "", heads, heads, hd, None)
    attention.o_proj = v["o"]
    mlp = SwiGLU(hidden, "", ff)
    mlp.load({"gate_proj.weight": v["gate"], "up_proj.weight": v["up"], "down_proj.weight": v["down"]})
    norms = [RMSNorm(hidden, "", 1e-6) for _ in range(2)]
    block = PreNormBlock(attention, mlp, *norms)
    ids = torch.zeros(tokens, dtype=torch.int32, device="cuda")
    ctx = StepContext(tokens, tokens, ids, ids, ids, ids, ids, ids, 1)
    attention.attend = lambda h, ctx, cache, write_cache: v["attn"]
    want = _plain(v, 1e-6)[0]
    for x, gain in ((v["x"], v["gains"][0]), (shifted(v["x"]), v["gains"][0]), (v["x"], shifted(v["gains"][0]))):
        norms[0].gain, norms[1].gain = v["gains"][1], gain
        aligned = x is v["x"] and gain is v["gains"][0]
        assert ops.decode_chain_takes(x, v["o"], mlp.gate_up_proj, v["down"], gain) == aligned
        got = block.forward(x, ctx, None)
        check_gemm_status()
        _close(got, want)
        if not aligned:
            with pytest.raises(ops.KernelLibraryError):
                ops.decode_chain(v["attn"], v["o"], x, gain, 1e-6, mlp.gate_up_proj, v["down"], torch.zeros(4, dtype=torch.int32, device="cuda"))
    strided = torch.stack([v["x"], v["x"]], dim=1)[:, 0]
    assert not ops.decode_chain_takes(strided, v["o"], mlp.gate_up_proj, v["down"], v["gains"][0])


LAYERS = 66  # more than the calls whose counters are zeroed together


def _model(dtype, schedule):
    import dataclasses

    import plain_qwen3 as plain
    from atomserve_b200.config.registry import config_from_dict
    from atomserve_b200.parts import build_model

    cfg = dict(architectures=["Qwen3ForCausalLM"], vocab_size=384, hidden_size=512, intermediate_size=1024, num_hidden_layers=LAYERS,
               num_attention_heads=4, num_key_value_heads=2, head_dim=128, rms_norm_eps=1e-6, rope_theta=1e6, tie_word_embeddings=False,
               max_position_embeddings=512)  # fmt: skip
    arch, config = config_from_dict(cfg)
    model = build_model(dataclasses.replace(arch.build_spec(config), schedule=schedule))
    w = plain.random_checkpoint(cfg, 4)
    model.load({s.name: (w[s.name] if s.kind == "gain" else w[s.name].bfloat16().to(dtype)).cuda() for s in model.tensor_specs()})
    return model


def _steps(model):
    """Logits of steps of a model: prompts, then single tokens of three requests (from a graph, three times the same step),
    a portion of five tokens beside two single ones, eight tokens of one request, and one token."""
    from atomserve_b200.config import EngineConfig
    from atomserve_b200.engine.engine import create_engine
    from atomserve_b200.engine.runner import Row

    engine = create_engine(model, EngineConfig(block_size=16, num_blocks=32, max_num_seqs=4, max_num_batched_tokens=64, max_model_len=256))
    runner, cache = engine.runner, engine.runner.cache
    requests, at = [cache.new_request() for _ in range(3)], [0, 0, 0]
    for rc in requests:
        assert cache.admit(rc) and cache.reserve(rc, 0, 64)
    g, logits = torch.Generator().manual_seed(9), []

    def step(lengths, times=1):
        rows = [Row(torch.randint(0, 384, (n,), generator=g).tolist(), at[i], requests[i], list(range(n))) for i, n in lengths]
        got = [runner.step(rows).clone() for _ in range(times)]
        assert all(torch.equal(got[0], again) for again in got)
        for i, n in lengths:
            at[i] += n
        logits.append(got[0])

    step([(0, 20), (1, 13), (2, 17)])
    step([(0, 1), (1, 1), (2, 1)], times=3)
    step([(0, 1), (1, 1), (2, 1)], times=3)
    step([(1, 5), (0, 1), (2, 1)], times=2)
    step([(2, 8)])
    step([(0, 1)], times=3)
    return logits


def test_a_model_with_and_without_the_chain(monkeypatch):
    """A model of more layers than share one zeroing of counters, two of which read another one's keys and values, through
    the runner, eagerly and from graphs. Both forms are draws of the same rounding noise around the float32 path: the chain's
    may be at most twice the other's, a step's error measured over all its logits (thousands of values)."""
    from atomserve_b200 import ops
    from atomserve_b200.ops import chain
    from atomserve_b200.ops.linear import check_gemm_status
    from atomserve_b200.parts import LayerCall

    schedule = tuple(LayerCall(i, cache_from={10: 9, 21: 9}.get(i)) for i in range(LAYERS))
    exact = _steps(_model(torch.float32, schedule))
    model, calls, run = _model(torch.bfloat16, schedule), [], ops.decode_chain
    monkeypatch.setattr(ops, "decode_chain", lambda *args, **kwargs: calls.append(kwargs["next_proj"]) or run(*args, **kwargs))
    with_chain = _steps(model)
    check_gemm_status()
    # the graphs' two shapes are run once for warming up and once captured; of the last layer nothing is handed on
    eager, captured = 3, 2 * 2
    assert len(calls) == LAYERS * (eager + captured) and sum(p is None for p in calls) == eager + captured
    assert {p.shape[0] for p in calls if p is not None} == {4 * 128, 8 * 128}
    calls.clear()
    monkeypatch.setattr(chain, "CHAIN", False)
    without = _steps(model)
    assert not calls
    for got, other, want in zip(with_chain, without, exact):
        error, allowed = (got - want).norm(), (other - want).norm()
        assert torch.isfinite(got).all() and error <= 2 * allowed, (error / want.norm(), allowed / want.norm())
    assert torch.equal(with_chain[0], without[0])  # (more tokens than the chain takes)
