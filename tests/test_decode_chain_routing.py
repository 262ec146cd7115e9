"""Which blocks hand their products to `ops.decode_chain`, and what travels from one to the next (no GPU: every operation is
plain float64 here, and attention a stand-in that reads what the entry keeps)."""

import pytest
import torch

from atomserve_b200 import ops
from atomserve_b200.parts import LayerCall, LayerSpec, ModelSpec, PartSpec, StepContext, register_part
from atomserve_b200.parts.attention import GQAttention
from atomserve_b200.parts.base import ProjectedInput, StreamStep
from atomserve_b200.parts.block import PreNormBlock
from atomserve_b200.parts.mlp import SwiGLU
from atomserve_b200.parts.model import DecoderModel
from atomserve_b200.parts.norms import RMSNorm

import toy_parts  # noqa: F401  (registers torch_embedding and torch_head)

HIDDEN, HEADS, KV, HEAD, FF, VOCAB, EPS = 16, 3, 1, 8, 24, 11, 1e-5


def _rms_norm(x, gain, eps, rows=None):
    x = x if rows is None else x[rows.long()]
    return gain * x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _attend(self, h, ctx, cache, write_cache):
    wide = HEADS * HEAD
    weight = self.qkv_proj if write_cache else self.qkv_proj[:wide]
    product = h.product if isinstance(h, ProjectedInput) else h @ weight.T
    assert product.shape[1] == weight.shape[0]
    if write_cache:
        cache.kept = product[:, wide:].mean(1, keepdim=True)
    return torch.tanh(product[:, :wide] + cache.kept)


class Chain:
    """The place of `ops.decode_chain`: calls are counted, and matrices in `refused` not taken."""

    def __init__(self):
        self.calls, self.handed_on, self.counters, self.refused = 0, 0, [], []

    def takes(self, x, *matrices):
        return x.shape[0] <= 8 and not any(w is r or w.data_ptr() == r.data_ptr() for w in matrices for r in self.refused)

    def run(self, attn, o_proj, x, gain, eps, gate_up, down, arrived, next_gain=None, next_eps=0.0, next_proj=None):
        assert arrived.shape == (4,) and arrived.dtype == torch.int32 and not arrived.any()
        arrived += 1  # as the kernel leaves them
        self.counters.append(arrived)
        self.calls += 1
        self.handed_on += next_proj is not None
        x1 = attn @ o_proj.T + x
        x2 = _swiglu(_rms_norm(x1, gain, eps), gate_up) @ down.T + x1
        return x2, (None if next_proj is None else _rms_norm(x2, next_gain, next_eps) @ next_proj.T)


def _swiglu(h, interleaved):
    both = h @ interleaved.T
    return torch.nn.functional.silu(both[:, ::2]) * both[:, 1::2]


@pytest.fixture
def chain(monkeypatch):
    chain = Chain()
    plain = dict(
        rms_norm=_rms_norm, linear_swiglu=_swiglu, linear_partial=lambda x, w: None, partial_add_rms_norm_fusable=lambda width: False,
        linear=lambda x, w, residual=None, **_: x @ w.T + (0 if residual is None else residual),
        decode_chain=chain.run, decode_chain_takes=chain.takes,
    )  # fmt: skip
    for name, function in plain.items():
        monkeypatch.setattr(ops, name, function)
    monkeypatch.setattr(GQAttention, "attend", _attend)
    return chain


def _model(layers, schedule=None, **kinds):
    """A model of `layers` pre-norm layers; kinds: other parts than the built-in ones, by family."""
    kind = {"block": "pre_norm", "mixer": "gqa_attention", "feed_forward": "swiglu", "norm": "rms_norm", "stream_steps": (), **kinds}
    made = [
        LayerSpec(
            kind["block"],
            PartSpec(kind["mixer"], dict(num_heads=HEADS, num_kv_heads=KV, head_dim=HEAD, qk_norm_eps=None), f"{i}.attn."),
            PartSpec(kind["feed_forward"], dict(intermediate_size=FF), f"{i}.mlp."),
            PartSpec(kind["norm"], dict(eps=EPS), f"{i}.n1."),
            PartSpec(kind["norm"], dict(eps=EPS), f"{i}.n2."),
        )
        for i in range(layers)
    ]
    model = DecoderModel(ModelSpec(
        hidden_size=HIDDEN, vocab_size=VOCAB, max_positions=64, embedding=PartSpec("torch_embedding", dict(vocab_size=VOCAB), "e."),
        layers=tuple(made), schedule=tuple(schedule or [LayerCall(i) for i in range(layers)]), final_norm=PartSpec("rms_norm", dict(eps=EPS), "n."),
        head=PartSpec("torch_head", dict(vocab_size=VOCAB, tied=False), "h."), stream_steps=kind["stream_steps"],
    ))  # fmt: skip
    g = torch.Generator().manual_seed(3)
    model.load({s.name: torch.randn(s.shape, generator=g, dtype=torch.float64) * (1 if len(s.shape) == 1 else s.shape[1] ** -0.5)
                for s in model.tensor_specs()})  # fmt: skip
    for block in model.blocks:
        ff = block.feed_forward
        if isinstance(ff, SwiGLU):
            gate, up = ff.gate_up_proj.chunk(2)
            ff.fused, ff.gate_up_proj = True, ops.interleave_gate_up(gate, up)
    return model


class View:
    kept = None


def _context(tokens):
    ids = torch.arange(tokens, dtype=torch.int32)
    return StepContext(tokens, tokens, ids, ids, None, None, None, ids, 1)


def _run(model, tokens, ctx=None):
    return model.forward(ctx or _context(tokens), [View() if c.cache_from is None else None for c in model.schedule])


def _off(monkeypatch, model, tokens):
    with monkeypatch.context() as m:
        m.setattr(ops, "decode_chain_takes", lambda x, *matrices: False)
        return _run(model, tokens)


class HalvedSwiGLU(SwiGLU):
    def hidden(self, h):
        return super().hidden(h) / 2


class DoubledAttention(GQAttention):
    def forward_then(self, h, residual, ctx, cache, write_cache, then):
        out = super().forward(h, residual, ctx, cache, write_cache) + residual
        return out, then.forward(out)


class OwnAttention(GQAttention):
    def attend(self, h, ctx, cache, write_cache):
        return super().attend(h * 2, ctx, cache, write_cache)


class ShiftedNorm(RMSNorm):
    def forward(self, x, rows=None):
        return super().forward(x, rows) + 1


class OwnBlock(PreNormBlock):
    def forward_chain(self, x, normed, ctx, cache, write_cache, then):
        return super().forward_chain(x, None if normed is None else normed * 2, ctx, cache, write_cache, then)


@pytest.mark.parametrize("family,part", [("feed_forward", HalvedSwiGLU), ("mixer", DoubledAttention), ("mixer", OwnAttention),
                                         ("norm", ShiftedNorm), ("block", OwnBlock)])  # fmt: skip
def test_a_derived_part_is_run_by_its_own_methods(chain, monkeypatch, family, part):
    """A part that derives from one the chain knows and changes what it does is not passed over (nor handed an input that
    its own methods do not know)."""
    register_part(family, "of_the_test", part)
    model = _model(3, **{family: "of_the_test"})
    plain = _off(monkeypatch, model, 4)
    assert torch.allclose(_run(model, 4), plain, rtol=1e-12, atol=1e-12)


def test_a_method_set_on_the_part_itself_is_run(chain, monkeypatch):
    model = _model(2)
    seen = []
    for block in model.blocks:
        inner = block.feed_forward.hidden
        monkeypatch.setattr(block.feed_forward, "hidden", lambda h, inner=inner: seen.append(h.shape) or inner(h))
    _run(model, 4)
    assert len(seen) == 2 and chain.calls == 0


class PairOfBlocks(PreNormBlock):
    """Two pre-norm blocks in the place of one (the second one with the first one's sublayers, over a cache of its own)."""

    def load(self, tensors):
        super().load(tensors)
        self.first, self.second = (PreNormBlock(self.mixer, self.feed_forward, self.mixer_norm, self.feed_forward_norm) for _ in range(2))
        self.second.mixer_norm = ShiftedGain(self.mixer_norm)
        self.inner = View()

    def forward_chain(self, x, normed, ctx, cache, write_cache, then):
        x, normed = self.first.forward_chain(x, normed, ctx, cache, write_cache, self.second.mixer_norm)
        return self.second.forward_chain(x, normed, ctx, self.inner, True, then)


class ShiftedGain(RMSNorm):
    def __init__(self, other):
        self.gain, self.eps, self.width = other.gain + 1, other.eps, other.width


def test_a_block_of_blocks_hands_on_between_its_own(chain, monkeypatch):
    """What follows a block in the run order is not what follows a block inside it: the norm that a block is told to run next
    says whose input it hands on."""
    register_part("block", "pair_of_the_test", PairOfBlocks)
    model = _model(2, block="pair_of_the_test")
    model.blocks[1] = model.blocks[1].first
    plain = _off(monkeypatch, model, 4)
    assert torch.allclose(_run(model, 4), plain, rtol=1e-12, atol=1e-12)
    assert chain.calls == 3


@pytest.mark.parametrize("layers", [1, 3, 64, 65, 130])
def test_every_pass_zeroes_counters_of_its_own(chain, layers):
    """A pass that is captured into a graph after another one over the same context has to hold the zeroing of all its
    counters: words that an earlier pass zeroed would be met at their end state by the second replay."""
    model, ctx = _model(layers), _context(4)
    words = []
    for _ in range(2):
        chain.counters.clear()
        _run(model, 4, ctx)
        assert chain.calls == layers
        chain.calls = 0
        words.append({c.untyped_storage().data_ptr(): c.untyped_storage() for c in chain.counters})
        assert len({c.data_ptr() for c in chain.counters}) == layers  # a call's own
    assert not words[0].keys() & words[1].keys()


class Halfway(StreamStep):
    def __init__(self, hidden_size, prefix):
        pass

    def forward(self, x, x0, number, ctx):
        return (x + x0) / 2


@pytest.mark.parametrize("tokens", [1, 8])
def test_a_run_order_with_shared_caches_repeated_layers_and_stream_steps(chain, monkeypatch, tokens):
    """An entry that reads another one's keys and values is handed its queries only; nothing is handed over a stream step."""
    schedule = [LayerCall(0), LayerCall(1, cache_from=0), LayerCall(2), LayerCall(1), LayerCall(0, before=(0, 1)), LayerCall(2, cache_from=4)]
    register_part("stream_step", "halfway_of_the_test", Halfway)
    model = _model(3, schedule, stream_steps=(PartSpec("halfway_of_the_test"),))
    plain = _off(monkeypatch, model, tokens)
    assert chain.calls == 0
    assert torch.allclose(_run(model, tokens), plain, rtol=1e-12, atol=1e-12)
    assert chain.calls == 6 and chain.handed_on == 4  # not before the stream step, nor at the end


def test_more_tokens_than_it_takes(chain, monkeypatch):
    model = _model(2)
    assert torch.equal(_run(model, 9), _off(monkeypatch, model, 9)) and chain.calls == 0


@pytest.mark.parametrize("what", ["next product", "output", "feed-forward"])
def test_a_matrix_that_is_not_taken(chain, monkeypatch, what):
    """The layer before hands on its normed output where the next product is not taken; a layer whose own matrices are not
    taken runs by itself on what it is handed."""
    model = _model(3)
    block = model.blocks[1]
    chain.refused = [{"next product": block.mixer.qkv_proj, "output": block.mixer.o_proj, "feed-forward": block.feed_forward.down_proj}[what]]
    plain = _off(monkeypatch, model, 5)
    assert torch.allclose(_run(model, 5), plain, rtol=1e-12, atol=1e-12)
    assert (chain.calls, chain.handed_on) == ((3, 1) if what == "next product" else (2, 1))
