"""What the sampler uploads for a step's requests, and the settings it refuses (no GPU: the kernel's place is taken)."""

import numpy as np
import pytest
import torch

from atomserve_b200.engine.sequence import SamplingParams, Sequence
from atomserve_b200.sampling import sampler as module


@pytest.fixture
def uploaded(monkeypatch):
    calls = []

    def sample_rows(logits, temperature, top_k, top_p, seeds, counters):
        calls.append([t.clone() for t in (temperature, top_k, top_p, seeds, counters)])
        return torch.zeros(logits.shape[0], dtype=torch.int32)

    monkeypatch.setattr(module.ops, "sample_rows", sample_rows)
    return calls


def _step(params, tokens=((3, 4, 5),)):
    seqs = [Sequence(i, list(tokens[i % len(tokens)]), p, num_prompt_tokens=2) for i, p in enumerate(params)]
    return module.Sampler("cpu", base_seed=7).launch(torch.zeros(len(seqs), 11), seqs)


def test_settings_arrive_as_they_were_asked_for(uploaded):
    params = [SamplingParams(0.6, 20, 0.95, seed=5), SamplingParams(0.0, 0, 1.0, seed=(1 << 63) + 9), SamplingParams(1.5, 1 << 30, 0.25, seed=0)]
    _step(params, [(3, 4, 5), (3, 4), (3, 4, 5, 6, 7)])
    temperature, top_k, top_p, seeds, counters = uploaded[0]
    assert torch.equal(temperature, torch.tensor([0.6, 0.0, 1.5])) and torch.equal(top_p, torch.tensor([0.95, 1.0, 0.25]))
    assert top_k.tolist() == [20, 0, 1 << 30] and top_k.dtype == torch.int32
    assert seeds.tolist() == [5, 9, 0] and counters.tolist() == [1, 0, 3] and seeds.dtype == counters.dtype == torch.int64


@pytest.mark.parametrize("name,value,arrives", [
    ("temperature", 1, 1.0), ("temperature", True, 1.0), ("temperature", np.float64(0.5), 0.5), ("temperature", torch.tensor(0.5), 0.5),
    ("temperature", 1e39, float("inf")), ("top_p", 1, 1.0), ("top_p", np.float32(0.25), 0.25), ("top_k", 20.0, 20), ("top_k", 2.5, 2),
    ("top_k", np.int64(7), 7), ("top_k", True, 1), ("top_k", -1, -1),
])  # fmt: skip
@pytest.mark.filterwarnings("error")
def test_every_kind_of_number_is_taken(uploaded, name, value, arrives):
    _step([SamplingParams(0.7, 3, 0.5, seed=1), SamplingParams(**{"temperature": 0.7, "seed": 2, name: value})])
    assert uploaded[0][["temperature", "top_k", "top_p"].index(name)][1].item() == arrives


@pytest.mark.parametrize("name,value", [
    ("temperature", None), ("temperature", "0.6"), ("top_p", None), ("top_p", "0.95"), ("top_k", None), ("top_k", "20"),
    ("top_k", 1 << 31), ("top_k", -(1 << 31) - 1), ("top_k", np.int64(1 << 40)), ("top_k", 3e9), ("top_k", float("nan")), ("temperature", 1j),
])  # fmt: skip
def test_what_is_no_number_is_refused(uploaded, name, value):
    """A setting that is missing or a text raises, and never becomes a NaN, under which a row would be drawn as if greedy."""
    with pytest.raises((TypeError, ValueError, RuntimeError, OverflowError)):
        _step([SamplingParams(0.7, 3, 0.5, seed=1), SamplingParams(**{"temperature": 0.7, "seed": 2, name: value})])
    assert not uploaded
