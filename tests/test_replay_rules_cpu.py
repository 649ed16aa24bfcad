"""Which decode steps with logits may replay a captured step: the engine's rules, which need no GPU."""
import pytest
import torch

from blaze_b200.config import named_config
from blaze_b200.llm import LLM
from blaze_b200.models import qwen3


def _engine(name="tiny", **kw):
    return LLM(named_config(name), device="cpu", dtype=torch.float32, max_seqs=4, max_model_len=128, seed=0, **kw).engine


def _decode_step(eng):
    return eng.plan([(eng.open_from(), [1], 1) for _ in range(2)])


def test_steps_that_something_follows_are_launched_one_by_one(monkeypatch):
    """Dumps, phase timers, routing statistics and kept hidden rows come from the layer loop itself, and an indexer reads the contexts'
    lengths on the host: a replayed step would leave them out, count its padding, or select keys for other lengths."""
    eng = _engine()
    step = _decode_step(eng)
    assert eng._logits_graphable(step)
    for name, value in (("_DUMP_DIR", "/nowhere"), ("_PROFILE_PHASES", True)):
        with monkeypatch.context() as m:
            m.setattr(qwen3, name, value)
            assert not eng._logits_graphable(step), name
    for obj, name, value in ((eng.model, "capture_layers", [0]), (eng.model, "heat", object()), (eng.model.cfg, "indexer_heads", 2)):
        with monkeypatch.context() as m:
            m.setattr(obj, name, value)
            assert not eng._logits_graphable(step), name
    assert eng._logits_graphable(step)


def test_routing_statistics_keep_sampled_steps_uncaptured():
    eng = _engine("tiny-hybrid", expert_heat=True)
    assert eng.model.heat is not None and not eng._logits_graphable(_decode_step(eng))


@pytest.mark.parametrize("name", ["tiny-sevevik", "tiny-niletar", "tiny-rapisun", "tiny-medodra"])
def test_designs_whose_keys_are_cut_by_the_longest_context(name):
    """Their kernels' runs of keys depend on a length that a captured step does not know: launched one by one, always."""
    eng = _engine(name)
    assert not eng._logits_graphable(_decode_step(eng))


@pytest.mark.parametrize("change", [{"want_logits": 0}, {"defer_state": True}, {"parents": [-1]}])
def test_rows_that_a_captured_step_does_not_hold(change):
    eng = _engine()
    step = _decode_step(eng)
    for k, v in change.items():
        setattr(step[1], k, v)
    assert not eng._logits_graphable(step)


def test_buckets_of_sampled_steps():
    """No padding up to 16 sequences and an eighth at most above; no bucket crosses a power of two, a row tile or a limit of the expert
    kernels, where products take other forms; a few buckets for every doubling."""
    eng = _engine()
    for limits in (set(), {21, 192, 768}):
        eng._limits = limits
        for n in range(1, 2049):
            b = eng._sampled_bucket(n)
            assert n <= b <= n * 9 // 8 and eng._sampled_bucket(b) == b
            assert not any(n <= r < b for r in [24, *limits, *(1 << i for i in range(12)), *range(128, 1025, 128)]), (n, b)
        assert len({eng._sampled_bucket(n) for n in range(17, 1025)}) <= 8 * 6 + len(limits)
