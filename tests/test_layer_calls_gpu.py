"""Layers that run from the recorded calls of a layer like them: the same bits and the same number of launches as layers
that run one by one, in prompts, mixed steps and both engines, and not for layers that differ."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def build(dtype, layers=6, window=None, seed=0):
    from socrates_b200 import Engine
    from socrates_b200.config import config_from_dict
    from socrates_b200.engine.model import Model
    config = config_from_dict({
        "architectures": ["Qwen3ForCausalLM"], "vocab_size": 300, "hidden_size": 256, "intermediate_size": 384,
        "num_hidden_layers": layers, "num_attention_heads": 4, "num_key_value_heads": 2, "head_dim": 64,
        "rms_norm_eps": 1e-6, "rope_theta": 1e4, "tie_word_embeddings": False, "max_position_embeddings": 4096,
        "sliding_window": window, "use_sliding_window": window is not None, "max_window_layers": 3})
    model = Model(config.plan())
    g = torch.Generator().manual_seed(seed)
    tensors = {}
    for name, spec in model.parameters().items():
        t = torch.randn(spec.shape, generator=g)
        tensors[name] = (1 + 0.1 * t if len(spec.shape) == 1 else (0.05 * t).to(dtype)).to(DEV)
    model.bind(tensors, dtype)
    return Engine((config, model), device="cuda:0", dtype=dtype, block_size=16, max_batch=4, max_len=2048, token_budget=600,
                  num_blocks=400)


def steps(engine, after_step=lambda: None):
    """Logits of a prompt, of its second portion beside two new prompts, and of a step that mixes both kinds."""
    from socrates_b200.engine.runner import StepEntry
    g = torch.Generator().manual_seed(5)
    ids = lambda n: torch.randint(0, 300, (n,), generator=g).tolist()
    cache, out, at = engine.cache, [], {}
    for row in range(4):
        cache.assign(row)
    for portions in ([(0, 70)], [(0, 200), (1, 9), (2, 130)], [(0, 1), (1, 1), (3, 300), (2, 1)], [(0, 5), (1, 2)]):
        entries = []
        for row, n in portions:
            start = at.get(row, 0)
            assert cache.reserve(row, start + n)
            entries.append(StepEntry(row, ids(n), start, [n - 1]))
        out.append(engine.runner.step(entries).logits.clone())
        after_step()
        for row, n in portions:
            at[row] = at.get(row, 0) + n
            cache.commit(row, at[row])
    return out, engine.runner.kernel_launches


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("window", [None, 40])
def test_recorded_layers_give_the_same_bits(dtype, window, monkeypatch):
    from socrates_b200.engine.model import Model
    from socrates_b200.kernels.layer_calls import Recording
    runs = []
    run = Recording.run
    monkeypatch.setattr(Recording, "run", lambda self, a: (runs.append(1), run(self, a))[1])
    so_far = []
    got, launches = steps(build(dtype, window=window), lambda: so_far.append(len(runs)))
    # in every step: of six layers alike the first finds nothing pending, the second is recorded and the last is followed
    # by another matrix; of three and three (with a window) only the fifth runs from another's calls
    assert so_far == [n * (3 if window is None else 1) for n in (1, 2, 3, 4)]
    monkeypatch.setattr(Model, "_like_another", lambda *a: False)
    want, plain = steps(build(dtype, window=window))
    assert launches == plain
    for a, b in zip(got, want):
        assert torch.equal(a, b)


def test_a_layer_with_a_tensor_of_another_type_runs_by_itself(monkeypatch):
    """One float32 matrix in a bfloat16 engine goes through another kernel."""
    from socrates_b200.engine.model import Model
    from socrates_b200.parts.linear import Linear

    def odd():
        engine = build(torch.bfloat16)
        layer = engine.model.layers[3]
        layer.mixer.o = Linear(layer.mixer.o.weight.float())
        return engine
    got, launches = steps(odd())
    monkeypatch.setattr(Model, "_like_another", lambda *a: False)
    want, plain = steps(odd())
    assert launches == plain and all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("how,kernel", [("auto", "sb_attention_decode_mma"), ("64", "sb_attention_decode_stream"),
                                        ("shares", "sb_attention_balanced"), ("mixed", "sb_attention_balanced")])
def test_decode_kernels_from_recorded_calls(how, kernel, monkeypatch):
    """The first step of a width, which launches its kernels one by one, and a mixed step with a long row: the same bits
    and launches as layers that run one by one, through each decode-attention kernel."""
    from socrates_b200.engine.model import Model
    from socrates_b200.engine.runner import StepEntry
    from socrates_b200.kernels.layer_calls import Recording
    if how == "64":
        monkeypatch.setenv("PAGED_PARTITION", "64")
    if how == "shares":
        monkeypatch.setattr(Model, "prefers_shares", lambda *a: True)
    names, runs, run = set(), [], Recording.run

    def seen(self, addresses):
        runs.append(1)
        names.update(name for name, _ in self._recorder.calls)
        return run(self, addresses)
    monkeypatch.setattr(Recording, "run", seen)

    def last_step():
        engine = build(torch.bfloat16)
        g = torch.Generator().manual_seed(6)
        ids = lambda n: torch.randint(0, 300, (n,), generator=g).tolist()
        for row, lengths in enumerate([(600, 600), (9,), (300,), (44,)]):
            engine.cache.assign(row)
            for i, n in enumerate(lengths):
                assert engine.cache.reserve(row, sum(lengths[:i + 1]) + 150)
                engine.runner.step([StepEntry(row, ids(n), sum(lengths[:i]), [n - 1])])
                engine.cache.commit(row, sum(lengths[:i + 1]))
        at, before = (1200, 9, 300, 44), len(runs)
        counts = (1, 1, 130, 1) if how == "mixed" else (1, 1, 1, 1)
        names.clear()
        logits = engine.runner.step([StepEntry(r, ids(n), at[r], [n - 1]) for r, n in enumerate(counts)]).logits.clone()
        return logits, engine.runner.kernel_launches, len(runs) - before
    got, launches, replayed = last_step()
    assert replayed == 3 and kernel in names
    monkeypatch.setattr(Model, "_like_another", lambda *a: False)
    want, plain, replayed = last_step()
    assert replayed == 0 and launches == plain and torch.equal(got, want)


@pytest.mark.parametrize("change", [
    lambda layer: setattr(layer.mixer, "window", 24), lambda layer: setattr(layer.mixer, "scale", 0.3),
    lambda layer: setattr(layer.norms[1], "eps", 0.5), lambda layer: setattr(layer.mixer.position, "magnitude", 1.5)])
def test_a_layer_that_was_changed_after_it_was_built(change, monkeypatch):
    from socrates_b200.engine.model import Model

    def odd():
        engine = build(torch.bfloat16)
        change(engine.model.layers[3])
        return engine
    got, launches = steps(odd())
    monkeypatch.setattr(Model, "_like_another", lambda *a: False)
    want, plain = steps(odd())
    assert launches == plain and all(torch.equal(a, b) for a, b in zip(got, want))
    same, _ = steps(build(torch.bfloat16))
    assert not torch.equal(got[0], same[0])             # the change shows at all


def test_a_wrapped_layer_is_called_in_every_step():
    engine, calls = build(torch.bfloat16), []
    layer = engine.model.layers[3]
    forward = layer.mixer.forward
    layer.mixer.forward = lambda *a: (calls.append(1), forward(*a))[1]
    got, _ = steps(engine)
    same, _ = steps(build(torch.bfloat16))
    assert len(calls) == 4 and all(torch.equal(a, b) for a, b in zip(got, same))


def test_words_per_entry_point():
    from socrates_b200.kernels.layer_calls import ENTRIES
    from socrates_b200.kernels.library import _SIGNATURES, library
    for name, number in ENTRIES.items():
        assert library().sb_run_calls_arity(number) == len(_SIGNATURES[name]), name
    assert library().sb_run_calls_arity(len(ENTRIES)) == -1
