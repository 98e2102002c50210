"""Decode attention in equal shares as the engine runs it: in first steps of a width, from recorded graphs beside the other
kernel's graph of the same width, recorded at start-up, and in mixed steps."""

import pytest
import torch

pytestmark = pytest.mark.gpu
ROWS, LONG = 20, 1300


def build(**limits):
    from socrates_b200 import Engine
    from socrates_b200.config import config_from_dict
    from socrates_b200.engine.engine import build_random_model
    built = build_random_model(config_from_dict({
        "architectures": ["Qwen3ForCausalLM"], "vocab_size": 300, "hidden_size": 256, "intermediate_size": 384,
        "num_hidden_layers": 3, "num_attention_heads": 16, "num_key_value_heads": 8, "head_dim": 128, "rms_norm_eps": 1e-6,
        "rope_theta": 1e4, "tie_word_embeddings": False}), 3, torch.bfloat16, torch.device("cuda:0"))
    return Engine(built, device="cuda:0", dtype="bfloat16", block_size=16, max_batch=ROWS, max_len=2048, token_budget=700,
                  num_blocks=400, **limits)


def ids(seed, n):
    return torch.randint(0, 300, (n,), generator=torch.Generator().manual_seed(seed)).tolist()


def filled(engine):
    """Row 0 holds 1,300 tokens, the others 10 to 67; returns the lengths."""
    from socrates_b200.engine.runner import StepEntry
    lengths = [LONG] + [10 + 3 * r for r in range(1, ROWS)]
    for row, n in enumerate(lengths):
        engine.cache.assign(row)
        assert engine.cache.reserve(row, n + 140)
        for start in range(0, n, 700):
            part = ids(row, n)[start:start + 700]
            engine.runner.step([StepEntry(row, part, start, [len(part) - 1])])
            engine.cache.commit(row, start + len(part))
    return lengths


def decode(engine, lengths, rows):
    from socrates_b200.engine.runner import StepEntry
    return engine.runner.step([StepEntry(r, ids(100 + r, 1), lengths[r], [0]) for r in rows]).logits.clone()


UNEVEN, EVEN = list(range(ROWS - 1)), list(range(1, ROWS))        # with and without the long row, 19 rows each


@pytest.fixture
def checked(monkeypatch):
    """Every call of the equal-shares kernel is compared with the float64 reference; the list of calls."""
    from socrates_b200.kernels import ops, reference
    calls, real = [], ops.attention_decode_balanced

    def balanced(out, q, k_pool, v_pool, table, starts, rows, first, Hq, scale, window, *scratch):
        real(out, q, k_pool, v_pool, table, starts, rows, first, Hq, scale, window, *scratch)
        if torch.cuda.is_current_stream_capturing():
            return
        calls.append(rows.numel())
        single = (starts[1:] - starts[:-1] == 1).nonzero().flatten()
        at = starts[single].long()
        want = reference.paged_attention_ref(q[at], k_pool, v_pool, table, rows[single], first[single], Hq, scale, window)
        # bfloat16 output (2^-9, doubled) of sums whose weights are two bfloat16 terms
        assert torch.allclose(out[at].double(), want, atol=2e-3, rtol=1.6e-2)
    monkeypatch.setattr(ops, "attention_decode_balanced", balanced)
    return calls


def test_both_graphs_of_a_width(checked):
    engine = build()
    lengths = filled(engine)
    assert engine.model.prefers_shares([lengths[r] + 1 for r in UNEVEN], 148)
    assert not engine.model.prefers_shares([lengths[r] + 1 for r in EVEN], 148)
    uneven, even = decode(engine, lengths, UNEVEN), decode(engine, lengths, EVEN)       # launched one by one
    assert checked == [19] * 3
    assert {key[2] for key in engine.runner._graphs} == set()
    for _ in range(3):                                  # recorded, then replayed, in turn: the counters end where they began
        assert torch.equal(decode(engine, lengths, UNEVEN), uneven)
        assert torch.equal(decode(engine, lengths, EVEN), even)
    assert {key for key in engine.runner._graphs} == {(19, False, True), (19, False, False)}
    assert engine.runner.graph_replays == 6 and checked == [19] * 3


def test_graphs_recorded_at_start_up_give_the_same_bits():
    cold, warm = build(), build(warmup=True)
    assert (19, True, True) in warm.runner._graphs and (4, True, True) not in warm.runner._graphs
    recorded = set(warm.runner._graphs)
    from socrates_b200.engine.runner import SamplingArgs, StepEntry
    results = []
    for engine in (cold, warm):
        lengths = filled(engine)
        entries = [StepEntry(r, ids(100 + r, 1), lengths[r], [0]) for r in UNEVEN]
        results.append(engine.runner.step(entries, [SamplingArgs(0.0, 0, 0)] * len(entries)).logits.clone())
    assert torch.equal(*results) and set(warm.runner._graphs) == recorded and warm.runner.graph_replays == 1


@pytest.mark.parametrize("from_keys,calls", [(LONG + 1, 3), (LONG + 2, 0)])
def test_mixed_step_with_a_long_row(checked, monkeypatch, from_keys, calls):
    """From SINGLES_APART_FROM keys in the longest request of one token on, such requests run in this kernel."""
    from socrates_b200.engine.runner import StepEntry
    from socrates_b200.parts import attention
    engine = build()
    lengths = filled(engine)
    entries = [StepEntry(r, ids(100 + r, 130 if r == 7 else 1), lengths[r], [129 if r == 7 else 0]) for r in range(9)]
    monkeypatch.setattr(attention, "SINGLES_APART_FROM", 10 ** 6)
    together = engine.runner.step(entries).logits.clone()
    assert checked == []
    monkeypatch.setattr(attention, "SINGLES_APART_FROM", from_keys)
    apart = engine.runner.step(entries).logits.clone()
    assert checked == [9] * calls
    # the same sums in another order, rounded to bfloat16 in three layers: 2^-9 of a value each, twice per layer at most
    assert float((apart - together).norm() / together.norm()) <= 6 * 2.0 ** -9
