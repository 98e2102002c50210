"""What a step asks of its kernels, as far as that is decided on the host: no GPU is needed."""

import pytest
import torch

from socrates_b200.engine import context
from socrates_b200.engine.context import Buffers, StepContext


def step(dtype=torch.bfloat16, **k):
    k = dict(all_decode=True, max_context=8192, num_sms=148, **k)
    return StepContext(dtype, torch.device("cpu"), Buffers(256, "cpu"), 4, 4, None, None, None, None, None, None, None, **k)


def test_only_bound_weights_are_read_ahead(monkeypatch):
    """The float32 product may fetch its matrix while the kernel before it runs where the matrix is one of the model's, and
    nowhere else (a product of two activations)."""
    asked = []
    monkeypatch.setattr(context.ops, "gemm_simt", lambda *a, splits, w_older=False: asked.append(w_older))
    ctx, x, bound, other = step(torch.float32), torch.zeros(4, 8), torch.zeros(6, 8), torch.zeros(6, 8)
    ctx.gemm(torch.zeros(4, 6), x, bound)
    ctx.weight_successor = {bound.data_ptr(): None}
    ctx.gemm(torch.zeros(4, 6), x, bound)
    ctx.gemm(torch.zeros(4, 6), x, other)
    assert asked == [False, True, False]


def test_every_streamed_weight_is_known():
    """The last one too, and none of them can be freed while its address stands for it."""
    from socrates_b200.config import config_from_dict
    from socrates_b200.engine.model import Model
    model = Model(config_from_dict({
        "architectures": ["Qwen3ForCausalLM"], "vocab_size": 32, "hidden_size": 32, "intermediate_size": 48,
        "num_hidden_layers": 2, "num_attention_heads": 2, "num_key_value_heads": 1, "head_dim": 16, "rms_norm_eps": 1e-6,
        "rope_theta": 1e4, "tie_word_embeddings": False, "max_position_embeddings": 64}).plan())
    model.bind({n: torch.zeros(s.shape) for n, s in model.parameters().items()}, torch.float32)
    weights = [w for layer in model.layers for w in layer.streamed_weights()] + model.head.streamed_weights()
    assert len(weights) == 9 and [w.data_ptr() for w in weights] == list(model.weight_successor)
    assert model.weight_successor[weights[-1].data_ptr()] is None


# ---------------------------------------------------------------------- layers that run from another's recorded calls
def qwen3(layers=3):
    from socrates_b200.config import config_from_dict
    from socrates_b200.engine.model import Model
    model = Model(config_from_dict({
        "architectures": ["Qwen3ForCausalLM"], "vocab_size": 32, "hidden_size": 32, "intermediate_size": 48,
        "num_hidden_layers": layers, "num_attention_heads": 2, "num_key_value_heads": 1, "head_dim": 16, "rms_norm_eps": 1e-6,
        "rope_theta": 1e4, "tie_word_embeddings": False, "max_position_embeddings": 64}).plan())
    model.bind({n: torch.zeros(s.shape) for n, s in model.parameters().items()}, torch.float32)
    return model


def facts_of(layer):
    from socrates_b200.kernels.layer_calls import layer_facts
    facts, tensors = [], []
    return (facts, tensors) if layer_facts(layer, facts, tensors) else None


def test_layers_of_equal_specs_are_alike():
    a, b = (facts_of(layer) for layer in qwen3().layers[:2])
    assert a[0] == b[0] and len(a[1]) == len(b[1]) == 9
    layer = qwen3().layers[0]
    assert {t.data_ptr() for t in layer.streamed_weights()} <= {t.data_ptr() for t in facts_of(layer)[1]}


@pytest.mark.parametrize("change", [
    lambda l: setattr(l.mixer, "window", 8), lambda l: setattr(l.mixer, "scale", 0.5),
    lambda l: setattr(l.mixer, "qk_norm_eps", 1e-3), lambda l: setattr(l.mixer, "q_gain", None),
    lambda l: setattr(l.norms[1], "eps", 1e-3), lambda l: setattr(l.feed_forward, "act", "gelu_tanh"),
    lambda l: setattr(l.mixer.position, "magnitude", 1.5)])
def test_a_layer_that_was_changed_is_like_no_other(change):
    first, second = qwen3().layers[:2]
    change(second)
    assert facts_of(second)[0] != facts_of(first)[0]


@pytest.mark.parametrize("pick,method", [
    (lambda l: l, "forward"), (lambda l: l.mixer, "forward"), (lambda l: l.feed_forward, "forward"),
    (lambda l: l.norms[0], "apply"), (lambda l: l.mixer.position, "tables"), (lambda l: l.mixer.o, "__call__")])
@pytest.mark.parametrize("where", ["instance", "class"])
def test_a_layer_with_a_wrapped_method_runs_by_itself(pick, method, where, monkeypatch):
    layer = qwen3().layers[1]
    part = pick(layer)
    plain = getattr(type(part), method)
    if where == "class":
        monkeypatch.setattr(type(part), method, lambda self, *a: plain(self, *a))
    else:
        setattr(part, method, lambda *a: plain(part, *a))
    assert facts_of(layer) is None


def test_other_parts_run_by_themselves():
    """A subclass, and a position encoding that says nothing of what its tables are."""
    from socrates_b200.parts.attention import GQAAttention
    from socrates_b200.parts.base import Part

    class Other(GQAAttention):
        pass

    class Fresh(Part):
        def tables(self, device):
            return torch.zeros(8), 16

    first, second = qwen3().layers[:2]
    first.mixer.__class__ = Other
    second.mixer.position = Fresh(None, "")
    assert facts_of(first) is None and facts_of(second) is None


def test_a_layer_with_a_tensor_elsewhere_is_left_to_the_entry_points_checks(monkeypatch):
    from socrates_b200.engine.model import Recording
    from socrates_b200.kernels.layer_calls import _REPLAYABLE
    from socrates_b200.parts.base import Branch, ResidualStream
    from socrates_b200.parts.block import PreNormBlock
    seen, table = [], torch.zeros(1, 1)

    def forward(self, ctx, stream, view):
        seen.append("own")
    known = _REPLAYABLE[PreNormBlock]
    monkeypatch.setattr(PreNormBlock, "forward", forward)
    monkeypatch.setitem(_REPLAYABLE, PreNormBlock, (known[0], forward, *known[2:]))
    monkeypatch.setattr(Recording, "__enter__", lambda self: self)
    monkeypatch.setattr(Recording, "__exit__", lambda self, *a: setattr(self, "words", []))
    monkeypatch.setattr(Recording, "run", lambda self, addresses: seen.append("run"))
    view = type("View", (), {"pools": lambda self: (torch.zeros(1), torch.zeros(1)), "block_table": lambda self: table})()
    model, stream, recordings = qwen3(6), ResidualStream(torch.zeros(4, 32)), {}
    stream.pending = waits = Branch(torch.zeros(1, 4, 32))
    model.layers[2].mixer.o.weight = model.layers[2].mixer.o.weight.to("meta")
    for i in range(1, 4):
        stream.pending = waits
        if not model._like_another(step(torch.float32, host_batch=[]), stream, view, i, recordings):
            seen.append("alone")
    assert seen[0] == "own" and seen[1] == "alone" and seen[2] in ("own", "run")


# ---------------------------------------------------------------------- kernels by the sizes of the cache
@pytest.mark.parametrize("pages,width,kernel", [
    (600, 4096, "attention_prefill_tcgen05"), (600, 4097, "attention_bias_tile"),     # 65,536 tokens in pages of 16
    (2 ** 25, 64, "attention_bias_tile")])                                            # 2^31 key rows in a pool
def test_windowed_attention_with_a_bias_takes_caches_of_any_size(pages, width, kernel, monkeypatch):
    from socrates_b200.config.plan import PartSpec
    from socrates_b200.parts import window_attention
    from socrates_b200.parts.window_attention import WindowBiasAttention
    part = WindowBiasAttention(PartSpec("window_bias_attention", dict(
        hidden_size=32, num_heads=4, num_kv_heads=4, key_dim=64, value_dim=64, scale=0.1, window=None, bias_far=16.0,
        softcap=-1.0)), "")
    ran = []
    for name in ("attention_prefill_tcgen05", "attention_bias_tile", "attention_bias"):
        monkeypatch.setattr(window_attention.ops, name, lambda *a, name=name, softcap=0.0, **k: ran.append((name, softcap)))
    monkeypatch.setattr(window_attention.ops, "short_conv", lambda *a: None)
    part.qkvg = lambda ctx, x, name: torch.zeros(x.shape[0], part.C + part.H)
    part.o = lambda ctx, x, name, out: torch.zeros(1, x.shape[0], 32)
    ctx = step(status=torch.zeros(1, dtype=torch.int32))
    ctx.all_decode, ctx.num_tokens = False, 40
    pool = torch.empty(pages, 4, 16, 64, device="meta", dtype=torch.bfloat16)
    cache = type("View", (), {"pools": lambda self: (pool, pool), "block_table": lambda self: torch.empty(4, width, device="meta")})()
    part.forward(ctx, torch.zeros(40, 32), cache)
    assert [name for name, _ in ran] == [kernel]
    assert kernel != "attention_prefill_tcgen05" or ran[0][1] >= 0    # a cap below zero was, and is, no cap


@pytest.mark.parametrize("M,N,K,parts", [
    (64, 2560, 4096, 0), (65, 2560, 4096, 13), (128, 2560, 4096, 13), (129, 2560, 4096, 7), (192, 2560, 4096, 7),
    (193, 2560, 4096, 0), (250, 2560, 4096, 0),                            # follows attention: not in a few heavy tiles
    (129, 4096, 4096, 0), (187, 5120, 8192, 0), (128, 4096, 4096, 8),      # ... nor in fewer than five parts
    (187, 2560, 9728, 7), (250, 2560, 9728, 7), (187, 4096, 12288, 4),
    (193, 4096, 12288, 0), (256, 5120, 25600, 0), (256, 6144, 2560, 3), (257, 2560, 9728, 0)])
def test_parts_of_products_of_65_to_256_rows(M, N, K, parts):
    """Tiles of 256 columns only where nine tenths of the SMs get a block, whatever the rule for short products is."""
    ctx, w = step(status=torch.zeros(1, dtype=torch.int32)), torch.empty(N, K, device="meta", dtype=torch.bfloat16)
    assert ctx.wide_splits(M, w, torch.bfloat16) == parts
    assert parts == 0 or M <= 192 or 10 * -(-N // 128) * parts >= 9 * 148


@pytest.mark.parametrize("Hkv,lengths,shares", [
    (8, [4000] * 9, False), (8, [4000] * 11, False), (8, [4000] * 12, True), (8, [2000] * 12, False),
    (8, [4000] + [250] * 8, True), (16, [4000] * 6, True), (16, [4000] * 7, False), (4, [4000] * 18, False),
    (4, [4000] * 24, True), (2, [4000] * 36, False), (2, [4000] * 48, True), (8, [2048] * 8, False)])
def test_shares_are_weighed_against_the_partitions_that_the_launch_has(Hkv, lengths, shares):
    """Counts of 3 and 4 partitions are stepped down where clusters fill the GPU badly; the rule counts with the same number."""
    from socrates_b200.config.plan import PartSpec
    from socrates_b200.kernels import ops
    from socrates_b200.parts.attention import GQAAttention, decode_partitions
    part = GQAAttention(PartSpec("gqa_attention", dict(hidden_size=64, num_heads=32, num_kv_heads=Hkv, head_dim=128,
                                                       position=PartSpec("none", {}))), "")
    assert part.prefers_shares(lengths, 148) == shares
    ctx = step()
    ctx.num_tokens = N = len(lengths)
    NP = decode_partitions(ctx, Hkv, ops.attention_decode_mma_blocks_per_sm(128), 128)
    longest, total = -(-max(lengths) // 64), sum(lengths) / 64 + N / 2
    assert (-(-longest // NP) - total / ops.attention_balanced_shares(32, Hkv, 128, N, 148) >= 8) == shares


@pytest.mark.parametrize("head_dim,N,shares", [(128, 19, True), (256, 19, False), (128, 1024, True), (128, 1025, False)])
def test_no_shares_where_their_kernel_does_not_serve(head_dim, N, shares):
    """A step that asked for them would only be recorded a second time, with the same kernels."""
    from socrates_b200.config.plan import PartSpec
    from socrates_b200.parts.attention import GQAAttention
    part = GQAAttention(PartSpec("gqa_attention", dict(hidden_size=64, num_heads=32, num_kv_heads=8, head_dim=head_dim,
                                                       position=PartSpec("none", {}))), "")
    assert part.prefers_shares([7001] + [437] * (N - 1), 148) == shares
