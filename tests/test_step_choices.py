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
