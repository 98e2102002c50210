"""What the engine is measured on: steps of the real Qwen3 shapes through `Engine.runner.step`, whole
generations through `Engine.generate`, and a prompt through one of the further designs.

A case is a dict of plain values.  kind "step" is one step of the engine, the unit that serving is made of:
`decodes` requests that bring one token each over `context` cached tokens (`ragged`: between a sixteenth of that
and all of it), and `portions` prompt portions that share `tokens` new tokens, each after `start` cached ones.  kind
"generate" is a whole call of `Engine.generate` with a small model.  kind "design" is one prompt through the Bofusun
decoder (retention, windowed attention with capped scores and a distance bias, a selective scan).

Sizes: the Qwen3-4B, 8B and 32B shapes with 18, 12 and 4 of their 36, 36 and 64 layers (a layer costs the same at any
depth; three states fit the card, and the bfloat16 rounding of the layers has not added up to more than two correct
implementations can be compared by); the tiny configurations of the tests.  Weights are
N(0, 0.02) and gains 1 + N(0, 0.1), cached keys and values N(0, 1) (what normed keys and projected values measure),
token ids uniform over the vocabulary, pages of 16 slots, rows of 8,192 tokens.
"""

import math
import zlib

import torch

from socrates_b200 import Engine
from socrates_b200.config import config_from_dict
from socrates_b200.engine.model import Model
from socrates_b200.engine.runner import SamplingArgs, StepEntry

PAGE, MAX_LEN = 16, 8192
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}


def _qwen3(hidden, inter, layers, heads, kv_heads, head_dim, vocab, tied, eps=1e-6, theta=1e6, window=None):
    return {"architectures": ["Qwen3ForCausalLM"], "vocab_size": vocab, "hidden_size": hidden,
            "intermediate_size": inter, "num_hidden_layers": layers, "num_attention_heads": heads,
            "num_key_value_heads": kv_heads, "head_dim": head_dim, "rms_norm_eps": eps, "rope_theta": theta,
            "tie_word_embeddings": tied, "max_position_embeddings": 40960, "sliding_window": window,
            "use_sliding_window": window is not None, "max_window_layers": 1}


MODELS = {
    "4b": _qwen3(2560, 9728, 18, 32, 8, 128, 151936, True),
    "8b": _qwen3(4096, 12288, 12, 32, 8, 128, 151936, False),
    "32b": _qwen3(5120, 25600, 4, 64, 8, 128, 151936, False),
    "4b_2_layers": _qwen3(2560, 9728, 2, 32, 8, 128, 151936, True),
    "tiny_a": _qwen3(64, 128, 2, 4, 2, 16, 256, True, theta=1e4),
    "tiny_b": _qwen3(96, 160, 3, 8, 2, 32, 384, False, eps=1e-5, window=37),
}

# Five retention layers around one parallel layer with a feed-forward, the middle layers run twice.
_HEADS, _WIDTH = 16, 2048
_RET = {"type": "retention", "mlp": None,
        "mixer": {"heads": _HEADS, "dim": _WIDTH // (2 * _HEADS), "vdim": _WIDTH // _HEADS,
                  "rot": {"dims": _WIDTH // (2 * _HEADS), "base": 1e6},
                  "decay": [1.0 - 2.0 ** (-5 - 6 * h / (_HEADS - 1)) for h in range(_HEADS)]}}
_PAR = {"type": "parallel", "mlp": {"kind": "dense", "ff": 4 * _WIDTH},
        "mixer": {"left": {"heads": _HEADS, "kv_heads": _HEADS // 4, "dim": 128, "vdim": 128, "conv": 3,
                           "scale": 128 ** -0.5, "softcap": 30.0, "bias_max": 2048, "mask": {"size": 1024}},
                  "right": {"inner": 2 * _WIDTH, "state": 16, "dt_rank": _WIDTH // 16, "conv": 4}}}
BOFUSUN = {"architecture": "Bofusun", "vocab": 32000, "width": _WIDTH, "norm": {"eps": 1e-5},
           "layers": [_RET, _RET, _PAR, _RET, _RET, _RET], "loop": {"start": 1, "stop": 3, "times": 2}}


# ------------------------------------------------------------------ cases
def _step(name, model, decodes=0, context=0, ragged=False, portions=0, tokens=0, start=0, dtype="bfloat16",
          temperature=0.0):
    return {"name": name, "kind": "step", "model": model, "dtype": dtype, "decodes": decodes, "context": context,
            "ragged": ragged, "portions": portions, "tokens": tokens, "start": start, "temperature": temperature}


def listed():
    return [
        # a command-line run of the tests' size: four short prompts cut under a small token budget, sampled
        {"name": "generate_tiny", "kind": "generate", "model": "tiny_b", "prompts": 4, "longest": 40, "new": 6,
         "budget": 8, "temperature": 0.8},
        # one user chatting: decode of a single request
        _step("decode_1", "4b", decodes=1, context=2048),
        # the benchmark's headline: decode of a small batch
        _step("decode_8", "4b", decodes=8, context=2048),
        # a full server: 64 requests of mixed lengths, sampled
        _step("decode_64_ragged", "4b", decodes=64, context=4096, ragged=True, temperature=0.8),
        # long conversations on the largest shape
        _step("decode_8_32b", "32b", decodes=8, context=4096),
        # an in-between batch with long rows of odd lengths
        _step("decode_19_long", "8b", decodes=19, context=7001, ragged=True),
        # time to first token of a chat message
        _step("prompt_187", "4b", portions=1, tokens=187),
        # the benchmark's prompt
        _step("prompt_2048", "4b", portions=1, tokens=2048),
        # a long document on the largest shape: its second portion
        _step("portion_1999_32b", "32b", portions=1, tokens=1999, start=2048),
        # continuous batching: live requests decode while two prompts come in
        _step("mixed_37", "8b", decodes=37, context=4096, ragged=True, portions=2, tokens=1023, temperature=0.8),
        # the true 32-bit path: a prompt beside decoding requests
        _step("mixed_float32", "4b_2_layers", decodes=3, context=511, portions=1, tokens=253, dtype="float32"),
        # a prompt through another design
        {"name": "bofusun_1500", "kind": "design", "tokens": 1500},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    pick = rng.random()
    if pick < 0.08:
        return {"kind": "generate", "model": rng.choice(["tiny_a", "tiny_b"]), "prompts": rng.randint(1, 6),
                "longest": _log(rng, 2, 120), "new": rng.randint(2, 12), "budget": rng.choice([8, 16, 64]),
                "temperature": rng.choice([0.0, 0.8])}
    if pick < 0.16:
        return {"kind": "design", "tokens": _log(rng, 33, 2048)}
    if pick < 0.26:
        decodes = rng.randint(0, 6)
        case = _step("", "4b_2_layers", decodes=decodes, context=_log(rng, 16, 1500), ragged=rng.random() < 0.5,
                     portions=1 if decodes == 0 else rng.randint(0, 2), tokens=_log(rng, 8, 320), dtype="float32")
    else:
        model = rng.choice(["4b", "8b", "32b"])
        temperature = rng.choice([0.0, 0.8])
        if pick < 0.58:                                 # decode
            batch = _log(rng, 1, 64)
            case = _step("", model, decodes=batch, context=_log(rng, 16, min(8000, 131072 // batch)),
                         ragged=rng.random() < 0.5, temperature=temperature)
        elif pick < 0.85:                               # prompts
            portions = rng.choice([1, 1, 2, 3])
            case = _step("", model, portions=portions, tokens=_log(rng, 4 * portions, 2048),
                         start=rng.choice([0, 0, 2048, _log(rng, 16, 4000)]), temperature=temperature)
        else:                                           # both
            case = _step("", model, decodes=_log(rng, 1, 48), context=_log(rng, 64, 4096), ragged=True,
                         portions=rng.randint(1, 2), tokens=_log(rng, 16, 1500), start=rng.choice([0, 0, 1024]),
                         temperature=temperature)
    del case["name"]
    if case["portions"] == 0:
        case["tokens"] = case["start"] = 0
    if case["decodes"] == 0:
        case["context"], case["ragged"] = 0, False
    return case


# ------------------------------------------------------------------ inputs, from the case and the seed alone
def _generator(seed, name):
    g = torch.Generator(device="cuda")
    g.manual_seed((seed * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFFFFFF)
    return g


def _normal(seed, name, shape, dtype, mean=0.0, std=1.0):
    t = torch.empty(shape, device="cuda", dtype=dtype)
    return t.normal_(mean, std, generator=_generator(seed, name))


def _numbers(seed, name, count, below):
    """`count` whole numbers in [0, below), as a list."""
    return torch.randint(0, below, (count,), device="cuda", generator=_generator(seed, name)).tolist()


def _qwen3_shapes(cfg):
    d, inter, D = cfg["hidden_size"], cfg["intermediate_size"], cfg["head_dim"]
    q, kv = cfg["num_attention_heads"] * D, cfg["num_key_value_heads"] * D
    out = {"model.embed_tokens.weight": (cfg["vocab_size"], d), "model.norm.weight": (d,)}
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        out.update({p + "input_layernorm.weight": (d,), p + "post_attention_layernorm.weight": (d,),
                    p + "self_attn.q_proj.weight": (q, d), p + "self_attn.k_proj.weight": (kv, d),
                    p + "self_attn.v_proj.weight": (kv, d), p + "self_attn.o_proj.weight": (d, q),
                    p + "self_attn.q_norm.weight": (D,), p + "self_attn.k_norm.weight": (D,),
                    p + "mlp.gate_proj.weight": (inter, d), p + "mlp.up_proj.weight": (inter, d),
                    p + "mlp.down_proj.weight": (d, inter)})
    if not cfg["tie_word_embeddings"]:
        out["lm_head.weight"] = (cfg["vocab_size"], d)
    return out


def _qwen3_tensor(seed, name, shape, dtype):
    """A matrix holds bfloat16 values in either engine; a gain is float32."""
    if len(shape) == 1:
        return _normal(seed, name, shape, torch.float32, 1.0, 0.1)
    return _normal(seed, name, shape, torch.bfloat16, 0.0, 0.02).to(dtype)


def _bofusun_shapes():
    d = _WIDTH
    out = {"embed": (32000, d), "embed.norm": (d,), "loop.step": (2, d), "final.norm": (d,), "head": (32000, d)}
    for i, spec in enumerate(BOFUSUN["layers"]):
        p, m = f"l{i}.", spec["mixer"]
        out.update({p + "norm1": (d,), p + "norm1b": (d,)})
        if spec["type"] == "retention":
            k, v = m["heads"] * m["dim"], m["heads"] * m["vdim"]
            out.update({p + "mix.q": (k, d), p + "mix.k": (k, d), p + "mix.v": (v, d), p + "mix.g": (v, d),
                        p + "mix.o": (d, v)})
            continue
        a, s, l, r = m["left"], m["right"], p + "mix.left.", p + "mix.right."
        for n, heads in (("q", a["heads"]), ("k", a["kv_heads"]), ("v", a["kv_heads"])):
            out.update({l + n: (heads * 128, d), l + n + ".b": (heads * 128,), l + n + ".conv": (heads * 128, a["conv"])})
        out.update({l + "rel": (32, a["heads"]), l + "g": (a["heads"], d), l + "o": (d, a["heads"] * 128), l + "out": (d,)})
        n, inner = s["state"], s["inner"]
        out.update({r + "in": (2 * inner, d), r + "conv": (inner, s["conv"]), r + "conv.b": (inner,),
                    r + "x": (s["dt_rank"] + 2 * n, inner), r + "dt": (inner, s["dt_rank"]), r + "dt.b": (inner,),
                    r + "A_log": (inner, n), r + "D": (inner,), r + "o": (d, inner), r + "out": (d,)})
        ff = spec["mlp"]["ff"]
        out.update({p + "norm2": (d,), p + "norm2b": (d,), p + "mlp.up": (ff, d), p + "mlp.up.b": (ff,),
                    p + "mlp.down": (d, ff), p + "mlp.down.b": (d,)})
    return out


def _bofusun_tensor(seed, name, shape):
    last = name.rsplit(".", 1)[-1]
    if name.endswith("dt.b"):
        return _normal(seed, name, shape, torch.float32).sigmoid_().mul_(3.0).sub_(4.0)
    if last == "A_log":
        return _normal(seed, name, shape, torch.float32).sigmoid_().mul_(2.5)
    if last in ("out", "D"):
        return _normal(seed, name, shape, torch.float32, 1.0, 0.1)
    if last in ("conv", "rel", "norm", "norm1", "norm1b", "norm2", "norm2b"):
        # taps and distance biases of order one half, offsets of a gain of order a tenth
        return _normal(seed, name, shape, torch.float32, 0.0, 0.5 if last in ("conv", "rel") else 0.1)
    if last in ("b", "step"):
        return _normal(seed, name, shape, torch.float32, 0.0, 0.02)
    return _normal(seed, name, shape, torch.bfloat16, 0.0, 0.02)


def _entries(case, seed):
    """[(new token ids, cached tokens)] of the requests of a step, decoding ones first."""
    V, B, P = MODELS[case["model"]]["vocab_size"], case["decodes"], case["portions"]
    cached = [case["context"]] * B
    if case["ragged"]:
        lo = max(1, case["context"] // 16)
        cached = [lo + n for n in _numbers(seed, "context", B, case["context"] - lo + 1)]
        cached[0] = case["context"]
    counts = [1] * B
    if P:                                               # portions of different sizes that add up to `tokens`
        each, left = case["tokens"] // P, case["tokens"]
        for i in range(P):
            n = left if i == P - 1 else max(1, each - each // 4 * (P - 1 - i))
            counts.append(n)
            cached.append(case["start"])
            left -= n
    ids = _numbers(seed, "ids", sum(counts), V)
    out = []
    for n, start in zip(counts, cached):
        out.append((ids[:n], start))
        ids = ids[n:]
    return out


def _cached(seed, cfg, layer, tokens, dtype):
    """Keys and values [tokens, kv heads, head_dim] that the requests of a step left in one layer, end to end."""
    shape = (tokens, cfg["num_key_value_heads"], cfg["head_dim"])
    return [_normal(seed, f"{what}{layer}", shape, torch.bfloat16).to(dtype) for what in "kv"]


# ------------------------------------------------------------------ the engine
def _engine(cfg, tensors, dtype, **limits):
    config = config_from_dict(cfg)
    model = Model(config.plan())
    model.bind(tensors, dtype)
    return Engine((config, model), device="cuda:0", dtype=dtype, block_size=PAGE, **limits)


def prepare(case, seed):
    if case["kind"] == "generate":
        cfg = MODELS[case["model"]]
        tensors = {n: _qwen3_tensor(seed, n, s, torch.float32) for n, s in _qwen3_shapes(cfg).items()}
        lengths = [1 + n for n in _numbers(seed, "lengths", case["prompts"], case["longest"])]
        lengths[0] = case["longest"]
        prompts = [_numbers(seed, f"prompt{i}", n, cfg["vocab_size"]) for i, n in enumerate(lengths)]
        engine = _engine(cfg, tensors, torch.float32, max_batch=case["prompts"], max_len=256,
                         max_new_tokens=case["new"], token_budget=case["budget"], warmup=True)
        return {"case": case, "engine": engine, "prompts": prompts, "seed": seed}
    if case["kind"] == "design":
        tensors = {n: _bofusun_tensor(seed, n, s) for n, s in _bofusun_shapes().items()}
        engine = _engine(BOFUSUN, tensors, torch.bfloat16, max_batch=1, max_len=MAX_LEN, token_budget=2048,
                         num_blocks=2048 // PAGE + 1)
        requests = [(_numbers(seed, "ids", case["tokens"], 32000), 0)]
    else:
        cfg, dtype = MODELS[case["model"]], DTYPES[case["dtype"]]
        tensors = {n: _qwen3_tensor(seed, n, s, dtype) for n, s in _qwen3_shapes(cfg).items()}
        requests = _entries(case, seed)
        pages = sum(-(-(start + len(ids)) // PAGE) for ids, start in requests)
        engine = _engine(cfg, tensors, dtype, max_batch=len(requests), max_len=MAX_LEN, token_budget=2048,
                         num_blocks=pages)
        del tensors
        _fill_cache(engine.cache, cfg, seed, requests, dtype)
    state = {"case": case, "engine": engine, "requests": requests,
             "sampling": [SamplingArgs(case.get("temperature", 0.0), seed & 0xFFFF, i) for i in range(len(requests))]}
    # a server is warm: every width it decodes has run once and has been recorded, its scratch exists
    for _ in range(2):
        _run_step(dict(state, requests=[(ids[:1] if i % 2 else ids[:max(1, len(ids) // 2)], start)
                                        for i, (ids, start) in enumerate(requests)]))
    return state


def _fill_cache(cache, cfg, seed, requests, dtype):
    """Open a row per request and write what it has cached into its pages."""
    pages, slots = [], []
    for row, (ids, start) in enumerate(requests):
        if start == 0:
            continue                                    # opened by each pass
        cache.assign(row)
        if not cache.reserve(row, start + len(ids)):
            raise RuntimeError("the pool is too small for the case")
        cache.commit(row, start)
        at = torch.arange(start)
        pages.append(cache.groups[0].host_table[row].long()[at // PAGE])
        slots.append(at % PAGE)
    if not pages:
        return
    pages, slots = torch.cat(pages).cuda(), torch.cat(slots).cuda()
    for layer in range(cfg["num_hidden_layers"]):
        for pool, values in zip(cache.pools(layer), _cached(seed, cfg, layer, len(pages), dtype)):
            pool[pages, :, slots] = values


def _run_step(state):
    engine = state["engine"]
    opened = []
    for row, (ids, start) in enumerate(state["requests"]):
        if start == 0:                                  # a new prompt opens its row and takes its pages
            engine.cache.assign(row)
            engine.cache.reserve(row, len(ids))
            opened.append(row)
    entries = [StepEntry(row, ids, start, [len(ids) - 1]) for row, (ids, start) in enumerate(state["requests"])]
    result = engine.runner.step(entries, state["sampling"])
    for row in opened:
        engine.cache.release(row)
    return result


def run(state):
    case = state["case"]
    if case["kind"] == "generate":
        out = state["engine"].generate(state["prompts"], max_new_tokens=case["new"], temperature=case["temperature"],
                                       seed=state["seed"])
        return torch.tensor(out)
    result = _run_step(state)
    if case.get("dtype") == "float32":
        return {"logits": result.logits, "tokens": result.tokens}
    # bfloat16: the step draws its tokens as well, but which of two logits a hundredth apart is the larger depends
    # on the order of the sums, so the logits stand for them
    return {"logits": result.logits}


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    if case["kind"] == "design":
        T, d = case["tokens"], _WIDTH
        ret, ff = 2 * d * d // 2 + 3 * d * d, 2 * d * 4 * d
        att = d * (2 * d + 2 * 512) + 16 * d
        scan = d * 4 * d * 2 + 2 * d * (128 + 32) + 128 * 2 * d
        runs = 7 * ret + 2 * (att + scan + 2 * d * d // 2 + ff)
        weights = 5 * ret + att + scan + ff + 32000 * d
        seen = T * min(T, 1024) - min(T, 1024) ** 2 // 2
        mix = 7 * 4 * T * d * 128 + 2 * (4 * seen * d + 6 * T * 2 * d * 16)
        return {"bytes": 2 * weights + 2 * T * d + 4 * 32000, "flops": 2 * T * runs + mix + 2 * 32000 * d}
    cfg = MODELS[case["model"]]
    d, V, D, L = cfg["hidden_size"], cfg["vocab_size"], cfg["head_dim"], cfg["num_hidden_layers"]
    Hq, Hkv = cfg["num_attention_heads"], cfg["num_key_value_heads"]
    linear = L * ((2 * Hq + 2 * Hkv) * D * d + 3 * d * cfg["intermediate_size"])
    if case["kind"] == "generate":
        tokens, steps = case["prompts"] * (case["longest"] // 2 + case["new"]), case["new"]
        return {"bytes": 4 * steps * (linear + V * d), "flops": 2 * tokens * (linear + V * d)}
    size = DTYPES[case["dtype"]].itemsize
    B, P, T, s = case["decodes"], case["portions"], case["tokens"], case["start"]
    context = case["context"] * (17 / 32 if case["ragged"] else 1)
    kv = B * context + P * s + B + T                     # cached tokens that are read, and those that are written
    pairs = B * (context + 1) + T * s + (T * T / (2 * P) if P else 0)
    rows = B + T
    return {"bytes": size * (linear + V * d + kv * L * 2 * Hkv * D) + 4 * (B + P) * V + size * rows * d,
            "flops": 2 * rows * linear + 2 * (B + P) * V * d + 4 * pairs * L * Hq * D}


def tolerance(case):
    if case["kind"] == "generate":
        return "exact"
    if case.get("dtype") == "float32":
        return {"rel": 2e-5, "max": 2e-4, "differ": 0.01}       # measured against 64 bits: 4.4e-6 and 2e-5
    # bfloat16 activations: 0.009 (4 layers) to 0.018 (18 layers) from 64 bits; 0.006 to 0.013 between two ways of
    # cutting the sums, whose roundings agree in most places
    return {"rel": 0.03, "max": 0.3}


# ------------------------------------------------------------------ the same in 64 bits
def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _rotate(x, positions, base):
    """x [T, heads, D]: dim j turns with dim j + D/2 by position * base^(-2j/D); float32 frequencies and angles."""
    D = x.shape[-1]
    inv = 1.0 / (base ** (torch.arange(0, D, 2, device=x.device, dtype=torch.float32) / D))
    angle = (positions.float()[:, None] * inv[None]).double()
    c, s = angle.cos()[:, None], angle.sin()[:, None]
    a, b = x[..., :D // 2], x[..., D // 2:]
    return torch.cat([a * c - b * s, b * c + a * s], dim=-1)


def _attend(q, k, v, start):
    """Causal softmax attention: q [t, Hq, D] at positions start.., k and v [start + t, Hkv, D]."""
    t, Hq, D = q.shape
    S, Hkv = k.shape[0], k.shape[1]
    out = torch.empty_like(q)
    keep = torch.arange(S, device=q.device)[None, :] <= torch.arange(start, start + t, device=q.device)[:, None]
    G = Hq // Hkv
    for h in range(Hkv):
        s = torch.einsum("tgd,sd->gts", q[:, h * G:(h + 1) * G], k[:, h]) * D ** -0.5
        p = torch.softmax(s.masked_fill_(~keep, float("-inf")), dim=-1)
        out[:, h * G:(h + 1) * G] = torch.einsum("gts,sd->tgd", p, v[:, h])
    return out


def _exact_step(case, seed):
    cfg = MODELS[case["model"]]
    shapes = _qwen3_shapes(cfg)
    eps, D = cfg["rms_norm_eps"], cfg["head_dim"]

    def w(name):
        return _qwen3_tensor(seed, name, shapes[name], torch.bfloat16).double()

    requests = _entries(case, seed)
    counts, starts = [len(ids) for ids, _ in requests], [start for _, start in requests]
    ids = torch.tensor([i for r, _ in requests for i in r], device="cuda")
    positions = torch.cat([torch.arange(s, s + n) for n, s in zip(counts, starts)]).cuda()
    x = _qwen3_tensor(seed, "model.embed_tokens.weight", shapes["model.embed_tokens.weight"], torch.bfloat16)[ids].double()
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, eps) * w(p + "input_layernorm.weight")
        q, k, v = ((h @ w(p + f"self_attn.{n}_proj.weight").T).unflatten(-1, (-1, D)) for n in "qkv")
        q = _rotate(_rms(q, eps) * w(p + "self_attn.q_norm.weight"), positions, cfg["rope_theta"])
        k = _rotate(_rms(k, eps) * w(p + "self_attn.k_norm.weight"), positions, cfg["rope_theta"])
        old_k, old_v = _cached(seed, cfg, i, sum(starts), torch.bfloat16) if sum(starts) else (k[:0], v[:0])
        o, at, old = torch.empty_like(q), 0, 0
        for n, s in zip(counts, starts):
            o[at:at + n] = _attend(q[at:at + n], torch.cat([old_k[old:old + s].double(), k[at:at + n]]),
                                   torch.cat([old_v[old:old + s].double(), v[at:at + n]]), s)
            at, old = at + n, old + s
        x = x + o.flatten(1) @ w(p + "self_attn.o_proj.weight").T
        h = _rms(x, eps) * w(p + "post_attention_layernorm.weight")
        act = torch.nn.functional.silu(h @ w(p + "mlp.gate_proj.weight").T) * (h @ w(p + "mlp.up_proj.weight").T)
        x = x + act @ w(p + "mlp.down_proj.weight").T
    last = torch.tensor(counts).cumsum(0).cuda() - 1
    h = _rms(x[last], eps) * w("model.norm.weight")
    return h @ w("model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight").T


def _conv(u, taps, bias=None):
    """Causal convolution per channel: u [T, C], taps [C, K], the last tap on the newest token."""
    T, K = u.shape[0], taps.shape[1]
    padded = torch.cat([u.new_zeros(K - 1, u.shape[1]), u])
    y = sum(taps[:, j] * padded[j:j + T] for j in range(K))
    return y if bias is None else y + bias


def _bofusun_retention(h, w, p, m, eps):
    T, H = h.shape[0], m["heads"]
    at = torch.arange(T, device=h.device)
    q = _rotate((h @ w(p + "q").T).view(T, H, -1), at, m["rot"]["base"])
    k = _rotate((h @ w(p + "k").T).view(T, H, -1), at, m["rot"]["base"]) * m["dim"] ** -0.5
    v = (h @ w(p + "v").T).view(T, H, -1)
    gap = (at[:, None] - at[None, :]).double()
    out = torch.empty_like(v)
    for i, decay in enumerate(m["decay"]):
        fade = torch.where(gap >= 0, decay ** gap.clamp(min=0), torch.zeros_like(gap))
        out[:, i] = ((q[:, i] @ k[:, i].T) * fade) @ v[:, i]
    return (_rms(out, eps).flatten(1) * torch.nn.functional.silu(h @ w(p + "g").T)) @ w(p + "o").T


def _bofusun_attention(h, w, p, m):
    T, H, window = h.shape[0], m["heads"], m["mask"]["size"]
    q, k, v = (_conv(h @ w(p + n).T + w(p + n + ".b"), w(p + n + ".conv")).unflatten(-1, (-1, 128)) for n in "qkv")
    rel = w(p + "rel")
    rows, half = rel.shape[0], rel.shape[0] // 2
    bucket = torch.tensor([n if n < half else min(rows - 1, half + int(math.floor(
        math.log(n / half) / math.log(m["bias_max"] / half) * (rows - half)))) for n in range(window)], device=h.device)
    at = torch.arange(T, device=h.device)
    gap = at[:, None] - at[None, :]
    keep = (gap >= 0) & (gap < window)
    out = torch.empty_like(q)
    for i in range(H):
        g = i // (H // m["kv_heads"])
        s = m["softcap"] * torch.tanh(q[:, i] @ k[:, g].T * m["scale"] / m["softcap"])
        s = s + rel[:, i][bucket[gap.clamp(0, window - 1)]]
        out[:, i] = torch.softmax(s.masked_fill(~keep, float("-inf")), dim=-1) @ v[:, g]
    return (out * torch.sigmoid(h @ w(p + "g").T)[:, :, None]).flatten(1) @ w(p + "o").T


def _bofusun_scan(h, w, p, m):
    inner, n, rank = m["inner"], m["state"], m["dt_rank"]
    silu = torch.nn.functional.silu
    x, z = (h @ w(p + "in").T).split(inner, dim=1)
    x = silu(_conv(x, w(p + "conv"), w(p + "conv.b")))
    dt, B, C = (x @ w(p + "x").T).split([rank, n, n], dim=1)
    dt = torch.nn.functional.softplus(dt @ w(p + "dt").T + w(p + "dt.b"))
    A = -torch.exp(w(p + "A_log"))
    state, y = x.new_zeros(inner, n), torch.empty_like(x)
    for t in range(x.shape[0]):
        state = torch.exp(dt[t][:, None] * A) * state + (dt[t] * x[t])[:, None] * B[t]
        y[t] = state @ C[t]
    return ((y + w(p + "D") * x) * silu(z)) @ w(p + "o").T


def _exact_design(case, seed):
    shapes, eps = _bofusun_shapes(), BOFUSUN["norm"]["eps"]

    def w(name):
        return _bofusun_tensor(seed, name, shapes[name]).double()

    def norm(x, name):
        return _rms(x, eps) * (1.0 + w(name))

    x = embedded = norm(w("embed")[torch.tensor(_numbers(seed, "ids", case["tokens"], 32000), device="cuda")], "embed.norm")
    for i, turn in [(0, None), (1, 0), (2, None), (1, 1), (2, None), (3, None), (4, None), (5, None)]:
        if turn is not None:
            x = x + (embedded if turn else 0.0) + w("loop.step")[turn]
        spec, p = BOFUSUN["layers"][i], f"l{i}."
        h = norm(x, p + "norm1")
        if spec["type"] == "retention":
            y = _bofusun_retention(h, w, p + "mix.", spec["mixer"], eps)
        else:
            left = _bofusun_attention(h, w, p + "mix.left.", spec["mixer"]["left"])
            right = _bofusun_scan(h, w, p + "mix.right.", spec["mixer"]["right"])
            y = 0.5 * (_rms(left, eps) * w(p + "mix.left.out") + _rms(right, eps) * w(p + "mix.right.out"))
        x = x + norm(y, p + "norm1b")
        if spec["mlp"] is not None:
            u = torch.relu(norm(x, p + "norm2") @ w(p + "mlp.up").T + w(p + "mlp.up.b"))
            x = x + norm((u * u) @ w(p + "mlp.down").T + w(p + "mlp.down.b"), p + "norm2b")
    return norm(x[-1:], "final.norm") @ w("head").T


def exact(case, seed):
    if case["kind"] == "generate":
        return None                                     # drawn tokens: whole numbers
    if case["kind"] == "design":
        return {"logits": _exact_design(case, seed)}
    logits = _exact_step(case, seed)
    return {"logits": logits, "tokens": None} if case["dtype"] == "float32" else {"logits": logits}
