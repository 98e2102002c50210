"""Grouped-query attention over the paged cache, with per-head QK-RMSNorm and rotation.

Formulas in the reference's order (model/qwen/qwen_kv_paged.py:130-175):
q, k, v = x Wq^T, x Wk^T, x Wv^T, viewed as heads of head_dim; q and k are RMS-normed
over head_dim with gains shared by all heads, then rotated by position; k and v go to
the row's pages; query head h attends over KV head h // G with scale head_dim^-0.5,
causally, optionally only over the last `window` keys; heads are concatenated and
projected by Wo.  The three projections are one matrix product here (the weights are
concatenated when they are bound).

Unlike the reference, whose prompt attention only sees the keys of the same call
(:166-174), every query reads its keys from the pages, so a prompt may arrive in
portions and portions of prompts share a step with decode tokens.
"""

from __future__ import annotations

import os
from typing import Dict, Mapping, Optional, Sequence

import torch

from ..cache.manager import CacheNeeds, PagedKVSpec
from ..kernels import ops
from ..kernels.layer_calls import replayable
from .base import Branch, ParamSpec, Part, build_part, register_part
from .linear import Linear


def paged_partition() -> Optional[int]:
    """PAGED_PARTITION as in the reference (model/kernels/__init__.py:23-41): keys per partition of
    the split-key decode attention, 0 = one pass over all keys; None for "auto" or unset."""
    v = os.environ.get("PAGED_PARTITION", "auto").strip().lower()
    if v in ("", "auto"):
        return None
    n = int(v)
    if n < 0:
        raise ValueError(f"PAGED_PARTITION must be 'auto' or a non-negative integer, not {v!r}")
    return n


def partitions_in(places: int, blocks: int, most: int = 16) -> int:
    """Key partitions of the split-key decode kernel for `blocks` (token, KV head) pairs on a GPU that holds `places` of its
    blocks at once: as many as keep every block resident, at most `most` and at most 16."""
    parts = max(1, min(places // max(1, blocks), most, 16))
    # 3 and 4 partitions are clusters that do not fill the last places of every GPC: with 9 rows of 8 KV heads
    # 4 partitions (288 of 296 places) take 26 us for 2,048 keys where 3 take 19, with 12 rows of 4,000 keys 3 take 56 us
    # and 2 take 42; 11 rows and 3 (264 places) still fit.
    while 3 <= parts <= 4 and blocks * parts > 0.9 * places:
        parts -= 1
    return parts


def decode_partitions(ctx, num_kv_heads: int, blocks_per_sm: int, keys_per_part: int) -> int:
    """Into how many key partitions the split-key decode kernel cuts each token's keys when
    PAGED_PARTITION is "auto": as many as keep every block resident at once (one wave, no tail),
    at most 16, never less than `keys_per_part` keys of the longest possible row in a partition.
    A function of the batch width and of limits only, so that a recorded graph stays valid."""
    return partitions_in(ctx.num_sms * blocks_per_sm, max(1, num_kv_heads * ctx.num_tokens),
                         max(1, -(-ctx.max_context // keys_per_part)))


# In a step that mixes prompt portions with decoding requests the tile kernel can serve both (a decoding request is a tile
# of one token: its key tiles one after the other, 1.1 us each and more).  From this many keys in the longest such request
# on, the decoding requests run in the equal-shares kernel beside it, one launch more.  Measured (8B shape, 12 layers, two
# prompts of 511 beside 37 requests, ms a step, together / apart): 512 keys 6.10 / 6.29, 1,024: 6.46 / 6.39, 2,048: 7.03 /
# 6.48, 4,096: 8.20 / 6.79.
SINGLES_APART_FROM = 1024


def balanced_attention(ctx, out, q, k_pool, v_pool, table, num_heads: int, scale: float, window: int) -> None:
    """The step's requests of one token through the equal-shares decode kernel, with scratch of the step."""
    Hkv, D, R = k_pool.shape[1], k_pool.shape[3], ctx.num_seqs
    shares = ops.attention_balanced_shares(num_heads, Hkv, D, R, ctx.num_sms)
    take = ctx.buffers.take_flat
    ops.attention_decode_balanced(out, q, k_pool, v_pool, table, ctx.seq_starts, ctx.seq_rows, ctx.seq_first_pos,
                                  num_heads, scale, window, shares,
                                  take("attn_share_o", num_heads * shares * 2 * D, torch.float32),
                                  take("attn_share_ml", num_heads * shares * 2 * 2, torch.float32),
                                  take("attn_share_counters", ctx.buffers.max_rows * Hkv, torch.int32, zeroed=True))


def paged_attention(ctx, out, q, k_pool, v_pool, table, num_heads: int, scale: float, window: int,
                    max_len: int) -> None:
    """Causal attention of every token of the step over its row's pages; this mixer's choice of kernel.

    bfloat16, a step in which every request brings one token (decode):
      * PAGED_PARTITION "auto": the split-key kernel (mma.sync), the partition COUNT chosen from
        the batch width so that one wave of blocks fills the GPU, or, where the rows' lengths differ so much
        that the longest would run on alone (`prefers_shares`), the equal-shares kernel.  Fastest; a
        request's numbers differ in rounding with the batch it is in.
      * PAGED_PARTITION = n: the streaming kernel over chunks of n keys at fixed key positions (the
        reference's meaning of the variable, model/kernels/csrc/paged_attention.cu:80-96; 0 = the
        whole row in one pass).  A request's numbers are the same bits alone and in a full batch;
        measured 12 to 25 % slower per decode step than "auto" on the 4B shape.
    bfloat16, other steps: the tile kernels (tcgen05 for head sizes 64 and 128, mma.sync for 16 and
    32); beside the tcgen05 kernel, decoding requests with long rows in the equal-shares kernel.  Everything else (the float32 engine above all): the SIMT kernel, whose split depends on
    `max_len` of the cache alone, so the float32 engine's numbers never depend on the batch.
    """
    Hkv, page_size, D = k_pool.shape[1], k_pool.shape[2], k_pool.shape[3]
    N = q.shape[0]
    bf16 = q.dtype == torch.bfloat16
    if bf16 and not ctx.all_decode:
        if ctx.status is not None and ops.attention_tcgen05_supports(num_heads, Hkv, D, page_size):
            apart = (paged_partition() is None and ctx.longest_single >= SINGLES_APART_FROM
                     and ops.attention_balanced_supports(num_heads, Hkv, D, page_size, ctx.num_seqs))
            ops.attention_prefill_tcgen05(out, q, k_pool, v_pool, table, ctx.seq_starts, ctx.seq_rows,
                                          ctx.seq_first_pos, num_heads, scale, ctx.status, window, skip_single=apart, meta_older=True)
            if apart:
                balanced_attention(ctx, out, q, k_pool, v_pool, table, num_heads, scale, window)
            return
        if ops.attention_mma_supports(num_heads, Hkv, D, page_size, False):
            ops.attention_prefill_mma(out, q, k_pool, v_pool, table, ctx.seq_starts, ctx.seq_rows,
                                      ctx.seq_first_pos, num_heads, scale, window)
            return
    fixed = paged_partition()
    take = ctx.buffers.take_flat
    if (bf16 and ctx.all_decode and fixed is not None and N <= 1024      # the kernel's limit of tokens a launch
            and ops.attention_decode_stream_supports(num_heads, Hkv, D, page_size)):
        chunk = max(16, -(-(fixed if fixed > 0 else max_len) // 16) * 16)
        span = min(max_len, window) if window else max_len
        chunks = 1 if chunk >= max_len else -(-span // chunk) + 1          # a span may straddle one edge more
        part_o = part_ml = counters = None
        if chunks > 1:
            part_o = take("attn_part_o", N * num_heads * chunks * D, torch.float32)
            part_ml = take("attn_part_ml", N * num_heads * chunks * 2, torch.float32)
            counters = take("attn_counters", ctx.buffers.max_rows * Hkv, torch.int32, zeroed=True)
        ops.attention_decode_stream(out, q, k_pool, v_pool, table, ctx.token_rows, ctx.positions, num_heads,
                                    scale, window, chunk, chunks, part_o, part_ml, counters,
                                    variant=int(os.environ.get("SOCRATES_DECODE_VARIANT", "1")))
        return
    use_mma = bf16 and ctx.all_decode and ops.attention_mma_supports(num_heads, Hkv, D, page_size, True)
    if use_mma:
        NP = decode_partitions(ctx, Hkv, ops.attention_decode_mma_blocks_per_sm(D), 128)
        if ctx.share_keys and ops.attention_balanced_supports(num_heads, Hkv, D, page_size, ctx.num_seqs):
            balanced_attention(ctx, out, q, k_pool, v_pool, table, num_heads, scale, window)
            return
    else:
        # SIMT: a partition is ceil(pages of the row / NP) pages, so a fixed NP cuts a row by its own length alone
        keys_per_part = 4 * page_size if fixed is None else fixed
        NP = 1 if keys_per_part == 0 else max(1, min(-(-max_len // keys_per_part), 16))
    part_o = part_ml = None
    if NP > 1:
        part_o = take("attn_part_o", N * num_heads * NP * D, torch.float32)
        part_ml = take("attn_part_ml", N * num_heads * NP * 2, torch.float32)
    if use_mma:
        ops.attention_decode_mma(out, q, k_pool, v_pool, table, ctx.token_rows, ctx.positions, num_heads,
                                 scale, window, NP, part_o, part_ml)
    else:
        ops.attention_simt(out, q, k_pool, v_pool, table, ctx.token_rows, ctx.positions, num_heads, scale,
                           window, NP, part_o, part_ml)


@replayable("forward", constants=("Hq", "Hkv", "D", "scale", "qk_norm_eps", "window"), optional=("q_gain", "k_gain"),
            parts=lambda self: (self.position, self.qkv, self.o))
class GQAAttention(Part):
    def __init__(self, spec, name):
        super().__init__(spec, name)
        p = spec.params
        self.hidden = int(p["hidden_size"])
        self.Hq = int(p["num_heads"])
        self.Hkv = int(p["num_kv_heads"])
        self.D = int(p["head_dim"])
        self.scale = float(p.get("scale", self.D ** -0.5))
        self.qk_norm_eps = p.get("qk_norm_eps")          # None: no QK-norm
        self.window: Optional[int] = p.get("window")
        self.position = build_part("position", p["position"], "")
        if self.Hq % self.Hkv:
            raise ValueError(f"{self.Hq} query heads are no multiple of {self.Hkv} KV heads")
        if self.D % 16 or not 16 <= self.D <= 256:
            raise ValueError(f"head_dim {self.D} must be a multiple of 16 between 16 and 256")
        self.qkv: Optional[Linear] = None
        self.o: Optional[Linear] = None
        self.q_gain = self.k_gain = None

    def parameters(self) -> Dict[str, ParamSpec]:
        n, D = self.name, self.D
        out = {
            n + "q_proj.weight": ParamSpec((self.Hq * D, self.hidden)),
            n + "k_proj.weight": ParamSpec((self.Hkv * D, self.hidden)),
            n + "v_proj.weight": ParamSpec((self.Hkv * D, self.hidden)),
            n + "o_proj.weight": ParamSpec((self.hidden, self.Hq * D)),
        }
        if self.qk_norm_eps is not None:
            out[n + "q_norm.weight"] = ParamSpec((D,), role="gain", init="gain")
            out[n + "k_norm.weight"] = ParamSpec((D,), role="gain", init="gain")
        return out

    def bind(self, tensors: Mapping[str, torch.Tensor], dtype) -> None:
        n = self.name
        self.qkv = Linear(torch.cat([tensors[n + "q_proj.weight"], tensors[n + "k_proj.weight"],
                                     tensors[n + "v_proj.weight"]], dim=0))
        self.o = Linear(tensors[n + "o_proj.weight"])
        self.position.tables(self.o.weight.device)      # made now: no copy from the host inside a step
        if self.qk_norm_eps is not None:
            self.q_gain = tensors[n + "q_norm.weight"]
            self.k_gain = tensors[n + "k_norm.weight"]

    def cache_needs(self) -> CacheNeeds:
        return CacheNeeds(paged=PagedKVSpec(self.Hkv, self.D, self.window))

    def streamed_weights(self):
        """The weight matrices in the order in which forward() reads them."""
        return [self.qkv.weight, self.o.weight]

    def prefers_shares(self, lengths: Sequence[int], num_sms: int) -> bool:
        """Whether a decode step over rows of so many keys should deal them in equal shares (attention_balanced.cu)
        rather than cut every row into the same number of partitions.

        In tiles of 64 keys, a block of the split-key kernel takes ceil(longest / partitions) and one of the other T / W;
        a row that two shares cut costs both a merge through memory, and the launch about 4 us.  (A short cache may leave
        fewer partitions than counted here; they hold 128 keys then, two tiles.)  Measured (us a launch in a graph, keys in
        no cache, 32 query and 8 KV heads of 128, split-key / shares; `a to b`: lengths evenly spaced; in brackets the tiles
        that a split-key block has more): 9 rows of 4,000 keys (6) 30.0 / 31.7, 12 of 2,000 (6) 24.9 / 24.5, 18 of 125 to
        2,000 (8) 23.6 / 22.4, 32 of 4,000 (8) 81.0 / 86.7, 16 of 125 to 2,000 (9) 22.3 / 20.6, 13 of 4,000 (10) 41.9 / 41.5,
        24 of 2,000 (11) 40.1 / 39.5, 12 of 4,000 (12) 41.8 / 38.8, 10 of 250 to 4,000 (12) 27.1 / 23.7, 19 of 2,000 (16)
        38.9 / 33.2, 12 of 250 to 4,000 (21) 36.5 / 25.5; 16 KV heads: 6 of 4,000 (11) 41.0 / 37.5; 4: 24 of 4,000 (12) 43.1 /
        41.1; 2: 36 of 250 to 4,000 (13) 27.7 / 25.9.  So from 8 tiles on.  More rows than shares are no partitions but whole
        rows in a second round of blocks: 64 rows of 512 keys 27.6 / 30.2, 48 of 1,000 45.8 / 39.8, 64 of 2,048 85.8 / 88.6,
        64 of 128 to 2,048 57.9 / 57.4, 64 of 256 to 4,096 109.4 / 97.7: from 16 tiles in the longest row on."""
        N = len(lengths)
        if N < 5 or paged_partition() is not None:          # few rows are cut into many partitions each: even anyway
            return False
        if not ops.attention_balanced_supports(self.Hq, self.Hkv, self.D, 16, N):       # (on pages of the usual size)
            return False
        parts = partitions_in(num_sms * ops.attention_decode_mma_blocks_per_sm(self.D), self.Hkv * N)
        shares = ops.attention_balanced_shares(self.Hq, self.Hkv, self.D, N, num_sms)
        if self.window:
            lengths = [min(n, self.window) for n in lengths]
        longest = -(-max(lengths) // 64)
        if N > shares:
            return longest >= 16
        total = sum(lengths) / 64 + N / 2
        return -(-longest // parts) - total / shares >= 8

    def forward(self, ctx, x: torch.Tensor, cache) -> Branch:
        N = x.shape[0]
        qkv = self.qkv(ctx, x, "qkv", out="model_or_partial")
        q = ctx.buffers.take("q", N, (self.Hq * self.D,), ctx.dtype)
        k_pool, v_pool = cache.pools()
        table = cache.block_table()
        inv_freq, rotary_dim = self.position.tables(x.device)
        eps = self.qk_norm_eps if self.qk_norm_eps is not None else 0.0
        ops.qk_norm_rope_kvwrite(
            qkv, q, k_pool if cache.writes else None, v_pool if cache.writes else None,
            self.q_gain, self.k_gain, inv_freq, rotary_dim, ctx.positions, ctx.token_rows, table,
            eps, self.Hq, self.Hkv, self.D, magnitude=getattr(self.position, "magnitude", 1.0))
        attn = ctx.buffers.take("attn", N, (self.Hq * self.D,), ctx.dtype)
        paged_attention(ctx, attn, q, k_pool, v_pool, table, self.Hq, self.scale, self.window or 0,
                        cache.manager.max_len)
        return Branch(self.o(ctx, attn, "branch", out="partial"))


register_part("mixer", "gqa_attention", GQAAttention)
