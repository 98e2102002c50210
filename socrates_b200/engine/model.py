"""A model built from a plan: embedding, layers run in the plan's order, norm, head.

Nothing here names an architecture.  `Model(plan)` builds every part through the part
registries; `parameters()` lists the tensors the checkpoint must hold; `bind()` hands
them out; `forward(ctx, cache)` runs one step and returns float32 logits at the rows
named by `ctx.logit_index`.
"""

from __future__ import annotations

from typing import Dict, List, Mapping, Optional

import torch

from ..cache.manager import CacheNeeds
from ..config.plan import ModelPlan
from ..kernels import ops
from ..kernels.layer_calls import Recording, layer_facts
from ..parts import ParamSpec, ResidualStream, build_part
from ..parts.base import _REGISTRIES
from .context import CacheView, StepContext


class Model:
    def __init__(self, plan: ModelPlan):
        plan.validate()
        self.plan = plan
        self.embedding = build_part("embedding", plan.embedding, plan.embedding.name)
        self.layers = []
        for spec in plan.layers:
            reg = _REGISTRIES["arrangement"]
            if spec.arrangement not in reg:
                raise KeyError(f"no arrangement {spec.arrangement!r}; known: {sorted(reg)}")
            self.layers.append(reg[spec.arrangement](spec))
        # parts that act on the stream right before a run (RunEntry.before), by order index
        self.stream_ops = {i: build_part("stream_op", e.before, e.before.name)
                           for i, e in enumerate(plan.order) if e.before is not None}
        self.keeps_embedding_output = any(getattr(op, "needs_embedding_output", False)
                                          for op in self.stream_ops.values())
        # A part may ask that the steps of its model launch their kernels one after the other (no
        # programmatic dependent launch): `serial_launches = True` on the part.
        self.dependent_launch = not any(getattr(p, "serial_launches", False)
                                        for layer in self.layers for p in getattr(layer, "parts", list)())
        dealers = {}
        for layer in self.layers:
            for p in getattr(layer, "parts", list)():
                if hasattr(p, "prefers_shares"):
                    dealers.setdefault((p.Hq, p.Hkv, p.D, p.window), p)
        self._key_dealers = list(dealers.values())
        # layers of equal specs that run after each order entry: a recording pays from the second on (the last layer's
        # products are followed by another matrix).  Whether layers are alike is for _like_another to see.
        kinds: List = []
        for spec in plan.layers:
            what = (spec.arrangement, spec.norms, spec.mixer, spec.feed_forward, spec.params)
            kinds.append(next((k for k, other in enumerate(plan.layers[:len(kinds)])
                               if what == (other.arrangement, other.norms, other.mixer, other.feed_forward, other.params)),
                              len(kinds)))
        self._alike_after = [sum(kinds[later.layer] == kinds[e.layer] for later in plan.order[i + 1:])
                             for i, e in enumerate(plan.order)]
        self.final_norm = build_part("norm", plan.final_norm, plan.final_norm.name)
        self.head = build_part("head", plan.head, plan.head.name)
        self.dtype: Optional[torch.dtype] = None

    # ------------------------------------------------------------------ weights
    def parameters(self) -> Dict[str, ParamSpec]:
        out: Dict[str, ParamSpec] = {}
        for part in (self.embedding, *self.layers, *self.stream_ops.values(), self.final_norm, self.head):
            for name, spec in part.parameters().items():
                if name in out and out[name].shape != spec.shape:
                    raise ValueError(f"{name} is asked for with shapes {out[name].shape} and {spec.shape}")
                out[name] = spec
        return out

    def duplicates(self) -> Dict[str, str]:
        """Tensors a checkpoint may hold beside the one a part reads ({file name: the name it must
        repeat}); parts say so through an optional `duplicates()`."""
        out: Dict[str, str] = {}
        for part in (self.embedding, *self.layers, self.final_norm, self.head):
            out.update(getattr(part, "duplicates", dict)())
        return out

    def bind(self, tensors: Mapping[str, torch.Tensor], dtype: torch.dtype) -> None:
        self.dtype = dtype
        for part in (self.embedding, *self.layers, *self.stream_ops.values(), self.final_norm, self.head):
            part.bind(tensors, dtype)
        # The weight matrices in the order in which a step streams them (parts that say so
        # through streamed_weights()), as a map from each one's address to its successor: a
        # kernel that streams one can ask for the head of the next in L2.
        order: List[torch.Tensor] = []
        for e in self.plan.order:
            order.extend(getattr(self.layers[e.layer], "streamed_weights", list)())
        order.extend(getattr(self.head, "streamed_weights", list)())
        # (The list keeps them: an address in the map is never another tensor's.)
        self._streamed = order
        self.weight_successor: Dict[int, Optional[torch.Tensor]] = {}
        for w, nxt in zip(order, [*order[1:], None]):
            self.weight_successor.setdefault(w.data_ptr(), nxt)

    # ------------------------------------------------------------------ cache
    def cache_needs(self) -> List[Optional[CacheNeeds]]:
        """What each order entry asks of the cache manager (None where it reads another's)."""
        out: List[Optional[CacheNeeds]] = []
        for e in self.plan.order:
            out.append(None if e.reads_cache_of is not None else self.layers[e.layer].cache_needs())
        return out

    @property
    def supports_graph(self) -> bool:
        return (all(l.supports_graph for l in self.layers)
                and all(getattr(op, "supports_graph", True) for op in self.stream_ops.values()))

    def prefers_shares(self, lengths, num_sms: int) -> bool:
        """Whether a decode step over rows of so many keys should deal the keys of all rows to the GPU's blocks in equal
        shares (parts say so through an optional `prefers_shares`; asked once for layers of one shape)."""
        return any(p.prefers_shares(lengths, num_sms) for p in self._key_dealers)

    # ------------------------------------------------------------------ one step
    def _like_another(self, ctx: StepContext, stream: ResidualStream, view: CacheView, i: int,
                      recordings: Dict[tuple, tuple]) -> bool:
        """Run order entry i from the calls of an earlier layer of this step that it is like, or record its own; False: it
        is to run as any layer.  For steps that launch their kernels from here (a recorded graph needs none of this): a
        prompt portion of 187 tokens through 18 layers of the 4B shape took the host 2.9 ms in single launches, longer
        than the GPU.  What makes layers alike is looked at in every step: every class, function and constant in them, the
        device, shape, type and alignment of every tensor, what the product after each is, the pages' table and what waits
        on the stream."""
        layer = self.layers[self.plan.order[i].layer]
        waits = stream.pending
        if (ctx.host_batch is None or ctx.after_run is not None or waits is None or not waits.plain
                or stream.add_rows is not None or stream.add_vec is not None or stream.streams is not None):
            return False
        if not recordings and self._alike_after[i] < 2:
            return False
        facts, tensors = [], []
        if not layer_facts(layer, facts, tensors):
            return False
        own = {t.data_ptr() for t in tensors}
        after = []                                      # which product follows each: one of the layer's own, or another's
        for w in layer.streamed_weights():
            nxt = self.weight_successor.get(w.data_ptr())
            after.append(nxt is not None and nxt.data_ptr() in own)
            if nxt is not None and not after[-1]:
                tensors.append(nxt)
        tensors.extend(view.pools())
        table, device = view.block_table(), waits.partial.device
        if any([t.device != device for t in tensors]):
            return False                                # refused, or brought over, by the layer itself
        key = (tuple(facts), tuple(after), table.data_ptr(), table.shape, waits.partial.data_ptr(), waits.partial.shape,
               tuple([(t.shape, t.dtype, t.is_contiguous(), t.data_ptr() & 127) for t in tensors]))
        addresses = [t.data_ptr() for t in tensors]
        known = recordings.get(key)
        if known is not None and known[0].usable:
            known[0].run(addresses)
            stream.pending = known[1]
            return True
        if known is not None or self._alike_after[i] < 2:
            return False
        recording = Recording(addresses)
        with recording:
            layer.forward(ctx, stream, view)
        recordings[key] = (recording, stream.pending)
        return True

    def forward(self, ctx: StepContext, cache) -> torch.Tensor:
        ctx.weight_successor = self.weight_successor
        ctx.dependent_launch = self.dependent_launch
        ops.set_dependent_launch(self.dependent_launch)
        stream = ResidualStream(self.embedding.forward(ctx))
        if self.keeps_embedding_output:
            # the residual is updated in place from here on: a stream op that adds the embedding's
            # output again later reads this copy
            keep = ctx.buffers.take("embedding_output", ctx.num_tokens, (self.plan.hidden_size,), torch.float32)
            keep.copy_(stream.residual)
            stream.embedding_output = keep
        recordings: Dict[tuple, tuple] = {}
        for i, e in enumerate(self.plan.order):
            op = self.stream_ops.get(i)
            if op is not None:
                op.apply(ctx, stream)
            src = e.reads_cache_of
            view = CacheView(cache, i if src is None else src, writes=src is None)
            if op is None and src is None and self._like_another(ctx, stream, view, i, recordings):
                continue
            self.layers[e.layer].forward(ctx, stream, view)
            if ctx.after_run is not None:
                ctx.after_run(i, stream)
        if ctx.logit_index is None:
            return None          # no logits wanted: the last branch is never needed
        h = self.final_norm.apply(ctx, stream, row_index=ctx.logit_index, buffer="normed_out")
        return self.head.forward(ctx, h)
