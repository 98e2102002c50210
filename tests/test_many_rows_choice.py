"""Which kernel a product of 257 rows and more whose output is partial sums runs on, from its shape (no GPU: the two host
functions of the library that the choice asks are stated here for 148 SMs)."""

import pytest
import torch

from socrates_b200.engine import context
from socrates_b200.engine.context import Buffers, StepContext


def shares_parts(M, N, K):
    tiles, blocks = -(-M // 256) * -(-N // 256), -(-K // 64)
    smallest = tiles * blocks // min(74, tiles * blocks)
    parts = -(-(blocks - 1) // smallest) + 1
    return parts if M > 256 and N >= 256 and parts <= 4 else 0


def splits(K, wanted):
    blocks = -(-K // 64)
    return -(-blocks // -(-blocks // max(1, min(wanted, blocks))))


@pytest.fixture()
def chosen(monkeypatch):
    monkeypatch.setattr(context.ops, "gemm_tcgen05_shares_parts", shares_parts)
    monkeypatch.setattr(context.ops, "gemm_tcgen05_splits", splits)
    monkeypatch.delenv("SOCRATES_GEMM_SHARES", raising=False)
    ctx = StepContext(torch.bfloat16, torch.device("cpu"), Buffers(64, "cpu"), 1, 1, None, None, None, None, None, None, None,
                      all_decode=False, max_context=1, num_sms=148, status=torch.zeros(1, dtype=torch.int32))

    def choice(M, N, K, shares=True):
        w = torch.empty(N, K, dtype=torch.bfloat16, device="meta")
        parts = ctx.gemm_splits(M, w, torch.bfloat16, shares=shares)
        if parts == 1:
            return "whole"
        return f"{'shares' if shares and parts == ctx.gemm_shares(M, w, torch.bfloat16) else 'cut'} {parts}"
    return choice


@pytest.mark.parametrize("shape,choices", [
    # o and down of 4B, 8B and 32B
    ((2560, 4096), {257: "cut 4", 385: "cut 3", 512: "cut 3", 513: "whole", 640: "whole", 896: "whole", 897: "whole", 1024: "whole"}),
    ((2560, 9728), {257: "cut 4", 512: "cut 3", 513: "whole", 640: "whole", 896: "whole", 897: "whole", 1152: "whole",
                    1153: "shares 3", 1280: "shares 3", 1281: "whole", 2048: "shares 2"}),
    ((4096, 4096), {257: "cut 3", 384: "cut 3", 385: "whole", 512: "whole", 513: "whole", 896: "whole", 1153: "shares 2"}),
    ((4096, 12288), {257: "cut 3", 384: "cut 3", 385: "cut 2", 512: "cut 2", 513: "whole", 896: "whole"}),     # beyond the cache
    ((5120, 8192), {257: "whole", 384: "whole", 385: "whole", 640: "whole", 896: "whole", 897: "shares 2", 1024: "shares 2"}),
    ((5120, 25600), {257: "cut 2", 384: "cut 2", 385: "whole", 896: "whole"}),
    # narrower models
    ((2048, 4096), {512: "cut 4", 513: "cut 3", 768: "cut 3", 769: "whole", 1023: "whole"}),
    ((1024, 3072), {513: "cut 4", 1023: "cut 4", 1024: "whole"}),
])
def test_partial_sums(chosen, shape, choices):
    assert {M: chosen(M, *shape) for M in choices} == choices


def test_a_refusal_is_for_the_kernel_that_then_runs(chosen):
    """Where equal shares serve a shape, what runs instead is whole tiles, whose cost they were weighed with, or a cut in
    three or more, never a cut in two."""
    for N, K in ((2560, 4096), (2560, 9728), (4096, 4096), (5120, 8192), (2048, 2048), (2048, 8192), (5120, 5120)):
        for M in range(257, 4097):
            if (M + N) * K * 2 <= 96 << 20 and shares_parts(M, N, K):
                assert chosen(M, N, K) != "cut 2", (M, N, K)


def test_without_shares_the_cut_is_as_it_was(chosen):
    assert chosen(300, 6144, 2560, shares=False) == "cut 2"
    assert chosen(640, 2560, 4096, shares=False) == "cut 2"
    assert chosen(1024, 2560, 4096, shares=False) == "whole"
