"""The equal-shares decode-attention kernel alone against the float64 reference: rows of one key to many beside
requests of several tokens (which it must leave alone), shares that cut a row many times or hold many rows, tile
and page seams, windows, group sizes 1 to 16, head sizes 16 to 128, and that its counters end at zero."""

import pytest
import torch

from test_kernels_gpu import paged_case, rand

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF = torch.bfloat16
# bfloat16 output (relative 2^-9, doubled for the value it is compared with) of sums whose weights are carried as
# two bfloat16 terms
TOL = dict(atol=2e-3, rtol=1.6e-2)


def as_int(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


@pytest.fixture(scope="module")
def ops():
    from socrates_b200.kernels import ops, require_kernels
    require_kernels()
    return ops


@pytest.fixture(scope="module")
def ref():
    from socrates_b200.kernels import reference
    return reference


def check(ops, ref, lens, counts, BS, Hq, Hkv, D, window, shares, seed=3):
    """`counts[r]` new tokens at the end of request r's `lens[r]` positions; cache rows in reverse order."""
    k_pool, v_pool, table = paged_case(lens, BS, Hkv, D, BF, seed=seed)
    R = len(lens)
    order = list(range(R))[::-1]
    starts = [0]
    for r in order:
        starts.append(starts[-1] + counts[r])
    N = starts[-1]
    q = rand(N, Hq * D, dtype=BF, seed=seed + 1)
    seq = as_int(starts), as_int(order), as_int([lens[r] - counts[r] for r in order])
    scratch = (torch.full((Hq * shares * 2 * D,), float("nan"), device=DEV),
               torch.full((Hq * shares * 2 * 2,), float("nan"), device=DEV),
               torch.zeros(R * Hkv, dtype=torch.int32, device=DEV))
    outs = []
    for _ in range(2):                                  # the counters are ready for a second call, the bits the same
        out = torch.full_like(q, 7.0)
        ops.attention_decode_balanced(out, q, k_pool, v_pool, table, *seq, Hq, D ** -0.5, window, shares, *scratch)
        assert int(scratch[2].abs().sum()) == 0
        outs.append(out)
    assert torch.equal(*outs)
    single = [s for s, r in zip(starts, order) if counts[r] == 1]
    rows = [r for r in order if counts[r] == 1]
    want = ref.paged_attention_ref(q[single], k_pool, v_pool, table, as_int(rows), as_int([lens[r] - 1 for r in rows]),
                                   Hq, D ** -0.5, window)
    assert torch.allclose(outs[0][single].double(), want, **TOL)
    others = [t for t in range(N) if t not in set(single)]
    assert bool((outs[0][others] == 7.0).all())


@pytest.mark.parametrize("Hq,Hkv,D", [(4, 2, 16), (8, 2, 32), (8, 8, 64), (32, 8, 128), (16, 1, 64), (12, 1, 128),
                                      (10, 2, 128)])
@pytest.mark.parametrize("window", [0, 37, 130])
@pytest.mark.parametrize("shares", [1, 3, 7, 40])
def test_balanced(ops, ref, Hq, Hkv, D, window, shares):
    lens = [1, 15, 1500, 65, 9, 130, 257, 700, 63, 128, 5]
    counts = [1, 1, 1, 1, 9, 1, 1, 1, 7, 1, 1]
    check(ops, ref, lens, counts, 16, Hq, Hkv, D, window, shares)


@pytest.mark.parametrize("BS", [1, 8, 32, 64, 128])
def test_balanced_page_sizes(ops, ref, BS):
    check(ops, ref, [1, BS, BS + 1, 5 * BS + 3, 300], [1] * 5, BS, 8, 2, 64, 0, 5)


def test_balanced_one_long_row_and_many_short(ops, ref):
    check(ops, ref, [7001] + [3 + 7 * i for i in range(140)], [1] * 141, 16, 32, 8, 128, 0, 37)


def test_balanced_no_single_token(ops):
    k_pool, v_pool, table = paged_case([40], 16, 2, 64, BF)
    q = rand(5, 256, dtype=BF, seed=1)
    out = torch.full_like(q, 7.0)
    ops.attention_decode_balanced(out, q, k_pool, v_pool, table, as_int([0, 5]), as_int([0]), as_int([35]), 4, 0.125, 0, 4,
                                  torch.empty(4 * 4 * 2 * 64, device=DEV), torch.empty(4 * 4 * 2 * 2, device=DEV),
                                  torch.zeros(2, dtype=torch.int32, device=DEV))
    assert bool((out == 7.0).all())


@pytest.mark.parametrize("Hq,Hkv,D", [(8, 2, 64), (32, 8, 128)])
def test_mixed_step_in_two_kernels(ops, ref, Hq, Hkv, D):
    """The tile kernel without the requests of one token and this kernel for them write every row between them."""
    lens, counts = [1500, 70, 1, 300, 33, 2], [1, 70, 1, 129, 1, 2]
    k_pool, v_pool, table = paged_case(lens, 16, Hkv, D, BF, seed=2)
    starts = [0]
    for c in counts:
        starts.append(starts[-1] + c)
    seq = as_int(starts), as_int(list(range(6))), as_int([n - c for n, c in zip(lens, counts)])
    q = rand(starts[-1], Hq * D, dtype=BF, seed=4)
    out = torch.full_like(q, float("nan"))
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.attention_prefill_tcgen05(out, q, k_pool, v_pool, table, *seq, Hq, D ** -0.5, status, skip_single=True)
    single = [s for s, c in zip(starts, counts) if c == 1]
    assert bool(out[single].isnan().all()) and int(out.isnan().any(1).sum()) == len(single)
    ops.attention_decode_balanced(out, q, k_pool, v_pool, table, *seq, Hq, D ** -0.5, 0, 5,
                                  torch.empty(Hq * 5 * 2 * D, device=DEV), torch.empty(Hq * 5 * 4, device=DEV),
                                  torch.zeros(6 * Hkv, dtype=torch.int32, device=DEV))
    rows = [r for r, c in enumerate(counts) for _ in range(c)]
    pos = [n - c + i for n, c in zip(lens, counts) for i in range(c)]
    want = ref.paged_attention_ref(q, k_pool, v_pool, table, as_int(rows), as_int(pos), Hq, D ** -0.5, 0)
    assert int(status) == 0 and torch.allclose(out.double(), want, **TOL)


def test_when_keys_are_dealt_in_shares(ops):
    """Rows alike, short or few keep their partitions; one long row among short ones does not."""
    from socrates_b200.config.plan import PartSpec
    from socrates_b200.parts.attention import GQAAttention
    part = GQAAttention(PartSpec("gqa_attention", dict(hidden_size=64, num_heads=32, num_kv_heads=8, head_dim=128,
                                                       position=PartSpec("none", {}))), "")
    dealt = lambda lengths: part.prefers_shares(lengths, 148)
    assert not dealt([8000]) and not dealt([8000] + [1] * 3) and not dealt([2048] * 8) and not dealt([2048] * 32)
    assert not dealt([500] * 64) and not dealt([60] * 200)
    assert dealt([7001] + [437] * 18) and dealt([4096] + [256] * 63) and dealt([4000] * 4 + [250] * 8)
