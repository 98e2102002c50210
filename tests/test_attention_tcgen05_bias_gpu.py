"""The tcgen05 tile kernel with a learned bias by distance (capped scores, window, gate per head) against float64 and
beside the CUDA-core tile kernel that served such layers before: seams of key tiles and query tiles, tables shorter and
longer than the rows, several requests."""

import pytest
import torch

from test_kernels_gpu import paged_case, rand

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF = torch.bfloat16


@pytest.fixture(scope="module")
def ops():
    from socrates_b200.kernels import ops, require_kernels
    require_kernels()
    return ops


def as_int(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def exact(q, k_pool, v_pool, table, rows, pos, Hq, scale, window, cap, bias, gate):
    pages, Hkv, BS, D = k_pool.shape
    G, out = Hq // Hkv, []
    for n, (row, p) in enumerate(zip(rows, pos)):
        lo = max(0, p + 1 - window) if window else 0
        at = torch.arange(lo, p + 1, device=DEV)
        k = k_pool[table[row].long()[at // BS], :, at % BS].double()       # [keys, Hkv, D]
        v = v_pool[table[row].long()[at // BS], :, at % BS].double()
        s = torch.einsum("hgd,khd->hgk", q[n].double().view(Hkv, G, D), k).flatten(0, 1) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s = s + bias.double()[:, (p - at).clamp(max=bias.shape[1] - 1)]
        o = torch.einsum("hgk,khd->hgd", torch.softmax(s, -1).view(Hkv, G, -1), v).flatten(0, 1)
        out.append(o * torch.sigmoid(gate[n].double())[:, None])
    return torch.stack(out).flatten(1)


@pytest.mark.parametrize("Hq,Hkv,D", [(8, 2, 64), (16, 4, 128), (5, 1, 64), (4, 4, 128)])
@pytest.mark.parametrize("window,L,cap", [(0, 40, 30.0), (64, 64, 30.0), (130, 130, 0.0), (37, 500, 2.5)])
def test_bias_by_distance(ops, Hq, Hkv, D, window, L, cap):
    lens, counts = [33, 257, 64, 150], [33, 129, 1, 70]
    k_pool, v_pool, table = paged_case(lens, 16, Hkv, D, BF, seed=6)
    starts = [0]
    for c in counts:
        starts.append(starts[-1] + c)
    N = starts[-1]
    q, gate = rand(N, Hq * D, dtype=BF, seed=7), rand(N, Hq, dtype=BF, seed=8)
    bias = rand(Hq, L, dtype=torch.float32, seed=9)
    seq = as_int(starts), as_int([0, 1, 2, 3]), as_int([n - c for n, c in zip(lens, counts)])
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    out = torch.full_like(q, float("nan"))
    ops.attention_prefill_tcgen05(out, q, k_pool, v_pool, table, *seq, Hq, D ** -0.5, status, window, gate=gate, softcap=cap,
                                  dist_bias=bias)
    before = torch.full_like(q, float("nan"))
    ops.attention_bias_tile(before, q, k_pool, v_pool, table, *seq, Hq, D ** -0.5, window, cap, bias, gate=gate)
    rows = [r for r, c in enumerate(counts) for _ in range(c)]
    pos = [n - c + i for n, c in zip(lens, counts) for i in range(c)]
    want = exact(q, k_pool, v_pool, table, rows, pos, Hq, D ** -0.5, window, cap, bias, gate)
    off = lambda x: float((x.double() - want).norm() / want.norm())
    assert int(status) == 0
    # both round the same float32 sums to bfloat16 (relative 2^-9 at most, about 2^-9.3 in the 2-norm), which differ by some
    # 2^-21 of themselves: in quadrature that is less than 2^-20 of the error
    assert off(out) <= (1 + 2.0 ** -16) * off(before) and off(before) < 2.0 ** -9


@pytest.mark.parametrize("Hq,Hkv,D", [(8, 2, 64), (16, 4, 128)])
@pytest.mark.parametrize("window,L,cap", [(0, 40, 30.0), (130, 130, 0.0), (37, 500, 2.5)])
def test_bias_by_distance_keeps_float32_weights(ops, Hq, Hkv, D, window, L, cap):
    """The rows before they are rounded.  Weights of 24 bits, float32 sums of a few hundred terms: some 2^-21 in the 2-norm.
    Weights of two bfloat16 terms are off by up to 2^-18 each, 2^-19.2 in the 2-norm of one, and 1.6e-6 and more here."""
    lens, counts = [33, 257, 64, 150], [33, 129, 1, 70]
    k_pool, v_pool, table = paged_case(lens, 16, Hkv, D, BF, seed=6)
    q = rand(sum(counts), Hq * D, dtype=BF, seed=7)
    bias = rand(Hq, L, dtype=torch.float32, seed=9)
    seq = as_int([0, 33, 162, 163, 233]), as_int([0, 1, 2, 3]), as_int([n - c for n, c in zip(lens, counts)])
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    out = torch.full(q.shape, float("nan"), device=DEV)
    ops.attention_prefill_tcgen05(None, q, k_pool, v_pool, table, *seq, Hq, D ** -0.5, status, window, softcap=cap,
                                  dist_bias=bias, out_float=out)
    rows = [r for r, c in enumerate(counts) for _ in range(c)]
    pos = [n - c + i for n, c in zip(lens, counts) for i in range(c)]
    open_gate = torch.full((q.shape[0], Hq), float("inf"), device=DEV)
    want = exact(q, k_pool, v_pool, table, rows, pos, Hq, D ** -0.5, window, cap, bias, open_gate)
    assert int(status) == 0 and float((out.double() - want).norm() / want.norm()) < 2.0 ** -20


def test_bias_of_the_lowest_value(ops):
    """A bias that rules keys out (the type's lowest value, minus infinity) and one row whose every key has the lowest."""
    Hq, Hkv, D = 4, 2, 64
    k_pool, v_pool, table = paged_case([150], 16, Hkv, D, BF, seed=6)
    q, gate = rand(150, Hq * D, dtype=BF, seed=7), rand(150, Hq, dtype=BF, seed=8)
    bias = rand(Hq, 40, dtype=torch.float32, seed=9)
    bias[0], bias[1, 3:], bias[2, 7:] = torch.finfo(torch.float32).min, torch.finfo(torch.float32).min, -float("inf")
    seq = as_int([0, 150]), as_int([0]), as_int([0])
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    out, before = torch.empty_like(q), torch.empty_like(q)
    ops.attention_prefill_tcgen05(out, q, k_pool, v_pool, table, *seq, Hq, D ** -0.5, status, 0, gate=gate, softcap=5.0,
                                  dist_bias=bias)
    ops.attention_bias_tile(before, q, k_pool, v_pool, table, *seq, Hq, D ** -0.5, 0, 5.0, bias, gate=gate)
    # one rounding to bfloat16 apart (2^-8 of a value where it falls on the other side)
    assert int(status) == 0 and bool(before.isfinite().all()) and torch.allclose(out.float(), before.float(), rtol=2.0 ** -7, atol=1e-5)


def test_a_table_wider_than_the_tile_kernel_takes(ops):
    """Short rows in a cache of very long ones: the tile kernel refuses the table, the CUDA-core kernel serves it."""
    from socrates_b200.kernels.library import KernelError
    Hq, Hkv, D = 4, 2, 64
    k_pool, v_pool, table = paged_case([70], 16, Hkv, D, BF, seed=6)
    wide = torch.zeros(1, 4097, dtype=torch.int32, device=DEV)
    wide[:, :table.shape[1]] = table
    q, gate, bias = rand(70, Hq * D, dtype=BF, seed=7), rand(70, Hq, dtype=BF, seed=8), rand(Hq, 40, dtype=torch.float32, seed=9)
    seq, status = (as_int([0, 70]), as_int([0]), as_int([0])), torch.zeros(1, dtype=torch.int32, device=DEV)
    assert not ops.attention_tcgen05_pages_supports(k_pool, wide)
    assert ops.attention_tcgen05_pages_supports(k_pool, wide[:, :4096])
    out, narrow = torch.empty_like(q), torch.empty_like(q)
    with pytest.raises(KernelError):
        ops.attention_prefill_tcgen05(out, q, k_pool, v_pool, wide, *seq, Hq, D ** -0.5, status, 0, gate=gate, dist_bias=bias)
    ops.attention_bias_tile(out, q, k_pool, v_pool, wide, *seq, Hq, D ** -0.5, 0, 30.0, bias, gate=gate)
    ops.attention_bias_tile(narrow, q, k_pool, v_pool, table, *seq, Hq, D ** -0.5, 0, 30.0, bias, gate=gate)
    assert torch.equal(out, narrow)
