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
    # both round the same sums to bfloat16 (relative 2^-9 at most, about 2^-9.3 in the 2-norm): the split weights and the
    # hardware exponentials add less than a hundredth of that
    assert off(out) <= 1.01 * off(before) + 1e-6 and off(before) < 2.0 ** -9
