"""Prompt attention on tcgen05 whose offsets and block table are read before the kernel before it has ended: the same bits
as without, and right, for tiles of few tokens, requests that end inside a tile and requests that bring one token."""

import pytest
import torch

from test_attention_mma_gpu import portions
from test_attention_tcgen05_gpu import BF, TOL, paged, status
from test_kernels_gpu import rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hq,Hkv,D,BS", [(32, 8, 128, 16), (8, 8, 64, 16), (16, 1, 64, 32), (9, 3, 64, 32), (14, 2, 128, 16)])
@pytest.mark.parametrize("apart", [False, True])
def test_meta_older(Hq, Hkv, D, BS, apart):
    from socrates_b200.kernels import ops, reference, require_kernels
    require_kernels()
    lens = [300, 70, 17, 1, 129, 700]
    k_pool, v_pool, table = paged(lens, BS, Hkv, D, seed=3)
    starts, rows, firsts, trows, pos = portions([(0, 250, 50), (1, 0, 70), (2, 15, 2), (3, 0, 1), (4, 128, 1), (5, 0, 700)])
    q = rand(int(starts[-1]), Hq * D, dtype=BF, seed=4)
    st, outs = status(), []
    for older in (False, True, True):
        out = torch.full_like(q, 7.0)
        ops.attention_prefill_tcgen05(out, q, k_pool, v_pool, table, starts, rows, firsts, Hq, D ** -0.5, st,
                                      skip_single=apart, meta_older=older)
        outs.append(out)
    assert int(st.item()) == 0
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    want = reference.paged_attention_ref(q, k_pool, v_pool, table, trows, pos, Hq, D ** -0.5, 0)
    if apart:
        for r in (122, 123):
            assert bool((outs[0][r] == 7.0).all())
            want[r] = 7.0
    assert torch.allclose(outs[0].double(), want, **TOL)


@pytest.mark.parametrize("Hq,Hkv,D,BS", [(32, 8, 128, 16), (8, 8, 64, 16)])
def test_behind_kernels_that_are_still_running(Hq, Hkv, D, BS):
    """Steps one after another without a wait of the host: offsets, rows and block table come by copies, queries and pages from
    the library's own kernels, which let the next one start at once."""
    from socrates_b200.kernels import ops, require_kernels
    require_kernels()
    lens = [300, 70, 17, 90, 129, 700]
    spec = [(0, 250, 50), (1, 0, 70), (2, 15, 2), (3, 0, 1), (4, 128, 1), (5, 0, 700)]
    steps = []
    for i in range(3):
        k, v, table = paged(lens, BS, Hkv, D, seed=10 + i)
        order = spec[i:] + spec[:i]
        meta = [t.cpu().pin_memory() for t in (*portions(order)[:3], table)]
        steps.append((rand(824, Hq * D, dtype=BF, seed=20 + i), k, v, meta))
    q, mid = torch.empty_like(steps[0][0]), torch.empty_like(steps[0][0])
    pools = [torch.empty_like(steps[0][1]) for _ in range(2)]
    held = [torch.empty_like(t, device=q.device) for t in steps[0][3]]
    st = status()

    def step(i, older):
        src, k, v, meta = steps[i]
        for t, m in zip(held, meta):
            t.copy_(m, non_blocking=True)
        out = torch.empty_like(q)
        ops.bias_act(mid, src, None, "identity")
        for pool, t in zip(pools, (k, v)):
            ops.bias_act(pool.view(-1, D), t.view(-1, D), None, "identity")
        ops.bias_act(q, mid, None, "identity")
        ops.attention_prefill_tcgen05(out, q, *pools, held[3], *held[:3], Hq, D ** -0.5, st, meta_older=older)
        return out

    want = []
    for i in range(3):
        want.append(step(i, False))
        torch.cuda.synchronize()
    outs = [(i, step(i, True)) for _ in range(4) for i in range(3)]
    assert int(st.item()) == 0
    assert all(torch.equal(out, want[i]) for i, out in outs)
