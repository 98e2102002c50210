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
