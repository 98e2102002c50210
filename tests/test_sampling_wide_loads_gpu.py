"""Sampling of rows that are read 16 bytes at a time against the same numbers one float off a 16-byte boundary, which are
read a value at a time: the same tokens, whatever the slices' ends, for the largest value and for draws."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("V", [4, 2044, 2052, 8188, 8192, 8196, 16388, 24580, 151936, 262148, 300004])
@pytest.mark.parametrize("temperature", [0.0, 0.7])
def test_wide_loads_pick_what_single_loads_pick(V, temperature):
    from socrates_b200.kernels import ops, require_kernels
    require_kernels()
    M = 6
    g = torch.Generator().manual_seed(V)
    x = torch.randn(M, V, generator=g)
    x[1] = 0.5                                      # ties: the lowest index
    x[2, V - 1] = 30.0
    x[3, V // 2] = x[3, V // 3] = 30.0
    x[4] = -float("inf")
    x[5, ::2] = float("nan")
    wide = x.to(DEV)
    store = torch.empty(M * V + 1, device=DEV)
    narrow = store[1:].view(M, V)
    narrow.copy_(wide)
    t = torch.full((M,), temperature, device=DEV)
    seeds = torch.arange(M, dtype=torch.int32, device=DEV)
    got = []
    for logits in (wide, narrow):
        out = torch.empty(M, dtype=torch.int32, device=DEV)
        ops.sample(out, logits, t, seeds, seeds + 5)
        got.append(out.tolist())
    assert got[0] == got[1]
    if temperature == 0.0:
        assert got[0][:5] == [int(x[0].argmax()), 0, V - 1, V // 3, 0]
