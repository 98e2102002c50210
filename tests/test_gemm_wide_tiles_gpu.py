"""Products of many rows in tiles wider than one tensor-core product: every width against float64 at sizes whose last tile is
nearly empty, ends inside either half, or has a second half outside the matrix; plain and gated; and the sizes at which the
choice by shape takes them."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF = torch.bfloat16


def run(out, a, w, **kw):
    from socrates_b200.kernels import ops, require_kernels
    require_kernels()
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    for _ in range(2):
        out.fill_(float("nan"))
        ops.gemm_tcgen05(out, a, w, status, **kw)
    assert int(status) == 0
    return out


@pytest.mark.parametrize("width", [0, 288, 352, 416])
@pytest.mark.parametrize("M,N,K", [(129, 584, 72), (300, 300, 64), (1024, 840, 200), (257, 1000, 2048), (2048, 2560, 320),
                                   (187, 19456, 128), (1024, 6144, 64), (1100, 6144, 136)])
def test_wide_tiles(width, M, N, K):
    g = torch.Generator(device=DEV).manual_seed(0)
    a = torch.randn(M, K, device=DEV, generator=g).to(BF)
    w = (torch.randn(N, K, device=DEV, generator=g) * K ** -0.5).to(BF)
    want = a.double() @ w.double().T
    # float32 sums: a sum (below 8 here) is cut off at its 24 bits for every 16 of K
    full = run(torch.empty(M, N, device=DEV), a, w, variant=width)
    assert float((full - want).abs().max()) < 8 * (K // 16 + 2) * 2.0 ** -22
    half = run(torch.empty(M, N, device=DEV, dtype=BF), a, w, variant=width)
    assert torch.equal(half, full.to(BF))
    gate, up = full.double()[:, 0::2], full.double()[:, 1::2]
    gated = run(torch.empty(M, N // 2, device=DEV, dtype=BF), a, w, variant=width, epilogue=1)
    assert torch.allclose(gated.double(), up * torch.nn.functional.silu(gate), rtol=2.0 ** -8, atol=1e-5)
