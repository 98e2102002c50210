"""Products of many rows in tiles wider than one tensor-core product: every width against float64 at sizes whose last tile is
nearly empty, ends inside either half, or has a second half outside the matrix; plain and gated; and the sizes from which, and
up to which, the choice by shape takes them."""

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


@pytest.mark.parametrize("N,widths", [
    # seven row tiles keep their width; the wide tiles end where they are more than one wave of 148
    (6144, {896: 160, 897: 352, 1024: 352, 1025: 416, 1152: 416, 1153: 256}),
    (19456, {187: 160, 384: 256, 2048: 256}),
    (2560, {512: 128, 897: 160, 1152: 160, 1153: 256, 1792: 256, 1793: 288, 2048: 288, 2049: 352, 2561: 416, 2689: 256}),
    (4096, {1152: 256, 1153: 352, 1408: 352, 1409: 352, 1537: 416, 1793: 256}),
    (5120, {896: 256, 897: 288, 1024: 288, 1025: 352, 1152: 352, 1153: 416, 1409: 256})])
def test_which_products_take_wide_tiles(N, widths):
    from socrates_b200.kernels import ops, require_kernels
    require_kernels()
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert {M: ops.gemm_tcgen05_tile_width(M, N) for M in widths} == widths


@pytest.mark.parametrize("M,N,K,other", [(1024, 6144, 2560, 256), (1100, 6144, 1000, 256), (1600, 4096, 512, 256)])
def test_wide_tiles_have_the_bits_of_256_columns(M, N, K, other):
    """A tile's sums go into one accumulator, as those of 256 columns do (128 and 160 columns: two, for halves of each K block)."""
    g = torch.Generator(device=DEV).manual_seed(1)
    a = torch.randn(M, K, device=DEV, generator=g).to(BF)
    w = torch.randn(N, K, device=DEV, generator=g).to(BF)
    wide, same = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    assert torch.equal(run(wide, a, w), run(same, a, w, variant=other))
