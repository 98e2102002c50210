"""The products of the 32-bit path against float64, and that a row's numbers are the same bits whichever kernel and form
serves it: 1 to 8 rows, tiles in clusters, whole tiles, edges of rows, columns and K."""

import pytest
import torch

from test_kernels_gpu import rand

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops():
    from socrates_b200.kernels import ops, require_kernels
    require_kernels()
    return ops


@pytest.mark.parametrize("N,K", [(1, 4), (31, 20), (65, 64), (200, 100), (2560, 256), (96, 1536), (57600, 64), (60000, 36)])
def test_gemm_f32(ops, N, K):
    a, w = rand(70, K, dtype=torch.float32, seed=1), rand(N, K, dtype=torch.float32, seed=2)
    exact = a.double() @ w.double().T
    # 16 chains of K/16 products and 5 additions: each rounds by at most 2^-24 of the sum of magnitudes
    bound = (K / 16 + 6) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    whole = None
    for M in (70, 1, 2, 3, 4, 5, 8, 9, 64, 65):
        out = torch.full((M, N), float("nan"), device=DEV)
        ops.gemm_simt(out, a[:M].contiguous(), w)
        assert bool(((out.double() - exact[:M]).abs() <= bound[:M]).all()), M
        whole = out if whole is None else whole
        assert torch.equal(out, whole[:M]), M


@pytest.mark.parametrize("N,K,rows", [(57600, 520, (65, 9, 64, 1, 8)), (14400, 1036, (256, 9, 64, 130, 1, 5))])
def test_whole_tiles_of_many_pieces(ops, N, K, rows):
    """Products with tiles enough for whole tiles (888 on 148 SMs) whose segments hold two to five pieces each, the last one
    cut: the refills and the joining of segments carry the result there.  14,400 columns by 64 rows and fewer are clusters
    of the same sums."""
    M = rows[0]
    a, w = rand(M, K, dtype=torch.float32, seed=1), rand(N, K, dtype=torch.float32, seed=2)
    exact = a.double() @ w.double().T
    bound = (K / 16 + 6) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)      # as above
    whole = torch.full((M, N), float("nan"), device=DEV)
    ops.gemm_simt(whole, a, w)
    assert bool(((whole.double() - exact).abs() <= bound).all())
    for m in rows[1:]:
        out = torch.full((m, N), float("nan"), device=DEV)
        ops.gemm_simt(out, a[:m].contiguous(), w)
        assert torch.equal(out, whole[:m]), m


@pytest.mark.parametrize("M,N,K", [(1, 2560, 1024), (8, 2560, 1024), (70, 2560, 1024), (64, 57600, 64)])
def test_a_matrix_that_the_kernel_before_writes(ops, M, N, K):
    """w is the result of the kernel right before this one on the stream, which lets its successor start early: nothing of
    w may be read before that kernel has ended (1 and 8 rows, tiles in clusters, whole tiles)."""
    a, x, y = (rand(n, k, dtype=torch.float32, seed=s) for n, k, s in ((M, K, 1), (N, 256, 2), (K, 256, 3)))
    w, out, want = torch.empty(N, K, device=DEV), torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    ops.gemm_simt(w, x, y)
    torch.cuda.synchronize()
    ops.gemm_simt(want, a, w.clone(), w_older=True)
    for _ in range(8):
        w.fill_(float("nan"))
        ops.gemm_simt(w, x, y)
        ops.gemm_simt(out, a, w)
        assert torch.equal(out, want)
