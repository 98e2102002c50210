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
