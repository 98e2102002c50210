"""The convolution's kernel for many values: the same bits as the kernel for few, which serves smaller steps and any call that has
no whole 16-byte pieces."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops():
    from socrates_b200.kernels import ops, require_kernels
    require_kernels()
    return ops


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("K", [2, 3, 4])
@pytest.mark.parametrize("bias,silu", [(False, True), (True, False)])
def test_runs(ops, dtype, K, bias, silu):
    heads, dim, page = 2, 16, 16
    C, dense = 40 + heads * dim, 40
    g = torch.Generator(device=DEV).manual_seed(K)
    lengths, firsts, rows = (70, 1, 9, 1, 2, 16), (0, 5, 2, 0, 1, 100), (3, 0, 5, 1, 2, 4)
    N = sum(lengths)
    x = torch.randn(N, C + 8, device=DEV, generator=g).to(dtype)
    taps, tail = torch.randn(C, K, device=DEV, generator=g), torch.randn(6, K - 1, C, device=DEV, generator=g)
    b1, b2 = (torch.randn(C, device=DEV, generator=g) if bias else None for _ in range(2))
    token_rows = torch.tensor([r for r, n in zip(rows, lengths) for _ in range(n)], dtype=torch.int32, device=DEV)
    positions = torch.tensor([f + i for f, n in zip(firsts, lengths) for i in range(n)], dtype=torch.int32, device=DEV)
    table = torch.arange(1, 6 * 8 + 1, dtype=torch.int32, device=DEV).view(6, 8)

    def run(x, taps):
        out = torch.full((N, dense), float("nan"), device=DEV, dtype=dtype)
        pool = torch.full((49, heads, page, dim), 7.0, device=DEV, dtype=dtype)
        ops.short_conv(x, b1, taps, b2, silu, tail, token_rows, positions, [(0, dense, out), (dense, C, pool)], table)
        return out, pool

    runs = run(x, taps)
    shifted = torch.empty(taps.numel() + 1, device=DEV)[1:].view(taps.shape).copy_(taps)      # not on 16 bytes: the other kernel
    for a, b in zip(runs, run(x, shifted)):
        assert torch.equal(a, b)
    # and the definition, in 64 bits, for the dense channels
    u = x[:, :dense].double() + (b1[:dense].double() if bias else 0.0)
    for n in (0, 1, K - 1, 69, 70, 71, 72, 79, 80, 81, 82, 83, N - 1):
        acc, mag, p = 0.0, 0.0, int(positions[n])
        for j in range(K):
            back = K - 1 - j
            if p - back < 0:
                continue
            start = int(positions[n]) - firsts[[i for i in range(6) if sum(lengths[:i]) <= n][-1]]
            v = u[n - back] if back <= start else tail[int(token_rows[n]), K - 1 - back + start, :dense].double()
            acc, mag = acc + taps[:dense, j].double() * v, mag + (taps[:dense, j].double() * v).abs()
        if bias:
            acc = acc + b2[:dense].double()
        if silu:
            acc = torch.nn.functional.silu(acc)
        # K + 2 float32 roundings, the gate's few, and the result's own
        bound = (K + 12) * 2.0 ** -24 * (mag + acc.abs() + 10) + (2.0 ** -8 * acc.abs() if dtype == torch.bfloat16 else 0)
        assert bool(((runs[0][n].double() - acc).abs() <= bound).all()), n


@pytest.mark.parametrize("N,C,K,requests,dtype,runs", [
    (64, 3072, 3, 64, torch.bfloat16, False), (64, 4096, 4, 64, torch.bfloat16, False), (256, 4096, 4, 256, torch.bfloat16, False),
    (319, 4096, 4, 3, torch.bfloat16, False), (320, 4096, 4, 320, torch.bfloat16, True), (187, 4096, 4, 1, torch.bfloat16, False),
    (255, 4096, 4, 1, torch.bfloat16, False), (256, 4096, 4, 2, torch.bfloat16, True), (1500, 3072, 3, 1, torch.bfloat16, True),
    (64, 4096, 4, 64, torch.float32, False), (128, 4096, 4, 1, torch.float32, True), (223, 4096, 4, 223, torch.float32, False),
    (224, 4096, 4, 224, torch.float32, True), (191, 8192, 2, 191, torch.bfloat16, False), (200, 8192, 2, 200, torch.bfloat16, True)])
def test_which_steps_go_by_runs(ops, N, C, K, requests, dtype, runs):
    assert ops.short_conv_pays_runs(N, C, K, requests, dtype) == runs


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("K", [2, 3, 4])
@pytest.mark.parametrize("lengths", [(1,) * 420, (331,), (300, 1, 9, 1, 2, 100)])
def test_wide_rows_by_runs(ops, dtype, K, lengths):
    """Enough values for runs: the same bits as a thread a value (taps off 16 bytes), dense and paged, and with a step that
    does not say how many requests it is of."""
    heads, dim, page, N, R = 8, 64, 16, sum(lengths), len(lengths)
    dense = 4608
    C = dense + heads * dim
    g = torch.Generator(device=DEV).manual_seed(K)
    assert ops.short_conv_pays_runs(N, C, K, R, dtype)
    x = torch.randn(N, C + 8, device=DEV, generator=g).to(dtype)
    taps, tail = torch.randn(C, K, device=DEV, generator=g), torch.randn(R, K - 1, C, device=DEV, generator=g)
    token_rows = torch.tensor([r for r, n in enumerate(lengths) for _ in range(n)], dtype=torch.int32, device=DEV)
    positions = torch.tensor([r % 5 + i for r, n in enumerate(lengths) for i in range(n)], dtype=torch.int32, device=DEV)
    pages = -(-(max(lengths) + 5) // page)
    table = torch.arange(1, R * pages + 1, dtype=torch.int32, device=DEV).view(R, pages)
    outs = []
    for shift, requests in ((0, R), (0, None), (1, R)):
        t = torch.empty(taps.numel() + shift, device=DEV)[shift:].view(taps.shape).copy_(taps)
        out = torch.full((N, dense), float("nan"), device=DEV, dtype=dtype)
        pool = torch.full((R * pages + 1, heads, page, dim), 7.0, device=DEV, dtype=dtype)
        ops.short_conv(x, None, t, None, True, tail, token_rows, positions, [(0, dense, out), (dense, C, pool)], table,
                       requests=requests)
        outs.append((out, pool))
    for out, pool in outs[1:]:
        assert torch.equal(out, outs[0][0]) and torch.equal(pool, outs[0][1])
    assert bool(torch.isfinite(outs[0][0]).all())
