"""The register-tile kernels of retention (three launches) against the recurrence in 64 bits: every head size they serve,
portions that end inside and at the edge of a chunk, several requests, rotation or none, and beside the kernels for other
heads, which serve the same call when its rows do not start on 16 bytes."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops():
    from socrates_b200.kernels import ops, require_kernels
    require_kernels()
    return ops


def recurrence(x, H, dk, dv, starts, rows, firsts, state, decay, freq, scale, eps):
    N = x.shape[0]
    q, k, v, g = (t.double().reshape(N, H, -1) for t in x.split([H * dk, H * dk, H * dv, H * dv], dim=1))
    out = torch.empty(N, H, dv, device=DEV, dtype=torch.float64)
    last = {}
    for r, row in enumerate(rows):
        a, b = starts[r], starts[r + 1]
        qr, kr = q[a:b], k[a:b]
        if freq is not None:
            angle = (firsts[r] + torch.arange(b - a, device=DEV).double())[:, None] * freq
            c, s = angle.cos()[:, None], angle.sin()[:, None]
            qr, kr = (torch.cat([t[..., :dk // 2] * c - t[..., dk // 2:] * s, t[..., dk // 2:] * c + t[..., :dk // 2] * s], -1)
                      for t in (qr, kr))
        S = state[row].double()
        for t in range(b - a):
            S = decay.double()[:, None, None] * S + scale * kr[t][:, :, None] * v[a + t][:, None, :]
            o = torch.einsum("hij,hi->hj", S, qr[t])
            out[a + t] = o / torch.sqrt((o * o).mean(-1, keepdim=True) + eps) * torch.nn.functional.silu(g[a + t])
        last[row] = S
    return out.reshape(N, H * dv), last


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("dk,dv,turns", [(64, 128, True), (16, 64, True), (48, 128, True), (128, 256, True), (96, 64, True),
                                         (32, 256, False), (64, 64, False)])
@pytest.mark.parametrize("lengths", [(129,), (192, 1), (64, 65, 70)])
def test_tiles(ops, dtype, dk, dv, turns, lengths):
    H, N, R = 3, sum(lengths), len(lengths)
    g = torch.Generator(device=DEV).manual_seed(N + dk + dv)
    wide = torch.randn(N, 2 * H * (dk + dv), device=DEV, generator=g).to(dtype)
    state = torch.randn(R + 1, H, dk, dv, device=DEV, generator=g)
    decay = torch.tensor([0.97, 0.995, 0.9995], device=DEV)
    freq = 1.0 / 1e4 ** (torch.arange(0, dk, 2, device=DEV).double() / dk)
    high = freq.float()
    low = (freq - high.double()).float()
    starts, rows, firsts = [sum(lengths[:i]) for i in range(R + 1)], list(range(R, 0, -1)), [1000 * r for r in range(R)]
    want, last = recurrence(wide, H, dk, dv, starts, rows, firsts, state, decay, freq if turns else None, dk ** -0.5, 1e-5)
    seq = [torch.tensor(t, dtype=torch.int32, device=DEV) for t in (starts, rows, firsts)]
    scratch = torch.full((ops.retention_scratch_size(N, R, H, dk, dv),), float("nan"), device=DEV)
    errors = []
    for shift in (0, 1):                                # by one element: rows no longer on 16 bytes, the other kernels
        buf = torch.empty(N * wide.shape[1] + shift, dtype=dtype, device=DEV)[shift:].view(wide.shape)
        buf.copy_(wide)
        st, out = state.clone(), torch.full((N, H * dv), float("nan"), device=DEV, dtype=dtype)
        ops.retention(out, buf, (0, H * dk, 2 * H * dk, 2 * H * dk + H * dv), st, decay, high, dk if turns else 0, *seq, 1e-5,
                      dk ** -0.5, chunked=True, inv_freq_lo=low, scratch=scratch)
        errors.append([float((out.double() - want).norm() / want.norm())] +
                      [float((st[row].double() - S).norm() / S.norm()) for row, S in last.items()])
        assert torch.equal(st[0], state[0])             # a row that is not in the step
    # float32 sums of up to dk + 64 products and up to four chunks, squares and roots: some tens of roundings, which add up like
    # their root; the result's own rounding in bfloat16 is 2^-9 at most
    for tiles, other in zip(*errors):
        assert tiles <= 16 * 2.0 ** -24 + (2.0 ** -9 if dtype == torch.bfloat16 else 0), errors
        assert tiles <= 1.5 * other + 2.0 ** -23, errors


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("dk,dv", [(64, 128), (32, 256), (96, 64)])
@pytest.mark.parametrize("at", [1, 7, 8, 37, 63, 64, 100])
def test_a_value_that_is_not_finite_reaches_no_earlier_token(ops, dtype, dk, dv, at):
    """An infinity among token `at`'s values: the tokens before it have the bits that they have without it, in the tile kernels
    and (rows off 16 bytes) in the kernels for other heads, with chunks as launches and with one block a request."""
    H, N = 3, 150
    g = torch.Generator(device=DEV).manual_seed(at)
    wide = torch.randn(N, 2 * H * (dk + dv), device=DEV, generator=g).to(dtype)
    decay = torch.tensor([0.97, 0.995, 0.9995], device=DEV)
    freq = 1.0 / 1e4 ** (torch.arange(0, dk, 2, device=DEV).double() / dk)
    seq = [torch.tensor(t, dtype=torch.int32, device=DEV) for t in ([0, N], [0], [0])]
    lent = torch.empty(ops.retention_scratch_size(N, 1, H, dk, dv), device=DEV)
    for shift, scratch in ((0, lent), (1, lent), (1, None)):
        outs = []
        for value in (None, float("inf")):
            buf = torch.empty(N * wide.shape[1] + shift, dtype=dtype, device=DEV)[shift:].view(wide.shape)
            buf.copy_(wide)
            if value is not None:
                buf[at, 2 * H * dk + dv + 5] = value            # head 1
            out = torch.full((N, H * dv), float("nan"), device=DEV, dtype=dtype)
            ops.retention(out, buf, (0, H * dk, 2 * H * dk, 2 * H * dk + H * dv), torch.zeros(1, H, dk, dv, device=DEV), decay,
                          freq.float(), dk, *seq, 1e-5, dk ** -0.5, chunked=True, inv_freq_lo=(freq - freq.float().double()).float(),
                          scratch=scratch)
            outs.append(out)
        assert torch.equal(outs[0][:at], outs[1][:at]), (shift, scratch is not None)
        assert not bool(torch.isfinite(outs[1][at, dv:2 * dv]).all())


@pytest.mark.parametrize("lent", [False, True])
def test_an_element_type_that_no_kernel_has_is_refused(ops, monkeypatch, lent):
    H, dk, dv, N = 2, 64, 128, 300
    x = torch.randn(N, 2 * H * (dk + dv), device=DEV).to(torch.bfloat16)
    seq = [torch.tensor(t, dtype=torch.int32, device=DEV) for t in ([0, N], [0], [0])]
    scratch = torch.empty(ops.retention_scratch_size(N, 1, H, dk, dv), device=DEV) if lent else None
    out = torch.full((N, H * dv), 7.0, device=DEV, dtype=torch.bfloat16)
    monkeypatch.setattr(ops, "_code", lambda dtype: 2)
    with pytest.raises(ops.KernelError, match="dtype 2"):
        ops.retention(out, x, (0, H * dk, 2 * H * dk, 2 * H * dk + H * dv), torch.zeros(1, H, dk, dv, device=DEV),
                      torch.full((H,), 0.9, device=DEV), torch.ones(dk // 2, device=DEV), 0, *seq, 1e-5, 1.0, chunked=True,
                      scratch=scratch)
    assert bool((out == 7.0).all())
