"""The selective scan's kernel for 8, 16, 32 and 64 states against the recurrence in 64 bits, in all its launch forms, and
beside the kernel for any number of states, which serves the same call when its tables do not start on 16 bytes."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops():
    from socrates_b200.kernels import ops, require_kernels
    require_kernels()
    return ops


def misaligned(t):
    out = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view(t.shape)
    return out.copy_(t)


def recurrence(c, dtype, starts, rows):
    """Output and final states in float64, and the same sums with every term's magnitude."""
    N, inner = c["x"].shape
    n = c["A_log"].shape[1]
    d = {k: v.double() for k, v in c.items()}
    dt = torch.nn.functional.softplus(d["dt_raw"] + d["dt_bias"])
    A = -torch.exp(d["A_log"])
    gate = torch.nn.functional.silu(d["z"])
    out, mag = torch.empty(N, inner, device=DEV).double(), torch.empty(N, inner, device=DEV).double()
    last = {}
    for r, row in enumerate(rows):
        S, P = d["state"][row], d["state"][row].abs()
        for t in range(starts[r], starts[r + 1]):
            e = torch.exp(dt[t][:, None] * A)
            add = (dt[t] * d["x"][t])[:, None] * d["bc"][t, :n]
            S, P = e * S + add, e * P + add.abs()
            out[t] = (S @ d["bc"][t, n:] + d["D"] * d["x"][t]) * gate[t]
            mag[t] = (P @ d["bc"][t, n:].abs() + (d["D"] * d["x"][t]).abs()) * gate[t].abs()
        last[row] = (S, P)
    return out, mag, last


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("states,inner", [(8, 70), (16, 33), (16, 128), (32, 17), (64, 9)])
@pytest.mark.parametrize("lengths", [(1,), (1, 1, 1), (15, 2), (16, 17), (33,), (129, 260)])
def test_quads(ops, dtype, states, inner, lengths):
    g = torch.Generator(device=DEV).manual_seed(sum(lengths) * states + inner)

    def randn(*shape):
        return torch.randn(*shape, device=DEV, generator=g)

    N, R = sum(lengths), len(lengths)
    c = {"x": randn(N, inner).to(dtype), "z": randn(N, 2 * inner).to(dtype)[:, inner:], "dt_raw": randn(N, inner),
         "dt_bias": randn(inner) - 2, "bc": randn(N, 2 * states).to(dtype), "A_log": randn(inner, states).sigmoid() * 2.5,
         "D": randn(inner), "state": randn(R + 1, inner, states)}
    starts = [sum(lengths[:i]) for i in range(R + 1)]
    rows = list(range(R, 0, -1))
    want, mag, last = recurrence(c, dtype, starts, rows)
    seq = [torch.tensor(v, dtype=torch.int32, device=DEV) for v in (starts, rows)]
    scratch = torch.full((ops.selective_scan_scratch_size(N, R, inner, states),), float("nan"), device=DEV)
    # a token rounds a state four times (dt A, its exponential, the new term, the multiply-add), the hardware exponential by
    # 2^-22 more and an exponent of up to 40 by 40 roundings; the softplus and the gate a few times each.  Decays fade what
    # the tokens before left, so the magnitudes' own recurrence carries it.
    unit = 2.0 ** -24 * (16 + 4 * 40)
    outs = []
    for aligned in (True, False):
        for lent in (None, scratch):
            state, out = c["state"].clone(), torch.full((N, inner), float("nan"), device=DEV, dtype=dtype)
            A_log = c["A_log"] if aligned else misaligned(c["A_log"])
            ops.selective_scan(out, c["x"], c["z"], c["dt_raw"], c["dt_bias"], c["bc"], A_log, c["D"], state, *seq, scratch=lent)
            bound = unit * mag + (2.0 ** -8 * want.abs() if dtype == torch.bfloat16 else 0)
            assert bool(((out.double() - want).abs() <= bound).all())
            for row, (S, P) in last.items():
                assert bool(((state[row].double() - S).abs() <= unit * P).all())
            assert torch.equal(state[0], c["state"][0])           # a row that is not in the step
            outs.append(out)


def test_portions_are_the_same_bits(ops):
    """Token by token and in one launch, with no scratch: the same walk."""
    g = torch.Generator(device=DEV).manual_seed(3)
    N, inner, n = 37, 40, 16
    x, z, bc = (torch.randn(N, k, device=DEV, generator=g) for k in (inner, inner, 2 * n))
    dt, A, D = (torch.randn(*s, device=DEV, generator=g) for s in ((N, inner), (inner, n), (inner,)))
    bias = torch.zeros(inner, device=DEV)
    row = torch.zeros(1, dtype=torch.int32, device=DEV)
    whole, state = torch.empty(N, inner, device=DEV), torch.zeros(1, inner, n, device=DEV)
    ops.selective_scan(whole, x, z, dt, bias, bc, A, D, state, torch.tensor([0, N], dtype=torch.int32, device=DEV), row)
    parts, cut = torch.empty_like(whole), torch.zeros_like(state)
    for a, b in ((0, 1), (1, 18), (18, 34), (34, N)):
        ops.selective_scan(parts[a:b], x[a:b], z[a:b], dt[a:b], bias, bc[a:b], A, D, cut,
                           torch.tensor([0, b - a], dtype=torch.int32, device=DEV), row)
    assert torch.equal(whole, parts) and torch.equal(state, cut)
