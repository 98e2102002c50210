"""The norm and activation kernels that hold a row in registers: against float64 at every width class, odd widths in whole
float4 columns, and beside the kernels that serve rows which do not start on 16 bytes."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, EPS = "cuda", 1e-5
# a float32 row of sums of S + 4 terms, its mean square and root, two products; then the result's own rounding
F32 = 2.0 ** -24 * 24


@pytest.fixture(scope="module")
def ops():
    from socrates_b200.kernels import ops, require_kernels
    require_kernels()
    return ops


def unit(x, eps=EPS):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def near(got, want, dtype):
    scale = want.abs() + want.abs().mean(-1, keepdim=True)
    return bool(((got.double() - want).abs() <= (F32 + (2.0 ** -8 if dtype == torch.bfloat16 else 0)) * scale).all())


@pytest.mark.parametrize("d", [4, 516, 1024, 2048, 2560, 3072, 4096, 5120, 6000, 8192, 8196])
@pytest.mark.parametrize("M,S", [(65, 2), (300, 0), (520, 1), (520, 3)])
def test_add_rmsnorm(ops, d, M, S):
    g = torch.Generator(device=DEV).manual_seed(d + M + S)
    res = torch.randn(M, d, device=DEV, generator=g)
    delta = torch.randn(S, M, d, device=DEV, generator=g) if S else None
    gain = torch.randn(d, device=DEV, generator=g)
    want = res.double() + (delta.double().sum(0) if S else 0)
    r, out = res.clone(), torch.full((M, d), float("nan"), device=DEV, dtype=torch.bfloat16)
    ops.add_rmsnorm(r, delta, gain, out, EPS)
    assert near(r, want, torch.float32) and near(out, unit(want) * gain.double(), torch.bfloat16)
    index = torch.arange(M - 1, -1, -1, dtype=torch.int32, device=DEV)
    again, picked = res.clone(), torch.empty_like(out)
    ops.add_rmsnorm(again, delta, gain, picked, EPS, row_index=index)
    assert torch.equal(again, res) and torch.equal(picked.flip(0), out)


@pytest.mark.parametrize("d", [8, 1024, 2052, 4096, 8192])
@pytest.mark.parametrize("form", ["plain", "normed", "bias", "tanh", "norm_residual", "stream", "fold"])
def test_fold_rmsnorm(ops, d, form):
    g = torch.Generator(device=DEV).manual_seed(d)
    M, S = 70, 0 if form == "bias" else 3

    def randn(*shape):
        return torch.randn(*shape, device=DEV, generator=g)

    res, gain, delta = randn(M, d), randn(d), randn(S, M, d) if S else None
    kw = {"normed": dict(branch_gain=randn(d), branch_eps=EPS, add_rows=randn(M, d), add_vec=randn(d)),
          "bias": dict(branch_bias=randn(d), res_scale=0.5), "tanh": dict(tanh_alpha=randn(1), tanh_bias=randn(d)),
          "norm_residual": dict(norm_residual=True, res_scale=2.0)}.get(form, {})
    b = (delta.double().sum(0) if S else 0) + (kw["branch_bias"].double() if "branch_bias" in kw else 0)
    if "branch_gain" in kw:
        b = unit(b) * kw["branch_gain"].double()
    v = res.double() * kw.get("res_scale", 1.0) + b + (kw["add_rows"].double() + kw["add_vec"].double() if "add_rows" in kw else 0)
    out_gain = None if form == "stream" else gain
    y = v if out_gain is None else unit(v) * gain.double()
    if form == "tanh":
        y = torch.tanh(kw["tanh_alpha"].double() * v) * gain.double() + kw["tanh_bias"].double()
    for shift in (0, 1):                                    # a residual off 16 bytes: the other kernel
        r = torch.empty(M * d + shift, device=DEV)[shift:].view(M, d).copy_(res)
        out = None if form == "fold" else torch.full((M, d), float("nan"), device=DEV, dtype=torch.bfloat16)
        ops.fold_rmsnorm(r, delta, None if form == "fold" else out_gain, out, EPS, **kw)
        assert near(r, y if form == "norm_residual" else v, torch.float32)
        assert out is None or near(out, y, torch.bfloat16)


@pytest.mark.parametrize("d", [8, 1024, 2052, 2560, 4096, 5120, 8192])
@pytest.mark.parametrize("S0,S1", [(1, 3), (2, 2), (9, 13)])
def test_normed_mean_rows_are_the_same_bits_in_any_batch(ops, d, S0, S1):
    g = torch.Generator(device=DEV).manual_seed(d + S0)
    x0, x1 = torch.randn(S0, 70, d, device=DEV, generator=g), torch.randn(S1, 70, d, device=DEV, generator=g)
    g0, g1 = torch.randn(d, device=DEV, generator=g), torch.randn(d, device=DEV, generator=g)
    whole, few = torch.empty(70, d, device=DEV), torch.empty(3, d, device=DEV)
    ops.normed_mean(whole, x0, g0, x1, g1, EPS, 0.5)
    ops.normed_mean(few, x0[:, :3].contiguous(), g0, x1[:, :3].contiguous(), g1, EPS, 0.5)
    assert torch.equal(few, whole[:3])
    a, b = unit(x0.double().sum(0)) * g0.double(), unit(x1.double().sum(0)) * g1.double()
    scale = (a.abs() + b.abs()) + (a.abs() + b.abs()).mean(-1, keepdim=True)
    assert bool(((whole.double() - 0.5 * (a + b)).abs() <= F32 * scale).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("act", ["identity", "relu_squared", "gelu_tanh", "silu", "tanh"])
@pytest.mark.parametrize("S", [0, 3])
def test_bias_act(ops, dtype, act, S):
    g = torch.Generator(device=DEV).manual_seed(1)
    N, F = 3101, 8 * 53                                     # more than the values from which the rows go by 16 bytes
    x = torch.randn(S, N, F, device=DEV, generator=g) if S else torch.randn(N, F, device=DEV, generator=g).to(dtype)
    bias = torch.randn(F, device=DEV, generator=g)
    outs = []
    for aligned in (True, False):                           # off 16 bytes: a value at a time
        out = torch.full((N * F + 8,), float("nan"), device=DEV, dtype=dtype)[0 if aligned else 1:][:N * F].view(N, F)
        ops.bias_act(out, x, bias, act)
        outs.append(out.clone())
    assert torch.equal(*outs) and bool(torch.isfinite(outs[0]).all())


@pytest.mark.parametrize("d", [4, 516, 1024, 2048, 2560, 3076, 4096, 5120, 8192])
@pytest.mark.parametrize("M,S", [(65, 2), (300, 0), (512, 1), (513, 2), (900, 3)])
def test_add_rmsnorm_rows_have_the_other_kernels_bits(ops, d, M, S):
    """float32 results come from the kernel with a row in shared memory: the same numbers, rounded once more."""
    g = torch.Generator(device=DEV).manual_seed(d * M + S)
    res, gain = torch.randn(M, d, device=DEV, generator=g), torch.randn(d, device=DEV, generator=g)
    delta = torch.randn(S, M, d, device=DEV, generator=g) if S else None
    sides = []
    for dtype in (torch.bfloat16, torch.float32):
        r, out = res.clone(), torch.full((M, d), float("nan"), device=DEV, dtype=dtype)
        ops.add_rmsnorm(r, delta, gain, out, EPS)
        sides.append((r, out.to(torch.bfloat16)))
    assert torch.equal(sides[0][0], sides[1][0]) and torch.equal(sides[0][1], sides[1][1])


@pytest.mark.parametrize("d", [8, 1024, 2052, 2560, 4096, 8192])
@pytest.mark.parametrize("M", [65, 512, 513])
@pytest.mark.parametrize("form", ["plain", "normed", "norm_residual"])
def test_fold_rmsnorm_rows_have_the_other_kernels_bits(ops, d, M, form):
    g = torch.Generator(device=DEV).manual_seed(d + M)
    res, delta = torch.randn(M, d, device=DEV, generator=g), torch.randn(3, M, d, device=DEV, generator=g)
    gain, inner = torch.randn(d, device=DEV, generator=g), torch.randn(d, device=DEV, generator=g)
    kw = {"normed": dict(branch_gain=inner, branch_eps=EPS), "norm_residual": dict(norm_residual=True)}.get(form, {})
    sides = []
    for dtype in (torch.bfloat16, torch.float32):
        r, out = res.clone(), torch.full((M, d), float("nan"), device=DEV, dtype=dtype)
        ops.fold_rmsnorm(r, delta, gain, out, EPS, **kw)
        sides.append((r, out.to(torch.bfloat16)))
    assert torch.equal(sides[0][0], sides[1][0]) and torch.equal(sides[0][1], sides[1][1])


ACTIVATIONS = {"identity": lambda x: x, "relu_squared": lambda x: x.clamp(min=0) ** 2, "silu": torch.nn.functional.silu,
               "gelu_tanh": lambda x: torch.nn.functional.gelu(x, approximate="tanh"), "tanh": torch.tanh}


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("act", list(ACTIVATIONS))
@pytest.mark.parametrize("S,bias", [(0, True), (3, True), (1, False)])
@pytest.mark.parametrize("N,F", [(3101, 424), (30, 424), (3101, 427)])
def test_bias_act_against_64_bits(ops, dtype, act, S, bias, N, F):
    """By 16 bytes (many values in rows of whole pieces) and a value at a time."""
    g = torch.Generator(device=DEV).manual_seed(N + F)
    x = torch.randn(S, N, F, device=DEV, generator=g) if S else torch.randn(N, F, device=DEV, generator=g).to(dtype)
    b = torch.randn(F, device=DEV, generator=g) if bias else None
    out = torch.full((N, F), float("nan"), device=DEV, dtype=dtype)
    ops.bias_act(out, x, b, act)
    terms = (x.double().abs().sum(0) if S else x.double().abs()) + (b.double().abs() if bias else 0)
    z = (x.double().sum(0) if S else x.double()) + (b.double() if bias else 0)
    want = ACTIVATIONS[act](z)
    # S + 1 float32 additions, an activation whose slope is at most 2 |z| + 1.2 and which itself takes some ten roundings of
    # numbers up to 1 + |z| + z^2, then the result's own rounding
    bound = 2.0 ** -24 * ((S + 1) * terms * (2 * z.abs() + 1.2) + 16 * (1 + z.abs() + z * z)) + \
        (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23) * want.abs()
    assert bool(((out.double() - want).abs() <= bound).all())
