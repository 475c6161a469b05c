"""Gates and convolutions whose results are fp32.  A gate's sigmoid is the library's exponential (2 units in the last place by CUDA's stated bound), one addition and a
correctly rounded division, down to the numbers below 2^-126: 4 units of 2^-23, and one step of 2^-149, which a sigmoid below 2^-126 is rounded to, times the number that
multiplies it.  The convolutions' silu has a reciprocal and two Newton steps in the division's place; its bound is the same."""
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, F64 = "cuda:0", torch.float64


@pytest.fixture(scope="module")
def ops():
    return importlib.import_module("nano-vllm-candle_b200.ops")


def numbers(n):
    return torch.cat([torch.linspace(-88.5, -87.4, n // 4), torch.linspace(-87.0, 87.0, n - n // 4)]).to(DEV)


def close(got, z, silu):
    want = torch.sigmoid(z.to(F64)) * (z.to(F64) if silu else 1.0)
    assert float(((got.to(F64) - want).abs() - 4 * 2.0 ** -23 * want.abs()).max()) <= 2.0 ** -149 * (90.0 if silu else 1.0)


@pytest.mark.parametrize("act", ["silu", "sigmoid"])
@pytest.mark.parametrize("groups,width", [(2, 128), (3, 64), (1, 20)])
def test_gates(ctx, ops, act, groups, width):
    N = 40
    z = numbers(N * groups * width).view(N, -1)
    got = ops.head_gate_w(ctx, torch.ones_like(z), z, None, groups, width, False, 1e-5, act, 1.0)
    close(got, z, act == "silu")


def test_convolutions_of_many_rows(ctx, ops):
    """from 512 rows on a tile of rows per warp"""
    H, G, dim, vdim, taps, N = 2, 1, 64, 64, 2, 600
    C = 2 * G * dim + H * vdim
    x = torch.zeros(N, C + 2 * H, device=DEV)
    x[:, 2 * G * dim:C] = numbers(N * H * vdim).view(N, -1)
    w = torch.zeros(taps, C, device=DEV)
    w[-1] = 1.0
    zero = lambda *s: torch.zeros(*s, device=DEV)  # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    v = ops.delta_rule(ctx, x, (0, G * dim, 2 * G * dim, C, C + H), H, G, dim, vdim, taps, w, zero(1, taps - 1, C), zero(1, H, dim, vdim), i32([0]), i32([0, N]),
                       i32(list(range(N))), zero(H), zero(H), max_qlen=N)[3]
    close(v, x[:, 2 * G * dim:C], True)


def far(n):
    return torch.cat([torch.linspace(-110.0, -60.0, n - 128), torch.linspace(-64.0001, -63.9999, 110), torch.tensor([0.0, -0.0, 1e-38, -1e-38, 1e-45, -1e-45, 88.8, 1e4, 3e38, -200.0, -1e4, -3e38,
                                                                                                                  float("inf"), -float("inf"), float("nan"), 1.0, -1.0, -32.0])]).to(DEV)


def same(got, z):
    """4 units of 2^-23 and one step of 2^-149 times |z|, which the exponential is rounded to; infinities, NaN and signs of zeros as x / (1 + exp(-x)) has them, NaN at -inf"""
    want = z.to(F64) / (1 + torch.exp(-z.to(F64)))
    odd = ~torch.isfinite(want)
    assert torch.equal(got[odd].isnan(), want[odd].isnan()) and torch.equal(got[odd & ~want.isnan()], z[odd & ~want.isnan()])
    assert torch.equal(torch.signbit(got[~odd]), torch.signbit(z[~odd]))
    assert float(((got.to(F64) - want).abs() - 4 * 2.0 ** -23 * want.abs() - 2.0 ** -149 * z.to(F64).abs())[~odd].max()) <= 2.0 ** -149


@pytest.mark.parametrize("N,vdim", [(600, 64), (300, 64), (300, 63)])      # a tile of rows per warp, a row per warp by fours, channel by channel
def test_delta_convolutions_far_from_zero(ctx, ops, N, vdim):
    H, G, dim, taps = 2, 1, 64, 2
    C = 2 * G * dim + H * vdim
    ld = C + 2 * H
    x = torch.zeros(N, ld, device=DEV)
    x[:, 2 * G * dim:C] = far(N * H * vdim).view(N, -1)
    w = torch.zeros(taps, C, device=DEV)
    w[-1] = 1.0
    x[:, 2 * G * dim:C][~x[:, 2 * G * dim:C].isfinite()] = 0       # a tap of weight 0 would carry them into the next row
    zero = lambda *s: torch.zeros(*s, device=DEV)  # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    v = ops.delta_rule(ctx, x, (0, G * dim, 2 * G * dim, C, C + H), H, G, dim, vdim, taps, w, zero(1, taps - 1, C), zero(1, H, dim, vdim), i32([0]), i32([0, N]),
                       i32(list(range(N))), zero(H), zero(H), max_qlen=N)[3]
    z = x[:, 2 * G * dim:C] + 0.0       # the sum of the taps starts at 0: -0 comes out as 0
    same(v, z)


@pytest.mark.parametrize("N,vdim", [(2048, 64), (300, 64), (300, 63)])
def test_state_space_convolutions_far_from_zero(ctx, ops, N, vdim):
    H, G, state, taps = 2, 1, 64, 1
    C = H * vdim + 2 * G * state
    x = torch.zeros(N, C + 2 * H, device=DEV)
    x[:, :H * vdim] = far(N * H * vdim).view(N, -1)
    zero = lambda *s: torch.zeros(*s, device=DEV)  # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    got = ops.ssd_prep(ctx, x, 0, C, H, vdim, G, state, taps, torch.ones(taps, C, device=DEV), zero(C), zero(1, 1, C), i32([0]), i32([0, N]), i32(list(range(N))), zero(H), zero(H))[0]
    same(got, x[:, :H * vdim] + 0.0)


def test_convolved_values_do_not_follow_the_portion(ctx, ops):
    """a row beside few and beside many others: the same bits from rows by warps and from tiles of rows, for the delta rule's values and a state space layer's"""
    g = torch.Generator(device=DEV).manual_seed(5)
    H, G, dim, vdim, taps, N = 2, 1, 64, 64, 4, 2048
    C = 2 * G * dim + H * vdim
    x, w, b = torch.randn(N, C + 2 * H, generator=g, device=DEV) * 3, torch.randn(taps, C, generator=g, device=DEV), torch.randn(C, generator=g, device=DEV)
    zero = lambda *s: torch.zeros(*s, device=DEV)  # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731

    def both(n):
        v = ops.delta_rule(ctx, x[:n], (0, G * dim, 2 * G * dim, C, C + H), H, G, dim, vdim, taps, w, zero(1, taps - 1, C), zero(1, H, dim, vdim), i32([0]), i32([0, n]),
                           i32(list(range(n))), zero(H), zero(H), max_qlen=n)[3]
        y = ops.ssd_prep(ctx, x[:n], 0, C, H, vdim, G, dim, taps, w, b, zero(1, taps - 1, C), i32([0]), i32([0, n]), i32(list(range(n))), zero(H), zero(H))
        return v, y[0], y[2], y[3]
    many = both(N)
    for n in (1, 7, 300, 511):
        for few, all_ in zip(both(n), many):
            assert torch.equal(few, all_[:n])
