"""Gates and convolutions whose results are fp32: a sigmoid is the library's exponential (2 units in the last place by CUDA's stated bound), one addition and a
correctly rounded division, down to the numbers below 2^-126.  Bound: 4 units of 2^-23, and one step of 2^-149, which a sigmoid below 2^-126 is rounded to, times
the number that multiplies it."""
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
