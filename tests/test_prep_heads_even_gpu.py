"""Preparation of projection rows whose warps hold heads of one kind, against the general kernel (an odd row stride takes it).  Bounds: the square sum's order
differs, a few 2^-24 of the norm, so 1e-6 of the largest number; a bf16 result may round to
the neighbouring number, which is up to 2^-7 of its value away (8 significant bits)."""
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("N", [3, 1100])
@pytest.mark.parametrize("rot,half", [(0, False), (24, False), (32, True)])
@pytest.mark.parametrize("H,G,d,vd", [(16, 8, 128, 128), (36, 4, 128, 100), (4, 4, 68, 128), (8, 8, 64, 64), (16, 8, 32, 60)])
def test_heads_of_one_kind_per_warp(ctx, dtype, N, rot, half, H, G, d, vd):
    ops = importlib.import_module("nano-vllm-candle_b200.ops")
    g = torch.Generator(device=DEV).manual_seed(H * d + rot)
    cols = (H + G) * d + G * vd
    x, bias = torch.randn(N, cols, generator=g, device=DEV), torch.randn(cols, generator=g, device=DEV)
    qn, kn = torch.randn(d, generator=g, device=DEV), torch.randn(d, generator=g, device=DEV)
    pos = torch.randint(0, 50, (N,), generator=g, device=DEV, dtype=torch.int32)
    slots = torch.randperm(N + 2, generator=g, device=DEV)[:N].to(torch.int32)
    slots[N // 2] = -1
    table = ops.rotary_table(ctx, 10000.0, rot, 50) if rot else None
    for normed, biased in ((True, True), (False, True), (True, False)):
        got = []
        for pad in (0, 1):
            rows = torch.zeros(N, cols + pad, device=DEV)
            rows[:, :cols] = x
            q = torch.zeros(N, H * d, device=DEV, dtype=dtype)
            k, v = torch.full((N + 2, G * d), 3.0, device=DEV, dtype=dtype), torch.full((N + 2, G * vd), 3.0, device=DEV, dtype=dtype)
            ops.qkv_prep(ctx, rows, 0, H * d, (H + G) * d, H, G, d, vd, q, k, v, bias=bias if biased else None, q_norm=qn if normed else None,
                         k_norm=kn if normed else None, rot_dims=rot, rot_half=half, rot_table=table, positions=pos if rot else None, k_scale=0.5, v_scale=2.0,
                         slot_mapping=slots)
            got.append([t.float() for t in (q, k, v)])
        tol = 1e-6 if dtype == torch.float32 else 2.0 ** -7
        for a, b in zip(*got):
            assert float(((a - b).abs() - tol * b.abs()).max()) <= 1e-6 * float(b.abs().max())
