"""Kernels that start while the one in front of them still runs read what that one writes only behind their wait: chains without a pause, every step on new numbers,
against the same steps one at a time."""
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    return importlib.import_module("nano-vllm-candle_b200.ops")


def chain(make, steps=40):
    """make(i) queues step i and returns its outputs; the same without anything in flight."""
    torch.cuda.synchronize()
    got = [make(i) for i in range(steps)]
    torch.cuda.synchronize()
    for i in range(steps):
        want = make(i)
        torch.cuda.synchronize()
        for a, b in zip(got[i], want):
            assert torch.equal(a, b), i


@pytest.mark.parametrize("N", [64, 3000])
def test_latent_rows_behind_a_gather(ctx, ops, N):
    table = torch.randn(500, 640, device=DEV)
    ids = torch.randint(0, 500, (40, N), device=DEV, dtype=torch.int32)
    w0, w1 = torch.randn(512, device=DEV), torch.randn(96, device=DEV)
    slots, pos, tab = torch.arange(N, device=DEV, dtype=torch.int32), torch.zeros(N, device=DEV, dtype=torch.int32), ops.rotary_table(ctx, 10000.0, 32, 4)

    def step(i):
        cache = torch.empty(N, 128, device=DEV, dtype=torch.bfloat16)
        return ops.latent_norm_store_rot(ctx, ops.embed_gather_f32(ctx, ids[i], table), 512, 512, 96, w0, w1, 1e-6, cache, slots, 32, 32, True, tab, pos, torch.bfloat16), cache
    chain(step)


@pytest.mark.parametrize("N", [64, 3000])
def test_gates_behind_a_gather(ctx, ops, N):
    table = torch.randn(500, 2048, device=DEV)
    ids = torch.randint(0, 500, (40, N), device=DEV, dtype=torch.int32)
    z, w = torch.randn(N, 2048, device=DEV), torch.randn(128, device=DEV)
    chain(lambda i: [ops.head_gate_w(ctx, ops.embed_gather_f32(ctx, ids[i], table), z, w, 16, 128, True, 1e-5, "silu", 1.0, out_dtype=torch.bfloat16)])


@pytest.mark.parametrize("N,E,top", [(40, 16, 2), (4000, 16, 2), (4000, 24, 3), (3000, 64, 5)])
def test_experts_passes_behind_one_another(ctx, ops, N, E, top):
    H = 1024
    table = torch.randn(500, E, device=DEV)
    ids = torch.randint(0, 500, (40, N), device=DEV, dtype=torch.int32)
    x, corr = torch.randn(N, H, device=DEV).to(torch.bfloat16), torch.zeros(E, device=DEV)
    rows_f32 = torch.randn(((N * top + E * 127 + 127) // 128) * 128, H, device=DEV)

    def step(i):
        idx, w = ops.moe_route_logits_ex(ctx, ops.embed_gather_f32(ctx, ids[i], table), corr, E, top, 1.0, ops.ROUTE_SOFTMAX, True)
        offsets, src, pos, groups = ops.moe_sort_padded(ctx, idx, E)
        rows = ops.gather_rows(ctx, x, src, offsets[E:])
        return idx, w, offsets, src, pos, groups, rows, ops.moe_combine(ctx, rows_f32, pos, w)
    chain(step, 20)
