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
