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


@pytest.mark.parametrize("pad", [0, 1])                 # rows that allow 16-byte accesses, and rows that do not
def test_latent_rows_with_slots_of_the_moment(ctx, ops, pad):
    """Slots and positions are static operands: another library's kernel may write them right in front of the call, which plain stream order covers."""
    N = 300
    table, ids = torch.randn(500, 640 + pad, device=DEV), torch.randint(0, 500, (40, N), device=DEV, dtype=torch.int32)
    w0, w1, tab = torch.randn(512, device=DEV), torch.randn(96, device=DEV), ops.rotary_table(ctx, 10000.0, 32, 1024)
    slots, pos = torch.arange(N, device=DEV, dtype=torch.int32), torch.zeros(N, device=DEV, dtype=torch.int32)

    def step(i):
        cache = torch.zeros(2 * N, 128, device=DEV, dtype=torch.bfloat16)
        x = ops.embed_gather_f32(ctx, ids[i], table)
        slots.copy_((torch.arange(N, device=DEV, dtype=torch.int32) * 7 + 11 * i) % (2 * N - 1))
        pos.copy_(slots + i)
        return ops.latent_norm_store_rot(ctx, x, 512, 512, 96, w0, w1, 1e-6, cache, slots, 32, 32, True, tab, pos, torch.bfloat16), cache
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


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("N,E,top", [(40, 16, 2), (3000, 24, 3)])
def test_narrow_and_16_bit_passes_behind_the_sort(ctx, ops, N, E, top, dt):
    """rows below 512 numbers, 16-bit rows to combine, identity experts, rows scaled on their way to the experts"""
    H = 256
    table = torch.randn(500, E, device=DEV)
    ids = torch.randint(0, 500, (20, N), device=DEV, dtype=torch.int32)
    x, corr = torch.randn(N, H, device=DEV).to(torch.bfloat16), torch.zeros(E, device=DEV)
    cap = ((N * top + E * 127 + 127) // 128) * 128
    y, shared, gate = torch.randn(cap, H, device=DEV).to(dt), torch.randn(N, H, device=DEV).to(dt), torch.rand(N, device=DEV)
    wr = torch.randn(E, H, device=DEV) * H ** -0.5

    def step(i):
        idx, w = ops.moe_route_logits_ex(ctx, ops.embed_gather_f32(ctx, ids[i], table), corr, E, top, 1.0, ops.ROUTE_SOFTMAX, True)
        offsets, src, pos, groups = ops.moe_sort_padded_ex(ctx, idx, E, E - 2)
        rows = ops.gather_rows(ctx, x, src, offsets[E:])
        both = ops.moe_combine(ctx, y, pos, w, shared, gate), ops.moe_combine_identity(ctx, y, pos, w, idx, E - 2, shared)
        return (rows, *both, ops.moe_scatter_scaled(ctx, shared, pos, w, cap), *ops.moe_route(ctx, ops.embed_gather_f32(ctx, ids[i] % N, shared.float()).to(dt), wr, corr, None, top, 1.0)[:2])
    chain(step, 20)


@pytest.mark.parametrize("N", [1, 32, 64])
def test_choice_and_draw_behind_their_product(ctx, ops, N):
    V, K = 32768, 256
    table, w = torch.randn(500, K, device=DEV).to(torch.bfloat16), (torch.randn(V, K, device=DEV) * 0.1).to(torch.bfloat16)
    ids = torch.randint(0, 500, (40, N), device=DEV, dtype=torch.int32)
    t, s = torch.full((N,), 0.8, device=DEV), torch.arange(N, device=DEV)

    def step(i):
        logits = ctx.gemm(ctx.embed_gather(ids[i], table), w, out_dtype=torch.float32)
        drawn = ctx.sample_gumbel(logits, t, s, i)
        chosen = ctx.argmax_last(logits)
        return (*drawn, *chosen, ctx.embed_gather(chosen[0], w))
    chain(step)


@pytest.mark.parametrize("B,ctx_len", [(1, 3000), (5, 700), (64, 300)])
def test_paged_decode_behind_its_queries(ctx, ops, B, ctx_len):
    """whole and split: the combination reads what the kernel in front of it wrote"""
    nh, kv, hd, bs = 16, 8, 128, 256
    pages = (ctx_len + bs - 1) // bs
    k, v = (torch.randn(B * pages * bs, kv * hd, device=DEV).to(torch.bfloat16) for _ in range(2))
    tables = torch.arange(B * pages, device=DEV, dtype=torch.int32).view(B, pages)
    lens = torch.full((B,), ctx_len, device=DEV, dtype=torch.int32)
    table, ids = torch.randn(500, nh * hd, device=DEV).to(torch.bfloat16), torch.randint(0, 500, (40, B), device=DEV, dtype=torch.int32)
    chain(lambda i: [ctx.paged_decode_attn(ctx.embed_gather(ids[i], table), k, v, tables, lens, nh, kv, hd, bs, hd ** -0.5)])


@pytest.mark.parametrize("N", [8, 2000])
@pytest.mark.parametrize("H", [256, 1008])
def test_norms_and_units_behind_a_gather(ctx, ops, N, H):
    table, w, r = torch.randn(500, H, device=DEV), torch.randn(H, device=DEV), torch.randn(N, H, device=DEV)
    half, wh = table.to(torch.bfloat16), w.to(torch.bfloat16)
    ids, last = torch.randint(0, 500, (40, N), device=DEV, dtype=torch.int32), torch.arange(0, N, 3, device=DEV, dtype=torch.int32)

    def step(i):
        new = lambda: ops.embed_gather_f32(ctx, ids[i], table)  # noqa: E731
        res = [torch.empty(N, H, device=DEV) for _ in range(2)]
        out = [*ops.rms_norm_pair(ctx, r, [new()], w), *ops.rms_norm_sandwich(ctx, r, new(), w, w), *ops.rms_norm_blend(ctx, r, new(), w, 0.5, w=w),
               ops.dyt_norm(ctx, new(), [], w, w, w[:1], write_back=False)[1], ops.act_mul(ctx, new(), H // 2, 1), ops.act_mul(ctx, ctx.embed_gather(ids[i], half), H // 2, 1),
               ctx.fused_add_rmsnorm(ctx.embed_gather(ids[i], half), wh, 1e-6, new(), res[0]), ctx.silu_and_mul(ctx.embed_gather(ids[i], half)),
               *ctx.gather_rows(ctx.embed_gather(ids[i], half), new(), last), *res[:1]]
        return [t for t in out if t is not None]
    chain(step)
