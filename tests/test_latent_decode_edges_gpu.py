"""Latent attention's decode step at its edges: the preparation's 16-byte rows against its general form, and decode attention over shared rows where clusters of
1 to 16 CTAs share a sequence's keys, down to empty shares.  Bounds: fp32 sums in another order differ by a few 2^-24 of the norm (1e-6 here), a bf16 result
may round to the neighbouring number, up to 2^-7 of its value away; attention keeps weights of 8 bits over fp32 sums (1e-2 of the largest output)."""
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    return importlib.import_module("nano-vllm-candle_b200.ops")


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n0,n1,rot_dim,rot_dims,half", [(4, 4, 0, 0, True), (512, 96, 32, 32, True), (516, 64, 64, 24, False), (1024, 112, 16, 8, True), (128, 100, 28, 12, False)])
def test_rows_of_the_latent_preparation(ctx, ops, dtype, n0, n1, rot_dim, rot_dims, half):
    N, off = 7, n0 + 4
    g = torch.Generator(device=DEV).manual_seed(n0)
    x = torch.randn(N, off + n1 + rot_dim + 4, generator=g, device=DEV)
    w0, w1 = torch.randn(n0, generator=g, device=DEV), torch.randn(n1, generator=g, device=DEV)
    slots, pos = i32([5, -1, 0, 9, 3, 8, 1]), i32([0, 3, 17, 4, 9, 1, 30])
    table = ops.rotary_table(ctx, 10000.0, rot_dims, 40) if rot_dims else None
    got = []
    for pad in (0, 1):                       # odd strides take the general form
        rows = torch.zeros(N, x.shape[1] + pad, device=DEV)
        rows[:, :x.shape[1]] = x
        cache = torch.full((10, n1 + rot_dim), 7.0, device=DEV, dtype=dtype)
        out = ops.latent_norm_store_rot(ctx, rows, n0, off, n1, w0, w1, 1e-6, cache, slots, rot_dim, rot_dims, half, table, pos if rot_dims else None, dtype)
        got.append((out.float(), cache.float()))
    tol = 1e-6 if dtype == torch.float32 else 2.0 ** -7
    for a, b in zip(*got):
        assert float(((a - b).abs() - tol * b.abs()).max()) <= 1e-6 * float(b.abs().max())


@pytest.mark.parametrize("heads", [8, 16, 24])
@pytest.mark.parametrize("lens,table", [([1, 16, 17], 64), ([129, 300], 320), ([5, 700], 704), ([2048], 2048), ([33] * 20 + [400], 400)])
@pytest.mark.parametrize("window", [0, 300])
def test_shared_decode_by_clusters(ctx, ops, heads, lens, table, window):
    D, R, bs, B = 128, 96, 16, len(lens)
    g = torch.Generator(device=DEV).manual_seed(heads + table)
    pages = table // bs
    cache = torch.randn(B * pages * bs, D, generator=g, device=DEV).to(torch.bfloat16)
    q = torch.randn(B, heads * D, generator=g, device=DEV).to(torch.bfloat16)
    tables = torch.randperm(B * pages, generator=g, device=DEV).to(torch.int32).view(B, pages)
    sink = torch.randn(heads, generator=g, device=DEV)
    o = ops.attn_paged_wide(ctx, q, cache, cache, tables, i32(lens), None, 1, bs, heads, 1, D, R, D ** -0.5, window=window, sink=sink)
    for b, n in enumerate(lens):
        j = torch.arange(max(0, n - window) if window else 0, n, device=DEV)
        k = cache[tables[b, j // bs].long() * bs + j % bs].double()
        s = q[b].view(heads, D).double() @ k.T * D ** -0.5
        w = torch.softmax(torch.cat([s, sink.double()[:, None]], 1), 1)[:, :-1]
        want = (w @ k[:, :R]).reshape(-1)
        assert float((o[b].double() - want).abs().max()) <= 1e-2 * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("sigmoid", [False, True])
@pytest.mark.parametrize("window,length", [(100, 300), (200, 300), (300, 420), (0, 1000)])       # 1, 2, 4 and 8 CTAs share the keys
def test_an_infinite_value_comes_out_as_one(ctx, ops, window, length, sigmoid):
    """Equal scores give every visible key a weight above 0, so an infinite value makes its column's result infinite and no other number anything but finite."""
    H, G, D, bs, B = 4, 2, 64, 16, 2
    g = torch.Generator(device=DEV).manual_seed(window)
    pages = 1024 // bs
    k, v = (torch.randn(B * pages * bs, G * D, generator=g, device=DEV).to(torch.bfloat16) for _ in range(2))
    tables = torch.arange(B * pages, device=DEV, dtype=torch.int32).view(B, pages)
    v[length - 20, 7], v[pages * bs + length - 90, D + 33] = float("inf"), -float("inf")
    o = ops.attn_paged_wide(ctx, torch.zeros(B, H * D, device=DEV, dtype=torch.bfloat16), k, v, tables, i32([length, length]), None, 1, bs, H, G, D, D, D ** -0.5, window=window,
                            sigmoid=sigmoid).float().view(B, H, D)
    want = torch.zeros_like(o)
    want[0, :2, 7], want[1, 2:, 33] = float("inf"), -float("inf")
    assert torch.equal(torch.where(o.isfinite(), torch.zeros_like(o), o), want)


@pytest.mark.parametrize("lens", [[28, 56, 60, 104, 112, 120, 224, 480], [28, 56, 28, 56, 28, 56] * 6])
def test_results_are_sums_over_sums_rounded_once(ctx, ops, lens):
    """Equal scores and whole values: sums and weights are exact, so a result is one division, rounded to bf16, whoever shares the keys.  (About a
    hundredth of these quotients lie in the middle between two bf16 numbers, where a product with a rounded reciprocal falls to either side.)"""
    D, R, bs, B, H = 128, 96, 16, len(lens), 8
    g = torch.Generator(device=DEV).manual_seed(5)
    pages = 704 // bs
    cache = (torch.rand(B * pages * bs, D, generator=g, device=DEV) * torch.randint(2, 129, (D,), generator=g, device=DEV)).floor().to(torch.bfloat16)
    tables = torch.arange(B * pages, device=DEV, dtype=torch.int32).view(B, pages)
    o = ops.attn_paged_wide(ctx, torch.zeros(B, H * D, device=DEV, dtype=torch.bfloat16), cache, cache, tables, i32(lens), None, 1, bs, H, 1, D, R, D ** -0.5)
    for b, n in enumerate(lens):
        total = cache[b * pages * bs:b * pages * bs + n, :R].float().sum(0)
        assert torch.equal(o[b].view(H, R), (total / torch.full_like(total, n)).to(torch.bfloat16).expand(H, R))
