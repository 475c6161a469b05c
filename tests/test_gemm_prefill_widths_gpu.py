"""Products over a few hundred to a few thousand rows take the tile width and split that fill the last wave: what is chosen, and every width with every split, against
fp32, at rows and columns around the tiles' edges.  Bound: bf16 results round by 2^-9 of the value (2^-8 is allowed, one more ulp for the sum); fp32 sums of K products of size K^-1/2 differ by less than 1e-4 of the largest."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, BF16 = "cuda:0", torch.bfloat16


@pytest.mark.parametrize("M", [257, 300, 511, 513, 700, 1100, 1300, 2600])
@pytest.mark.parametrize("N,K", [(1024, 2048), (1024, 3072), (1040, 1024), (2048, 6144), (4096, 1024), (2064, 2048), (272, 512), (512, 4096), (1024, 6144)])
def test_widths_and_splits(ctx, M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M + N)
    a = torch.randn(M, K, generator=g, device=DEV).to(BF16)
    w = (torch.randn(N, K, generator=g, device=DEV) * K ** -0.5).to(BF16)
    want = a.float() @ w.float().T
    out = torch.full((M + 1, N), 7.0, device=DEV, dtype=BF16)
    ctx.gemm(a, w, out=out[:M])
    top = float(want.abs().max())
    assert float(((out[:M].float() - want).abs() - 2.0 ** -8 * want.abs()).max()) <= 1e-4 * top
    assert bool((out[M] == 7.0).all())
    f32 = ctx.gemm(a, w, out_dtype=torch.float32)
    assert float((f32 - want).abs().max()) <= 1e-4 * top


@pytest.mark.parametrize("M,I,K", [(300, 3072, 1024), (512, 6144, 2048), (1100, 1552, 1024), (700, 400, 2048), (300, 1536, 2048)])
def test_widths_of_gated_products(ctx, M, I, K):
    g = torch.Generator(device=DEV).manual_seed(M + I)
    a = torch.randn(M, K, generator=g, device=DEV).to(BF16)
    gu = (torch.randn(2 * I, K, generator=g, device=DEV) * K ** -0.5).to(BF16)
    z = a.float() @ gu.float().T
    want = torch.nn.functional.silu(z[:, :I]) * z[:, I:]
    got = ctx.gemm_silu_mul(a, ctx.interleave_gate_up(gu))
    assert float(((got.float() - want).abs() - 2.0 ** -8 * want.abs()).max()) <= 1e-4 * float(want.abs().max())


@pytest.mark.parametrize("S", [1, 2, 3, 4])
@pytest.mark.parametrize("NT", [128, 160, 192, 224, 256])
@pytest.mark.parametrize("M,N,K", [(300, 1040, 1024), (515, 272, 448)])
def test_every_width_with_every_split(ctx, M, N, K, NT, S):
    g = torch.Generator(device=DEV).manual_seed(M + NT + S)
    a = torch.randn(M, K, generator=g, device=DEV).to(BF16)
    w = (torch.randn(N, K, generator=g, device=DEV) * K ** -0.5).to(BF16)
    forced = dict(force_bn=512, force_splits=10000 * S + 1000 + NT)
    want = a.float() @ w.float().T
    out = torch.full((M + 1, N), 7.0, device=DEV, dtype=torch.float32)
    ctx.gemm(a, w, out_dtype=torch.float32, out=out[:M], **forced)
    assert float((out[:M] - want).abs().max()) <= 1e-4 * float(want.abs().max()) and bool((out[M] == 7.0).all())
    gu = torch.cat([w[:N // 32 * 16], w[:N // 32 * 16].flip(0)])
    z = a.float() @ gu.float().T
    want = torch.nn.functional.silu(z[:, :N // 32 * 16]) * z[:, N // 32 * 16:]
    got = ctx.gemm_silu_mul(a, ctx.interleave_gate_up(gu), **forced)
    assert float(((got.float() - want).abs() - 2.0 ** -8 * want.abs()).max()) <= 1e-4 * float(want.abs().max())


@pytest.mark.parametrize("M,N,K", [(300, 17424, 1024), (1100, 16400, 1024), (4400, 16400, 1024), (2100, 1552, 12288), (600, 256, 65600), (515, 4112, 4160)])
@pytest.mark.parametrize("f32", [False, True])
def test_bands_of_row_tiles(ctx, M, N, K, f32):
    """Weights above 32 MB are walked in bands of row tiles: the same sums as the same weights in pieces below it, bit by bit."""
    g = torch.Generator(device=DEV).manual_seed(M + N)
    a = torch.randn(M, K, generator=g, device=DEV).to(BF16)
    w = (torch.randn(N, K, generator=g, device=DEV) * K ** -0.5).to(BF16)
    dt = torch.float32 if f32 else BF16
    cut = N // 32 * 16
    assert N * K * 2 > 32 << 20 >= (N - cut) * K * 2 >= cut * K * 2
    out = torch.full((M + 1, N), 7.0, device=DEV, dtype=dt)
    ctx.gemm(a, w, out_dtype=dt, out=out[:M], force_bn=512, force_splits=1)
    pieces = torch.cat([ctx.gemm(a, p.contiguous(), out_dtype=dt, force_bn=512, force_splits=1) for p in (w[:cut], w[cut:])], 1)
    assert torch.equal(out[:M], pieces) and bool((out[M] == 7.0).all())
