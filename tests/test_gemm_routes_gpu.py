"""Products inside the ranges where the library chooses another kernel by size: the fused query / key / value projection, narrow products over many rows on
tiles of 32, 64 and 128 columns, products of few rows and of two row tiles.  The first is compared with the two kernels that it took the place of, bit by bit, the second
with the kernel before it: the same exact bf16 products summed in fp32 in another order, 64-term partial sums of numbers near 1, below 1e-3."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.mark.parametrize("M,nh,kv,K,fused", [(1500, 4, 2, 2048, False), (1501, 32, 8, 4096, True), (3001, 16, 8, 2048, True), (5500, 16, 8, 1024, True), (6000, 16, 8, 1024, True),
                                             (6555, 16, 8, 1024, True), (8191, 8, 4, 512, True), (2400, 5, 1, 2048, False), (1000, 16, 8, 1024, True), (2000, 16, 8, 1024, True),
                                             (3000, 16, 8, 1024, True), (700, 32, 8, 2560, True), (2600, 16, 8, 2048, True),
                                             (257, 58, 2, 256, False), (257, 60, 2, 256, True),      # 62 and 64 tiles on 74 pairs of SMs, one row in the second row tile
                                             (2049, 13, 1, 1024, True), (4097, 5, 1, 2048, True),    # an odd number of heads: the last tile has one
                                             (2523, 16, 8, 1024, True), (2523, 16, 8, 4096, False), (1300, 16, 8, 2048, False),
                                             (5120, 66, 4, 512, True)])      # 740 tiles: ten full waves
def test_fused_projection_between_its_thresholds(ctx, nvc, M, nh, kv, K, fused):
    g = torch.Generator().manual_seed(M + K)
    N, slots = (nh + 2 * kv) * 128, M + 64
    a, w = torch.randn(M, K, generator=g).to(BF16).cuda(), (torch.randn(N, K, generator=g) / math.sqrt(K)).to(BF16).cuda()
    qw, kw = ((1 + 0.2 * torch.randn(128, generator=g)).to(BF16).cuda() for _ in range(2))
    pos = torch.randint(0, 2000, (M,), generator=g, dtype=torch.int32).cuda()
    slot = torch.randperm(slots, generator=g)[:M].to(torch.int32)
    slot[2] = -1
    slot, tab, got = slot.cuda(), ctx.rope_table(1e6, 128, 2000), []
    for off in (0, 1):
        nvc.lib().nvc_debug_set(7, off)
        try:
            kc = torch.zeros(slots, kv, 128, dtype=BF16, device="cuda")
            vc = torch.zeros_like(kc)
            before = nvc.lib().nvc_ctx_launch_count(ctx.h)
            got.append((ctx.qkv_proj_norm_rope(a, w, qw, kw, 1e-6, tab, pos, nh, kv, 128, slot_mapping=slot, k_cache=kc, v_cache=vc), kc, vc))
            assert nvc.lib().nvc_ctx_launch_count(ctx.h) - before == (1 if fused and not off else 2)
        finally:
            nvc.lib().nvc_debug_set(7, 0)
    for x, y in zip(*got):
        assert torch.equal(x.view(torch.int16), y.view(torch.int16))


def test_projection_refuses_rows_that_overlap(ctx):
    """A row stride below the row's length is an error in the fused range too: 128 tiles, two waves that are 86 % full."""
    M, nh, kv, K = 2000, 16, 8, 2048
    N = (nh + 2 * kv) * 128
    a, w, qkv = (torch.zeros(n, m, dtype=BF16, device="cuda") for n, m in ((M, K), (N, K), (M, N)))
    one, tab, pos = torch.ones(128, dtype=BF16, device="cuda"), ctx.rope_table(1e6, 128, M), torch.arange(M, dtype=torch.int32, device="cuda")
    call = lambda lda: ctx.l.nvc_qkv_proj_norm_rope(ctx.h, a.data_ptr(), lda, w.data_ptr(), qkv.data_ptr(), M, K, one.data_ptr(), one.data_ptr(), 1e-6,  # noqa: E731
                                                    tab.data_ptr(), pos.data_ptr(), None, None, None, nh, kv, 128, torch.cuda.current_stream().cuda_stream)
    before = ctx.l.nvc_ctx_launch_count(ctx.h)
    assert call(K) == 0 and ctx.l.nvc_ctx_launch_count(ctx.h) == before + 1
    assert call(K - 8) != 0 and call(K // 2) != 0
    torch.cuda.synchronize()


@pytest.mark.parametrize("M", [129, 200, 1000, 2368, 2369, 18944, 18945])
@pytest.mark.parametrize("N", [16, 48, 64, 240, 256])
@pytest.mark.parametrize("K", [64, 192, 2048])
def test_narrow_products_over_many_rows(ctx, M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a, w = torch.randn(M, K, generator=g, device="cuda").to(BF16), (torch.randn(N, K, generator=g, device="cuda") / math.sqrt(K)).to(BF16)
    buf = torch.full((M, N + 16), float("nan"), device="cuda")
    got = ctx.gemm(a, w, out=buf[:, :N])
    assert float((got - ctx.gemm(a, w, out_dtype=torch.float32, force_bn=512)).abs().max()) < 1e-3
    assert bool(torch.isnan(buf[:, N:]).all())


@pytest.mark.parametrize("M", [1, 7, 15, 16, 17, 33, 63, 64, 65, 100, 128])
@pytest.mark.parametrize("N,K", [(16, 512), (48, 256), (1024, 3072), (2048, 1024), (2064, 2048), (6144, 2560), (4096, 4096), (19456, 512), (1040, 6144), (12288, 2048)])
def test_few_rows(ctx, M, N, K):
    """Up to 64 rows run on products of 64 rows, 65 to 128 on products of 128, with the width and split of their choice.  Sums of K exact products of size K^-1/2 in fp32, in
    another order: 1e-4 of the largest; bf16 results one more rounding, 2^-8 of the value.  Rows and columns around the results of either type keep their marks."""
    ops = __import__("importlib").import_module("nano-vllm-candle_b200.ops")
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a, w = torch.randn(M, K, generator=g, device="cuda").to(BF16), (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(BF16)
    want = a.double() @ w.double().T
    top = float(want.abs().max())
    buf = torch.full((M + 1, N + 16), 7.0, device="cuda")
    ctx.gemm(a, w, out_dtype=torch.float32, out=buf[:M, :N])
    assert float((buf[:M, :N] - want).abs().max()) <= 1e-4 * top and bool((buf[M] == 7.0).all()) and bool((buf[:, N:] == 7.0).all())
    near = lambda got, ref: float(((got.double() - ref).abs() - 2.0 ** -8 * ref.abs()).max()) <= 1e-4 * float(ref.abs().max())  # noqa: E731
    buf = torch.full((M + 1, N + 16), 7.0, device="cuda", dtype=BF16)
    ctx.gemm(a, w, out=buf[:M, :N])
    assert near(buf[:M, :N], want) and bool((buf[M] == 7.0).all()) and bool((buf[:, N:] == 7.0).all())
    assert near(ops.gemm_act(ctx, a, w, ops.ACT_RELU2), want.clamp(min=0) ** 2)
    if N % 32 == 0:
        gu = torch.cat([w[:N // 2], w[N // 2:]])
        buf = torch.full((M + 1, N // 2 + 16), 7.0, device="cuda", dtype=BF16)
        ctx.gemm_silu_mul(a, ctx.interleave_gate_up(gu), out=buf[:M, :N // 2])
        assert bool((buf[M] == 7.0).all()) and bool((buf[:, N // 2:] == 7.0).all())
        assert near(buf[:M, :N // 2], torch.nn.functional.silu(want[:, :N // 2]) * want[:, N // 2:])


@pytest.mark.parametrize("M", [129, 192, 255, 256, 257])
@pytest.mark.parametrize("N,K", [(16, 1600), (64, 2048), (2368, 64), (2400, 512), (4736, 192), (4768, 2048), (9472, 128), (9504, 1024), (1024, 2048), (1024, 2112)])
def test_two_row_tiles(ctx, M, N, K):
    """129 to 256 rows over K up to 2 048, of few columns up to 1 664, run on two row tiles of 32, 64 or 128 columns as long as these are one wave; a column tile more, a row
    more or a longer K does not.  The same bounds and marks as for few rows."""
    test_few_rows(ctx, M, N, K)


@pytest.mark.parametrize("bn,kps", [(32, 4), (64, 4), (128, 2), (256, 1)])
@pytest.mark.parametrize("M", [1, 17, 63, 64, 65, 100, 128])
@pytest.mark.parametrize("S", [1, 2, 3, 4])
def test_sums_in_one_block_are_those_of_a_cluster(ctx, M, bn, kps, S):
    """Parts of K that one CTA sums in accumulators of its own and those of a cluster of one CTA per part: the same bits, inside bands that keep their marks.  22 k-blocks: a short last part; 1 040
    columns: a ragged last tile.  Sums of exact products in fp32: 1e-4 of the largest."""
    N, K = 1040, 1408
    g = torch.Generator(device="cuda").manual_seed(M + bn + S)
    a, w = torch.randn(M, K, generator=g, device="cuda").to(BF16), (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(BF16)
    want = a.double() @ w.double().T
    for dt in (BF16, torch.float32):
        apart = ctx.gemm(a, w, out_dtype=dt, force_bn=bn + 1000 * kps, force_splits=100 + S if S > 1 else 1)
        assert float(((apart.double() - want).abs() - (2.0 ** -8 if dt == BF16 else 0) * want.abs()).max()) <= 1e-4 * float(want.abs().max())
        buf = torch.full((M + 1, N + 16), 7.0, device="cuda", dtype=dt)
        if bn * S > 512:
            with pytest.raises(RuntimeError):
                ctx.gemm(a, w, out_dtype=dt, out=buf[:M, :N], force_bn=bn + 1000 * kps, force_splits=200 + S)
            continue
        ctx.gemm(a, w, out_dtype=dt, out=buf[:M, :N], force_bn=bn + 1000 * kps, force_splits=200 + S)
        assert torch.equal(buf[:M, :N], apart) and bool((buf[M] == 7.0).all()) and bool((buf[:, N:] == 7.0).all())


@pytest.mark.parametrize("N,K,S", [(1024, 2048, 4), (2048, 2048, 4), (4096, 2048, 4), (2560, 4096, 4), (4096, 4096, 4), (6144, 4096, 4), (5120, 8192, 4), (1024, 3072, 4), (4096, 1024, 1)])
@pytest.mark.parametrize("dt", [BF16, torch.float32])
def test_a_row_alone_and_beside_others(ctx, N, K, S, dt):
    """Products of up to 128 rows sum K in as many parts as before, whichever tile runs them: those of the forced cluster, bit by bit, and the same for a row alone and beside any number of others."""
    g = torch.Generator(device="cuda").manual_seed(N + K)
    a, w = torch.randn(128, K, generator=g, device="cuda").to(BF16), (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(BF16)
    forced = ctx.gemm(a, w, out_dtype=dt, force_bn=4064, force_splits=100 + S if S > 1 else 1)
    for M in (1, 16, 17, 40, 41, 49, 64, 65, 100, 128):
        assert torch.equal(ctx.gemm(a[:M], w, out_dtype=dt), forced[:M])


@pytest.mark.parametrize("M", [129, 200, 256])
@pytest.mark.parametrize("N,K", [(1024, 1024), (1024, 2048), (4096, 2048), (2048, 2048), (3584, 1792), (64, 2048), (9472, 576), (4096, 3072)])
def test_two_row_tiles_sum_like_pairs(ctx, M, N, K):
    """129 to 256 rows: the same bits as on CTA pairs with the splits of their schedule, plain and gated, inside bands that keep their marks"""
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a, w = torch.randn(M, K, generator=g, device="cuda").to(BF16), (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(BF16)
    buf = torch.full((M + 1, N + 16), 7.0, device="cuda", dtype=BF16)
    ctx.gemm(a, w, out=buf[:M, :N])
    assert torch.equal(buf[:M, :N], ctx.gemm(a, w, force_bn=512)) and bool((buf[M] == 7.0).all()) and bool((buf[:, N:] == 7.0).all())
    if N % 32 == 0:
        buf = torch.full((M + 1, N // 2 + 16), 7.0, device="cuda", dtype=BF16)
        ctx.gemm_silu_mul(a, w, out=buf[:M, :N // 2])
        assert torch.equal(buf[:M, :N // 2], ctx.gemm_silu_mul(a, w, force_bn=512)) and bool((buf[M] == 7.0).all()) and bool((buf[:, N // 2:] == 7.0).all())
