"""Products inside the ranges where the library chooses another kernel by size: the fused query / key / value projection below 8 192 rows, and
narrow products over many rows on tiles of 32, 64 and 128 columns.  Both are compared with the kernel they took the place of: the first is
bit-identical; the second sums the same exact bf16 products in fp32 in another order: 64-term partial sums of numbers near 1, below 1e-3."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


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
