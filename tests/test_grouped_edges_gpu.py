"""The grouped product on its persistent grid: few and many tiles (all three tile widths), more tiles than SMs, column counts around the tiles, groups
without rows and groups without a product, against 64-bit sums (bf16 operands: exact products, fp32 sums of up to 1 024 terms stay within 1e-5 of the
largest value; a bf16 result within half of its last place more).  Rows that no group computes are zeros; the rows behind the groups keep the
marks of the sort and the gather."""
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    return importlib.import_module("nano-vllm-candle_b200.ops")


@pytest.mark.parametrize("tokens,E,E_real,top,N,K", [(1, 3, 3, 1, 16, 64), (64, 16, 16, 2, 400, 128), (300, 5, 3, 2, 256, 192), (2500, 6, 6, 2, 1040, 64),
                                                     (4000, 9, 8, 1, 3072, 128), (129, 1, 1, 1, 128, 1024),
                                                     (200, 8, 8, 2, 1536, 448), (64, 8, 8, 1, 768, 1024), (40, 4, 4, 2, 176, 640)])      # 128 and 64 columns, rings that wrap
@pytest.mark.parametrize("dt,act", [(torch.float32, 0), (torch.bfloat16, 1)])
def test_grouped_product(ctx, ops, tokens, E, E_real, top, N, K, dt, act):
    g = torch.Generator(device=DEV).manual_seed(tokens + N)
    h, W = (torch.randn(*s, generator=g, device=DEV).bfloat16() for s in ((tokens, K), (E_real, N, K)))
    idx = torch.rand(tokens, E, generator=g, device=DEV).topk(top, -1).indices.to(torch.int32)
    if tokens > 1000:
        idx[idx == 0] = 1 % E                              # a group without rows
    offsets, src, pos, tiles = ops.moe_sort_padded_ex(ctx, idx, E, E_real)
    x = ops.gather_rows(ctx, h, src, offsets[E:])
    y = ops.gemm_grouped(ctx, x, W, tiles, act=act, out_dtype=dt)
    end = int(offsets[E])
    assert (src[end:] == -7).all() and (x[end:] == 3).all() and (tiles[end // 128:] == -1).all()
    grp = tiles.repeat_interleave(128)
    assert (y[grp < 0] == 0).all()
    flat, e = pos.long(), idx.flatten().long()
    for k in range(E_real):
        rows = flat[e == k]
        want = h.double()[torch.nonzero(e == k)[:, 0] // top] @ W[k].double().T
        want = want.clamp(min=0) ** 2 if act else want
        tol = (1e-5 if dt == torch.float32 else 2.0 ** -8) * float(want.abs().max() if len(rows) else 0)
        assert ((y[rows].double() - want).abs() <= tol).all(), k


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_gathered_rows_of_any_16_bit_type(ctx, ops, dt):
    """Rows are copied as they are; those behind the last group hold 3 in their own type."""
    x = torch.randn(9, 64, generator=torch.Generator().manual_seed(1)).to(dt).to(DEV)
    src, n = torch.tensor([4, -1, 0, 7, 7], dtype=torch.int32, device=DEV), torch.tensor([3], dtype=torch.int32, device=DEV)
    got = ops.gather_rows(ctx, x, src, n)
    assert torch.equal(got[0], x[4]) and (got[1] == 0).all() and torch.equal(got[2], x[0]) and (got[3:] == 3).all()
