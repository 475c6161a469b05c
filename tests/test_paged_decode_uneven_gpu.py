"""Paged decode with contexts of different lengths: taken in order of length by teams of two or four warps, against plain fp32 attention
(the bound of the other paged decode tests: probabilities and results are bf16)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("nh,kv,block,lens", [
    (32, 8, 256, [200 + 20 * i for i in range(64)]),            # longest under 7/4 of the average: teams of two
    (32, 8, 256, [100 + 31 * ((i * 37) % 64) for i in range(64)]),       # teams of four, two units per CTA
    (16, 8, 16, [33] * 63 + [9000]),
    (16, 8, 64, [1, 31, 32, 33, 255, 256, 257, 5000] * 8),
    (16, 16, 64, [7, 900] + [64] * 35),                         # 592 units: the last that two per CTA hold
    (8, 8, 16, [300, 20] * 37 + [1]),                           # 600 units: one per CTA
    (16, 16, 64, [40 * (1 + i % 11) for i in range(150)] + [8000, 1]),   # teams of two in order
    (8, 2, 32, [100] * 599 + [1001]),
    (8, 2, 32, [3] * 200),                                      # short: no order
    (40, 4, 64, [64 * (1 + i % 3) for i in range(90)] + [7777] * 3),     # ten heads per key head
])
def test_uneven_contexts(ctx, nh, kv, block, lens):
    g = torch.Generator(device=DEV).manual_seed(len(lens) + nh)
    B, hd = len(lens), 128
    need = [(n + block - 1) // block for n in lens]
    pages = torch.randperm(sum(need), generator=g, device=DEV).to(torch.int32)
    tables = torch.full((B, max(need)), -1, dtype=torch.int32, device=DEV)
    at = 0
    for b, n in enumerate(need):
        tables[b, :n] = pages[at:at + n]
        at += n
    k, v = (torch.randn(at, block, kv, hd, generator=g, device=DEV).bfloat16() for _ in range(2))
    q = torch.randn(B, nh * hd, generator=g, device=DEV).bfloat16()
    run = lambda: ctx.paged_decode_attn(q, k, v, tables, torch.tensor(lens, dtype=torch.int32, device=DEV), nh, kv, hd, block, hd ** -0.5)  # noqa: E731
    got = run()
    assert torch.equal(run(), got)
    for b in range(0, B, 1 + B // 100):
        rows = (tables[b, :need[b]].long()[:, None] * block + torch.arange(block, device=DEV)).flatten()[:lens[b]]
        kk, vv = (t.view(-1, kv, hd)[rows].float().repeat_interleave(nh // kv, 1) for t in (k, v))
        w = torch.softmax(torch.einsum("hd,nhd->hn", q[b].float().view(nh, hd), kk) * hd ** -0.5, -1)
        want = torch.einsum("hn,nhd->hd", w, vv)
        assert float((got[b].float().view(nh, hd) - want).abs().max()) <= 2e-2 * max(1e-1, float(want.abs().max())), b
