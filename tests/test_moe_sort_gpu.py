"""The experts' counting sort against a stable sort, at the edges of its batches (32 pairs, 8 x 32 per warp, 32 warps) and with pairs that name no expert."""
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("E", [1, 2, 3, 16, 33, 256, 320])
@pytest.mark.parametrize("P", [1, 31, 32, 33, 1025, 8192, 8193, 20000])
@pytest.mark.parametrize("kind", ["any", "one", "none among them"])
def test_sort_is_a_stable_one(ctx, P, E, kind):
    ops = importlib.import_module("nano-vllm-candle_b200.ops")
    g = torch.Generator().manual_seed(P * 1000 + E)
    low, high = {"any": (0, E), "one": (E - 1, E), "none among them": (-2, E + 2)}[kind]
    idx = torch.randint(low, high, (P, 1), generator=g, dtype=torch.int32)
    there = (idx[:, 0] >= 0) & (idx[:, 0] < E)
    order = torch.sort(torch.where(there, idx[:, 0], E), stable=True).indices[:int(there.sum())]
    offsets, src, pos = (t.cpu() for t in ops.moe_sort(ctx, idx.to(DEV), E))
    assert offsets.tolist() == [0] + torch.bincount(idx[there, 0], minlength=E).cumsum(0).tolist()
    assert torch.equal(src[:order.numel()].long(), order)
    want = torch.zeros(P, dtype=torch.int32)
    want[order] = torch.arange(order.numel(), dtype=torch.int32)
    assert torch.equal(pos, want)
    # groups padded to whole tiles: the same order behind other starts, -1 between, every tile's group
    offsets, src, pos, groups = (t.cpu() for t in ops.moe_sort_padded(ctx, idx.to(DEV), E, 128))
    tiles = (torch.bincount(idx[there, 0], minlength=E) + 127) // 128
    starts = torch.cat([torch.zeros(1, dtype=torch.long), tiles.cumsum(0) * 128])
    assert torch.equal(offsets.long(), starts)
    assert torch.equal(groups[:int(tiles.sum())].long(), torch.repeat_interleave(torch.arange(E), tiles)) and bool((groups[int(tiles.sum()):] == -1).all())
    rows = src[:int(starts[-1])].long()
    assert torch.equal(rows[rows >= 0], order) and bool((rows >= -1).all())
    at = pos[there].long()
    assert torch.equal(rows[at], there.nonzero()[:, 0]) and torch.equal(groups[at // 128], idx[there, 0])
