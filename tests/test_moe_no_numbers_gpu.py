"""Tokens whose router scores are no numbers (a NaN that came in from below): every choice names an expert, the other tokens come out as without them, and
their own results are NaN."""
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("E,top", [(16, 2), (24, 3), (64, 5)])
@pytest.mark.parametrize("score", ["ROUTE_SIGMOID", "ROUTE_SOFTMAX", "ROUTE_CHOSEN"])
def test_tokens_without_numbers(ctx, E, top, score):
    ops = importlib.import_module("nano-vllm-candle_b200.ops")
    N, H, bad = 300, 512, [0, 7, 299]
    g = torch.Generator(device=DEV).manual_seed(E)
    z, corr = torch.randn(N, E, generator=g, device=DEV), torch.randn(E, generator=g, device=DEV) * 0.1
    x = torch.randn(N, H, generator=g, device=DEV).to(torch.bfloat16)

    def run(z):
        idx, w = ops.moe_route_logits_ex(ctx, z, corr, E, top, 1.0, getattr(ops, score), True)
        offsets, src, pos, groups = ops.moe_sort_padded(ctx, idx, E)
        assert bool(((idx >= 0) & (idx < E)).all()) and bool(((pos >= 0) & (pos < src.numel())).all())
        return idx, w, ops.moe_combine(ctx, ops.gather_rows(ctx, x, src, offsets[E:]).float(), pos, w)
    want, (idx, w, got) = run(z), run(z.index_fill(0, torch.tensor(bad, device=DEV), float("nan")))
    good = torch.ones(N, dtype=torch.bool, device=DEV)
    good[bad] = False
    for a, b in zip((idx, w, got), want):
        assert torch.equal(a[good], b[good])
    assert bool(w[~good].isnan().all()) and bool(got[~good].isnan().all())
    h = torch.full((3, H), float("nan"), device=DEV)
    idx, w, _ = ops.moe_route(ctx, h, torch.randn(E, H, generator=g, device=DEV), corr, None, top, 1.0)
    assert bool(((idx >= 0) & (idx < E)).all()) and bool(w.isnan().all())
