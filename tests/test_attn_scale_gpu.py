"""Prompt attention with a scale of any sign, through every entry point that has a tcgen05 route: that kernel takes maxima and masks before it
scales, so a scale that is not positive has to reach another one.  Compared with softmax written out in 64 bits.  The bound: weights rounded to
bf16 (2^-9 relative, errors of different keys add up by chance) and a bf16 result, together below 2e-2 of the largest output."""
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


def plain(q, k, v, pos0, scale, window, sink):
    """q [T, H, d] at positions pos0 ..; k, v [Tk, G, d]."""
    T, H, Tk = q.shape[0], q.shape[1], k.shape[0]
    out = torch.zeros_like(q)
    i, j = torch.arange(pos0, pos0 + T)[:, None], torch.arange(Tk)[None]
    for h in range(H):
        g = h // (H // k.shape[1])
        s = (q[:, h] @ k[:, g].T * scale).masked_fill((j > i) | ((i - j >= window) if window else False), float("-inf"))
        m = s.max(-1, keepdim=True).values
        e = (s - m).exp()
        den = e.sum(-1, keepdim=True) + (0 if sink is None else (sink[h] - m).exp())
        out[:, h] = e / den @ v[:, g]
    return out


@pytest.mark.parametrize("scale", [-0.1, 0.0, 0.1])
@pytest.mark.parametrize("entry,window,sink", [("wide", 0, False), ("wide", 70, True), ("window", 0, True), ("window", 40, False), ("shared", 0, True), ("varlen", 0, False)])
def test_prompts_with_a_scale_of_any_sign(ctx, ops, entry, window, sink, scale):
    g = torch.Generator().manual_seed(5)
    H, G, d, block = 4, 2, 128, 32
    q_lens, old = [129, 64], ([0, 0] if entry == "varlen" else [0, 75])
    N, ctx_lens = sum(q_lens), [a + b for a, b in zip(q_lens, old)]
    need = [(n + block - 1) // block for n in ctx_lens]
    pages = torch.randperm(sum(need), generator=g).tolist()
    tables = [[pages.pop() for _ in range(n)] + [-1] * (max(need) - n) for n in need]
    q = torch.randn(N, H * d, generator=g).bfloat16()
    k, v = (torch.randn(sum(need) * block, G * d, generator=g).bfloat16() for _ in range(2))
    if entry == "shared":
        v = k
    sk = torch.randn(H, generator=g) if sink else None
    skd = sk.to(DEV) if sink else None
    cu = [0, q_lens[0], N]
    rows = [torch.tensor([tables[b][t // block] * block + t % block for t in range(n)]) for b, n in enumerate(ctx_lens)]
    kd, vd = k.to(DEV), v.to(DEV)
    if entry == "shared":
        vd = kd
    paged = (i32(tables), i32(ctx_lens), i32(cu), max(q_lens), block, H, G)
    if entry == "wide":
        got = ops.attn_paged_wide(ctx, q.to(DEV), kd, vd, *paged, d, d, scale, window=window, sink=skd)
    elif entry == "window":
        got = ops.prefill_attn_window(ctx, q.to(DEV), kd, vd, *paged, scale, window, sink=skd)
    elif entry == "shared":
        got = ops.prefill_attn_shared(ctx, q.to(DEV), kd, *paged, scale, sink=skd)
    else:
        new = [torch.cat([x[r] for r in rows]).to(DEV) for x in (k, v)]
        call = lambda: ctx.prefill_attn(q.to(DEV), *new, i32(cu), max(q_lens), H, G, d, scale)  # noqa: E731
        if scale <= 0:                        # no other kernel behind this one: an error, where results were wrong
            with pytest.raises(Exception, match="scale"):
                call()
            return
        got = call()
    for b, n in enumerate(q_lens):
        want = plain(q[cu[b]:cu[b + 1]].double().view(n, H, d), k[rows[b]].double().view(-1, G, d), v[rows[b]].double().view(-1, G, d), old[b], scale, window,
                     None if sk is None else sk.double())
        err = (got[cu[b]:cu[b + 1]].double().cpu().view(n, H, d) - want).abs().max()
        assert float(err) <= 2e-2 * max(1.0, float(want.abs().max())), (b, float(err))
