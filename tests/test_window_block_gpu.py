"""Preparation and attention of the window block at the edges of their kernels.  Attention on tcgen05 is compared with the same call on
numbers kept in float32 (the FMA kernel): 128 keys of weight near 1 / 128 whose bf16 rounding errors of 2^-9 add up by chance stay below
2e-2 of the largest output.  The preparation in float32 is compared with 64-bit arithmetic (1e-5: sums of 128 squares, one division)."""
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


@pytest.mark.parametrize("q_lens,old", [([64], [0]), ([1, 127, 128], [5, 0, 70]), ([129, 63, 200], [0, 64, 1]), ([256, 17], [300, 0])])
@pytest.mark.parametrize("window,sink,gate,scale,block,G", [(0, False, False, 1.0, 64, 2), (1, True, True, 0.5, 16, 1), (64, True, False, 2.0, 32, 4), (130, False, True, 1.0, 128, 2)])
def test_portions_with_window_sink_gate_and_factor(ctx, ops, q_lens, old, window, sink, gate, scale, block, G):
    g = torch.Generator().manual_seed(sum(q_lens) + window)
    H, d, N = 4, 128, sum(q_lens)
    ctx_lens = [a + b for a, b in zip(q_lens, old)]
    need = [(n + block - 1) // block for n in ctx_lens]
    pages = torch.randperm(sum(need) + 2, generator=g).tolist()
    tables = [[pages.pop() for _ in range(n)] + [-1] * (max(need) - n) for n in need]
    slots = (sum(need) + 2) * block
    q, k, v = (torch.randn(n, w * d, generator=g).bfloat16() for n, w in ((N, H), (slots, G), (slots, G)))
    for b, n in enumerate(ctx_lens):                       # rows behind a context hold anything
        if n % block:
            at = tables[b][n // block] * block
            k[at + n % block:at + block] = float("nan")
            v[at + n % block:at + block] = float("nan")
    cu = [0]
    for n in q_lens:
        cu.append(cu[-1] + n)
    s = torch.randn(H, generator=g).to(DEV) if sink else None
    z = torch.randn(N, H * d + 8, generator=g).to(DEV)[:, :H * d] if gate else None
    run = lambda dt: ops.attn_paged_wide(ctx, q.to(DEV, dt), k.to(DEV, dt), v.to(DEV, dt), i32(tables), i32(ctx_lens), i32(cu), max(q_lens), block, H, G, d, d,  # noqa: E731
                                         d ** -0.5, window=window, sink=s, gate=z, out_scale=scale).float()
    got, want = run(torch.bfloat16), run(torch.float32)
    assert torch.isfinite(got).all()
    assert float((got - want).abs().max()) <= 2e-2 * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("N", [13, 600])                     # tokens of few heads: a warp per head up to 512 rows
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,d,vd,rot,half,norm", [(16, 8, 128, 128, 64, False, "weight"), (3, 1, 64, 64, 64, True, "weight"), (5, 2, 68, 124, 24, True, "unit"),
                                                    (4, 2, 8, 60, 4, False, None), (1, 1, 128, 4, 128, True, "unit"), (7, 7, 100, 100, 0, False, "weight")])
def test_preparation_of_heads_in_registers(ctx, ops, dt, H, G, d, vd, rot, half, norm, N):
    g = torch.Generator().manual_seed(H * d + vd)
    eps, pad, rows = 1e-5, 4, N + 7
    qw, kw, vw = H * d, G * d, G * vd
    x, bias, first = torch.randn(N, pad + qw + kw + vw, generator=g), torch.randn(pad + qw + kw + vw, generator=g), torch.randn(N, vw, generator=g)
    qn, kn = ((1 + 0.3 * torch.randn(d, generator=g)).to(DEV) for _ in range(2)) if norm == "weight" else (None, None)
    pos = torch.randint(0, 300, (N,), generator=g)
    slots = torch.randperm(rows, generator=g)[:N].to(torch.int32)
    slots[3] = -1
    lam = torch.tensor([0.3], device=DEV)
    q, kc, vc = torch.zeros(N, qw, dtype=dt, device=DEV), torch.full((rows, kw), 9.0, dtype=dt, device=DEV), torch.full((rows, vw), 9.0, dtype=dt, device=DEV)
    ops.qkv_prep(ctx, x.to(DEV), pad, pad + qw, pad + qw + kw, H, G, d, vd, q, kc, vc, bias=bias.to(DEV), q_norm=qn, k_norm=kn, eps=eps, rot_dims=rot, rot_half=half,
                 rot_table=ops.rotary_table(ctx, 5000.0, rot, 300) if rot else None, positions=i32(pos.tolist()), k_scale=0.5, blend=2, lam=lam, v_first=first.to(DEV),
                 slot_mapping=slots.to(DEV), v_scale=1.5, unit_norm=norm == "unit")
    xb = (x + bias).double()[:, pad:]

    def heads(t, n, w):
        y = t.reshape(N, n, d)
        if norm:
            y = y / torch.sqrt((y * y).mean(-1, keepdim=True) + eps) * (1.0 if w is None else w.cpu().double())
        if rot:
            a = pos.double()[:, None, None] * 5000.0 ** (-2.0 * torch.arange(rot // 2).double() / rot)
            y = y.clone()
            u, z = (y[..., :rot // 2].clone(), y[..., rot // 2:rot].clone()) if half else (y[..., 0:rot:2].clone(), y[..., 1:rot:2].clone())
            r = (u * a.cos() - z * a.sin(), z * a.cos() + u * a.sin())
            if half:
                y[..., :rot // 2], y[..., rot // 2:rot] = r
            else:
                y[..., 0:rot:2], y[..., 1:rot:2] = r
        return y.reshape(N, n * d)
    tol = 1e-5 if dt == torch.float32 else 2.0 ** -8
    ok = slots >= 0
    at = slots[ok].long()
    v = 1.5 * (0.7 * xb[:, qw + kw:] + 0.3 * first.double())
    for got, want in ((q.cpu(), heads(xb[:, :qw], H, qn)), (kc.cpu()[at], 0.5 * heads(xb[:, qw:qw + kw], G, kn)[ok]), (vc.cpu()[at], v[ok])):
        assert ((got.double() - want).abs() <= tol * (1 + want.abs())).all()
    rest = torch.ones(rows, dtype=torch.bool)
    rest[at] = False
    assert (kc.cpu()[rest] == 9).all() and (vc.cpu()[rest] == 9).all()


@pytest.mark.parametrize("gate", [False, True])
@pytest.mark.parametrize("B", [64, 65])                     # up to 64 sequences the q tiles that exist are listed; several items per CTA, every length of a last tile
def test_ragged_batches_of_many_portions(ctx, ops, B, gate):
    g = torch.Generator().manual_seed(B)
    H, G, d, block, window = 8, 2, 128, 64, 200
    q_lens = [(1 + 37 * i * i) % 450 + (i % 5 == 0) for i in range(B)]
    N, need = sum(q_lens), [max(1, (n + block - 1) // block) for n in q_lens]
    pages = torch.randperm(sum(need), generator=g).tolist()
    tables = [[pages.pop() for _ in range(n)] + [-1] * (max(need) - n) for n in need]
    q, k, v = (torch.randn(n, w * d, generator=g).bfloat16() for n, w in ((N, H), (sum(need) * block, G), (sum(need) * block, G)))
    cu = [0]
    for n in q_lens:
        cu.append(cu[-1] + n)
    z = torch.randn(N, H * d, generator=g).to(DEV) if gate else None
    run = lambda dt: ops.attn_paged_wide(ctx, q.to(DEV, dt), k.to(DEV, dt), v.to(DEV, dt), i32(tables), i32(q_lens), i32(cu), max(q_lens), block, H, G, d, d,  # noqa: E731
                                         d ** -0.5, window=window, gate=z).float()
    got, want = run(torch.bfloat16), run(torch.float32)
    assert torch.isfinite(got).all()
    assert float((got - want).abs().max()) <= 2e-2 * max(1.0, float(want.abs().max()))
