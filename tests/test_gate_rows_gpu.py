"""Output stage of a mixer in groups of columns, and the units of a feed-forward layer: widths around the lanes' shares, grids under and over the point where a warp takes several units, and
rows whose last units end inside a warp, against 64-bit arithmetic.  Bounds: a mean of up to 1 028 squares, a root, an exponential and three products
in 32 bits stay below 3e-6 relative; bf16 results add their rounding, 2^-8."""
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
ops = importlib.import_module("nano-vllm-candle_b200.ops")


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,groups,size", [
    (3, 3, 4), (3167, 3, 4), (5, 3, 60), (3161, 3, 64), (1, 1, 68), (3163, 3, 128), (9473, 1, 124), (7, 3, 132), (4741, 2, 256), (3, 5, 260),
    (343, 3, 512), (341, 3, 512), (411, 10, 516), (1367, 3, 1024), (5, 3, 1024), (2, 2, 1028)])
def test_gate_rows(ctx, rows, groups, size, dt):
    g = torch.Generator(device=DEV).manual_seed(rows + size)
    W = groups * size
    o, z = (torch.randn(rows, W + 4, generator=g, device=DEV) for _ in range(2))
    o, z = o[:, 4:] * 3, z[:, :W]
    w = 1 + 0.2 * torch.randn(W, generator=g, device=DEV)
    o64, z64, w64 = o.double().view(rows, groups, size), z.double().view(rows, groups, size), w.double().view(groups, size)
    norm = lambda x: x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-6)  # noqa: E731
    silu, sig = z64 * torch.sigmoid(z64), torch.sigmoid(z64)
    head = lambda gate, n, act, s: ops.head_gate_w(ctx, o, gate, w[:size].contiguous(), groups, size, n, 1e-6, act, s, out_dtype=dt)  # noqa: E731
    for got, want in [
        (head(z, True, "silu", 0.6), norm(o64) * w64[0] * silu * 0.6),
        (head(z, False, "sigmoid", 1.0), o64 * w64[0] * sig),
        (head(None, True, "silu", 1.0), norm(o64) * w64[0]),
        (ops.group_norm_gate(ctx, o, z, w, groups, size, True, 1e-6, "silu", out_dtype=dt), norm(o64 * silu) * w64),
        (ops.group_norm_gate(ctx, o, z, w, groups, size, False, 1e-6, "sigmoid", out_dtype=dt), norm(o64) * w64 * sig),
        (ops.group_norm_gate(ctx, o, None, None, groups, size, False, 1e-6, "silu", out_dtype=dt), norm(o64)),
    ]:
        err = ((got.double().view(want.shape) - want).abs() / (want.abs() + 1e-6)).max()
        assert float(err) <= 3e-6 + (2 ** -8 if dt == torch.bfloat16 else 0), float(err)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,F", [(4736, 8), (4737, 24), (4739, 264), (4738, 1536), (4741, 2056), (9001, 768), (2371, 100), (2369, 256), (2367, 256)])
@pytest.mark.parametrize("kind", [1, 2, 3, 4, 5])
def test_units_of_many_rows(ctx, rows, F, kind, dt):
    """Four rows per CTA: the numbers of one row per CTA, the last rows included, and a neighbour's buffer untouched."""
    g = torch.Generator(device=DEV).manual_seed(rows + F)
    x = (torch.randn(rows, 2 * F, generator=g, device=DEV) * 2).to(dt)
    act = lambda t: ops.act_mul_p(ctx, t, F, F, kind, 3.0, 1.7)  # noqa: E731
    got = act(x)
    for lo, n in ((0, 9), (rows // 2, 5), (rows - 7, 7)):
        assert torch.equal(got[lo:lo + n], act(x[lo:lo + n]))
    a, b = x[:, :F].double(), x[:, F:].double()
    if kind == 5:
        want = a * torch.sigmoid(a) * b
        assert float(((got.double() - want).abs() / (want.abs() + 1e-6)).max()) <= 3e-6 + (2 ** -8 if dt == torch.bfloat16 else 0)
    if kind == 1:
        want = torch.relu(a).square()
        assert float(((got.double() - want).abs() / (want + 1e-6)).max()) <= 1e-6 + (2 ** -8 if dt == torch.bfloat16 else 0)
        ops.check(ctx.l.nvc_act_mul(ctx.h, x.data_ptr(), 2 * F, x.data_ptr(), 2 * F, 0 if dt == torch.bfloat16 else 1, rows, F, F, kind,
                                    torch.cuda.current_stream().cuda_stream), "nvc_act_mul", ctx.h)
        assert torch.equal(x[:, :F], got) and torch.equal(x[:, F:].double(), b)


@pytest.mark.parametrize("kind,F,Fp", [(2, 256, 256), (2, 250, 264), (1, 256, 256), (2, 256, 128)])
@pytest.mark.parametrize("ldo", [0, 8])
def test_units_in_place(ctx, kind, F, Fp, ldo):
    """out inside in: the same numbers as out of place where every number is written by the thread that read it, an error elsewhere."""
    N, two = 200, kind == 2
    x = torch.randn(N, (Fp + F if two else F) + 8, generator=torch.Generator().manual_seed(F)).bfloat16().to(DEV)
    want = torch.empty(N, F, dtype=torch.bfloat16, device=DEV)
    call = lambda out, ld: ctx.l.nvc_act_mul(ctx.h, x.data_ptr(), x.stride(0), out.data_ptr(), ld, 0, N, F, Fp, kind, torch.cuda.current_stream().cuda_stream)  # noqa: E731
    assert call(want, F) == 0
    ok = ldo == 0 and (not two or Fp >= F)
    assert (call(x, x.stride(0) - ldo) == 0) == ok
    if ok:
        assert torch.equal(x[:, :F], want)
