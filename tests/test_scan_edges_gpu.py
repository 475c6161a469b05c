"""The chunked recurrences on the tensor pipe at their edges - chunk and half-chunk lengths, channel and column counts around the tiles, more
sequences than are ordered by length - against the recurrences written out in 64 bits.  Bound: an fp32 number keeps 24 bits through the three
bf16 parts, so what is left is the rounding of fp32 sums of up to 128 + 32 terms per chunk, carried by a state whose decays sum to below 20
tokens: 2e-6 of the largest value is four times the 5e-7 of that."""
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F64 = torch.float64
LENS = {"edges": [1, 15, 16, 17, 31, 32, 33, 63, 64, 65, 97], "one": [70], "many": [5 + i % 3 for i in range(300)], "crowd": [17 + i % 3 for i in range(260)]}


@pytest.fixture(scope="module")
def ops():
    return importlib.import_module("nano-vllm-candle_b200.ops")


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def rows(lens, g, *shape):
    return torch.randn(sum(lens), *shape, generator=g).to(DEV)


def close(got, want):
    return float((got.to(F64) - want).abs().max()) <= 2e-6 * max(1.0, float(want.abs().max()))


def shapes(vdims):
    return [(d, vd, "edges") for d in (1, 20, 64, 65, 127, 128) for vd in vdims[:1]] + [(128, vd, "edges") for vd in vdims[1:]] + [(32, 16, "many"), (32, 16, "crowd"), (128, 64, "one")]


@pytest.mark.parametrize("fixed", [False, True])
@pytest.mark.parametrize("dim,vdim,which", shapes([33, 1, 63, 64, 65, 130]))
def test_decayed_scan_edges(ctx, ops, dim, vdim, which, fixed):
    lens, H, G = LENS[which], 2, 1
    g = torch.Generator().manual_seed(dim * 131 + vdim)
    B = len(lens)
    q, k, v, skip = rows(lens, g, G, dim) * dim ** -0.5, rows(lens, g, G, dim) * dim ** -0.5, rows(lens, g, H, vdim), rows(lens, g, H, vdim)
    ld = -rows(lens, g, H).abs()
    decay, sw = torch.tensor([0.0, 0.95], device=DEV), torch.tensor([0.5, -1.0], device=DEV)
    slots = torch.randperm(B, generator=g).to(torch.int32).to(DEV)
    state = torch.randn(B, H, dim, vdim, generator=g).to(DEV)
    cu = torch.tensor([0] + lens).cumsum(0)
    first = [b % 2 * 3 for b in range(B)]                    # every other sequence goes on from its state
    S0, pos = state.to(F64), i32([first[b] + t for b, n in enumerate(lens) for t in range(n)])
    o = ops.decay_scan(ctx, q.view(-1, G * dim), k.view(-1, G * dim), v.view(-1, H * vdim), state, slots, i32(cu.tolist()), pos, H, G, dim, vdim,
                       decay=decay if fixed else None, log_decay=None if fixed else ld, skip=None if fixed else skip.view(-1, H * vdim),
                       skip_w=None if fixed else sw, max_qlen=max(lens))
    keep = decay.to(F64).expand(sum(lens), H) if fixed else ld.to(F64).exp()
    for b, n in enumerate(lens):
        S = S0[slots[b]] * (first[b] > 0)
        for t in range(int(cu[b]), int(cu[b + 1])):
            S = S * keep[t][:, None, None] + k[t].to(F64).expand(H, dim)[:, :, None] * v[t].to(F64)[:, None]
            want = torch.einsum("hdv,hd->hv", S, q[t].to(F64).expand(H, dim))
            if not fixed:
                want = want + sw.to(F64)[:, None] * skip[t].to(F64)
            if n > 90 or t in (int(cu[b]), int(cu[b + 1]) - 1):
                assert close(o[t].view(H, vdim), want), (b, t)
        assert close(state[slots[b]], S), b


@pytest.mark.parametrize("dim,vdim,which", shapes([33, 1, 63, 64, 65, 130]))
def test_delta_rule_edges(ctx, ops, dim, vdim, which):
    lens, H, G, taps = LENS[which], 2, 1, 2
    g = torch.Generator().manual_seed(dim * 137 + vdim)
    B, C = len(lens), 2 * G * dim + H * vdim
    x = rows(lens, g, C + 2 * H)
    slots = torch.randperm(B, generator=g).to(torch.int32).to(DEV)
    state, cs = torch.randn(B, H, dim, vdim, generator=g).to(DEV) * 0.5, torch.randn(B, taps - 1, C, generator=g).to(DEV)
    cu = torch.tensor([0] + lens).cumsum(0)
    first = [b % 2 * 3 for b in range(B)]
    S0, pos = state.to(F64), i32([first[b] + t for b, n in enumerate(lens) for t in range(n)])
    o, q, k, v, gb = ops.delta_rule(ctx, x, (0, G * dim, 2 * G * dim, C, C + H), H, G, dim, vdim, taps, torch.randn(taps, C, generator=g).to(DEV), cs, state, slots,
                                    i32(cu.tolist()), pos, torch.zeros(H, device=DEV), torch.full((H,), -1.0, device=DEV), max_qlen=max(max(lens), 8))
    q, k, v = q.to(F64).view(-1, G, dim).expand(-1, H, dim), k.to(F64).view(-1, G, dim).expand(-1, H, dim), v.to(F64).view(-1, H, vdim)
    gb = gb.to(F64).view(-1, H, 2)
    for b, n in enumerate(lens):
        S = S0[slots[b]] * (first[b] > 0)
        for t in range(int(cu[b]), int(cu[b + 1])):
            S = S * gb[t, :, 0].exp()[:, None, None]
            u = gb[t, :, 1][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None]
            if n > 90 or t in (int(cu[b]), int(cu[b + 1]) - 1):
                assert close(o[t].view(H, vdim), torch.einsum("hdv,hd->hv", S, q[t])), (b, t)
        assert close(state[slots[b]], S), b
        assert torch.equal(cs[slots[b]][0], x[int(cu[b + 1]) - 1, :C]), b


@pytest.mark.parametrize("B,n,H,d,vd", [(65600, 5, 1, 16, 16), (1300, 9, 2, 64, 80)])
def test_decayed_scan_over_more_sequences_than_the_tensor_pipe_takes(ctx, ops, B, n, H, d, vd):
    """More sequences than a grid dimension holds, and many brief portions: one call (FMA) against the same in two (tensor pipe)."""
    g = torch.Generator(device=DEV).manual_seed(3)
    q, k, v = (torch.randn(B * n, H * w, generator=g, device=DEV) * 0.25 for w in (d, d, vd))
    ld = -torch.rand(B * n, H, generator=g, device=DEV)
    pos = torch.arange(n, device=DEV, dtype=torch.int32).repeat(B)

    def run(b0, b1):
        cu = torch.arange(0, (b1 - b0) * n + 1, n, device=DEV, dtype=torch.int32)
        state, at = torch.zeros(b1 - b0, H, d, vd, device=DEV), slice(b0 * n, b1 * n)
        o = ops.decay_scan(ctx, q[at], k[at], v[at], state, torch.arange(b1 - b0, device=DEV, dtype=torch.int32), cu, pos[at], H, H, d, vd, log_decay=ld[at], max_qlen=n)
        return o, state
    for a, x, y in zip(run(0, B), run(0, B // 2), run(B // 2, B)):
        assert close(a, torch.cat([x, y]).to(F64))


@pytest.mark.parametrize("front,behind,lens", [(5, 0, [13, 20]), (8, 3, [40]), (3, 9, [1, 1, 30]), (6, 2, [2, 1]), (5, 3, [13, 520]), (12, 0, [600]), (3, 6, [1, 1, 511])])
def test_delta_rule_leaves_rows_outside_the_sequences_alone(ctx, ops, front, behind, lens):
    """Rows in front of the first sequence and behind the last one are in the call's rows: the sequences between them come out as without them."""
    H, G, dim, vdim, taps, B = 2, 1, 64, 64, 4, len(lens)
    g = torch.Generator().manual_seed(front)
    C = 2 * G * dim + H * vdim
    x = torch.randn(front + sum(lens) + behind, C + 2 * H, generator=g).to(DEV)
    w = torch.randn(taps, C, generator=g).to(DEV)
    S, cs = torch.randn(B, H, dim, vdim, generator=g).to(DEV) * 0.5, torch.randn(B, taps - 1, C, generator=g).to(DEV)
    cu = torch.tensor([0] + lens).cumsum(0)

    def run(x, cu, pos):
        s, c = S.clone(), cs.clone()
        out = ops.delta_rule(ctx, x, (0, G * dim, 2 * G * dim, C, C + H), H, G, dim, vdim, taps, w, c, s, i32(list(range(B))), i32(cu.tolist()), i32(pos),
                             torch.zeros(H, device=DEV), torch.full((H,), -1.0, device=DEV), max_qlen=max(lens))
        return out, s, c
    pos = [b % 2 * 7 + t for b, n in enumerate(lens, 1) for t in range(n)]          # the first sequence goes on from its state
    want, s0, c0 = run(x[front:front + sum(lens)].contiguous(), cu, pos)
    got, s1, c1 = run(x, cu + front, [0] * front + pos + [0] * behind)
    for a, b in zip(got, want):
        assert torch.equal(a[front:front + sum(lens)], b)
    assert torch.equal(s0, s1) and torch.equal(c0, c1)


PORTIONS = {"few": [1, 2, 3, 7, 8, 9, 500], "one": [523], "many": [4 + i % 9 for i in range(140)]}


@pytest.mark.parametrize("H,G,dim,vdim,taps", [(2, 1, 64, 64, 4), (3, 1, 20, 132, 2), (2, 2, 128, 8, 1), (5, 5, 4, 4, 3), (4, 2, 68, 64, 4)])
@pytest.mark.parametrize("which", list(PORTIONS))
@pytest.mark.parametrize("channels", [False, True])
def test_delta_preparation_in_tiles_of_rows(ctx, ops, H, G, dim, vdim, taps, which, channels):
    """512 rows and more in one call (tiles of rows) against the portions one by one (a warp per row and head).  Both are fp32 with at most 4 taps
    and 128 squares in another order: 2e-6 of the largest value."""
    lens = PORTIONS[which] if which != "one" else [511, 523]
    B, g = len(lens), torch.Generator().manual_seed(dim + taps)
    C = 2 * G * dim + H * vdim
    ld = (C + 2 * H + 3) // 4 * 4
    x = torch.randn(sum(lens), ld, generator=g).to(DEV)
    w, cs = torch.randn(taps, C, generator=g).to(DEV), torch.randn(B, max(taps - 1, 1), C, generator=g).to(DEV)
    ca = torch.randn(sum(lens), H * dim, generator=g).to(DEV) if channels else None
    A, dt = torch.randn(H, generator=g).to(DEV), torch.randn(H * dim if channels else H, generator=g).to(DEV)
    cu = [0] + torch.tensor(lens).cumsum(0).tolist()
    pos = [b % 2 * 5 + t for b, n in enumerate(lens) for t in range(n)]

    def run(a, b):
        r = slice(cu[a], cu[b])
        out = ops.delta_rule(ctx, x[r], (0, G * dim, 2 * G * dim, C, C + H), H, G, dim, vdim, taps, w, cs.clone(), torch.zeros(B, H, dim, vdim, device=DEV),
                             i32(list(range(a, b))), i32([c - cu[a] for c in cu[a:b + 1]]), i32(pos[r]), A, dt, max_qlen=max(lens), channel_a=ca[r].contiguous() if channels else None)
        return out[1:]                                   # q, k, v and (log decay, beta)
    parts = [run(b, b + 1) for b in range(B)] if which != "one" else [run(0, 1)]
    whole = run(0, B)
    for i, got in enumerate(whole):
        want = torch.cat([p[i] for p in parts]).to(F64)
        if i == 3 and channels:                          # the decay per head is not written then
            got, want = got[:, 1::2], want[:, 1::2]
        assert close(got[:want.shape[0]], want), i


@pytest.mark.parametrize("H,vdim,Gs,state,taps", [(3, 64, 1, 64, 4), (2, 4, 1, 12, 2), (5, 132, 1, 20, 3), (34, 16, 2, 8, 1)])
@pytest.mark.parametrize("lens", [[700, 330], [9 + i % 2 for i in range(230)], [1, 1023, 1100]])
def test_state_space_preparation_in_tiles_of_rows(ctx, ops, H, vdim, Gs, state, taps, lens):
    """Rows enough for tiles against the same in calls that are not, each portion cut from its neighbours: fp32 sums of 4 taps, 2e-6."""
    g = torch.Generator().manual_seed(H + vdim)
    B, C = len(lens), H * vdim + 2 * Gs * state
    x = torch.randn(sum(lens), (C + H + 3) // 4 * 4, generator=g).to(DEV)
    w, bias = torch.randn(taps, C, generator=g).to(DEV), torch.randn(C, generator=g).to(DEV)
    cs = torch.randn(B, max(taps - 1, 1), C, generator=g).to(DEV)
    A, dt = torch.randn(H, generator=g).to(DEV), torch.randn(H, generator=g).to(DEV)
    cu = [0] + torch.tensor(lens).cumsum(0).tolist()
    pos = [b % 2 * 5 + t for b, n in enumerate(lens) for t in range(n)]

    def run(a, b, step):
        st, out = cs.clone(), []
        for r0 in range(cu[a], cu[b], step):
            r1 = min(r0 + step, cu[b])
            sel = [k for k in range(a, b) if cu[k] < r1 and cu[k + 1] > r0]
            out.append(ops.ssd_prep(ctx, x[r0:r1], 0, C, H, vdim, Gs, state, taps, w, bias, st, i32(sel), i32([max(cu[k], r0) - r0 for k in sel] + [r1 - r0]), i32(pos[r0:r1]), A, dt))
        return [torch.cat(t) for t in zip(*out)] + [st]
    for got, want in zip(run(0, B, 1 << 20), run(0, B, 400)):
        assert close(got, want.to(F64))


@pytest.mark.parametrize("dim,vdim,n", [(128, 64, 250), (64, 33, 33), (20, 130, 97)])
def test_scans_over_rows_and_columns_of_any_size(ctx, ops, dim, vdim, n):
    """Rows and state columns are scaled to fp16's range one by one: queries, keys and values of sizes from 1e-12 to 1e12, rows of zeros among them, give the
    result of the same numbers at size 1, times their sizes.  Powers of two, so that the scaling itself is exact: the results agree bit by bit."""
    H, G = 2, 1
    g = torch.Generator().manual_seed(dim)
    q, k, v = rows([n], g, G, dim) * dim ** -0.5, rows([n], g, G, dim) * dim ** -0.5, rows([n], g, H, vdim)
    k[n // 2] = 0.0
    q[n // 3] = 0.0
    ld = -rows([n], g, H).abs()
    sq = 2.0 ** torch.randint(-40, 41, (n, 1, 1), generator=g).to(DEV)
    sv = 2.0 ** torch.randint(-40, 41, (1, 1, vdim), generator=g).to(DEV)
    state = torch.randn(1, H, dim, vdim, generator=g).to(DEV)
    cu, pos, slot = i32([0, n]), i32(list(range(3, 3 + n))), i32([0])

    def run(q, v, state, sk=1.0):
        state = state.clone()
        o = ops.decay_scan(ctx, (q * 1.0).view(-1, G * dim), (k * sk).view(-1, G * dim), (v / sk).reshape(-1, H * vdim), state, slot, cu, pos, H, G, dim, vdim,
                           log_decay=ld, max_qlen=n)
        return o.view(n, H, vdim), state
    o0, s0 = run(q, v, state)
    o1, s1 = run(q * sq, v * sv, state * sv)
    assert torch.equal(o1, o0 * sq * sv) and torch.equal(s1, s0 * sv)
    o2, s2 = run(q, v, state, sk=2.0 ** 37)
    assert torch.equal(o2, o0) and torch.equal(s2, s0)


def spread(dim, e, g):
    """2^a per channel, a between -e and e in any order"""
    return (2.0 ** (torch.rand(dim, generator=g) * 2 * e - e)).to(DEV)


def off(got, want, dims):
    """the largest relative error of the vectors along `dims`"""
    return float(((got.to(F64) - want).norm(dim=dims) / want.norm(dim=dims)).max())


# Channels far apart in size inside one row: queries are large where keys, and so the state's rows, are small, and every channel has its share of a result.  Each
# channel of the state and each token's outputs have to come out with the error of fp32 sums, as above but of its own size and not of its neighbours': 2e-6.
@pytest.mark.parametrize("fixed", [False, True])
@pytest.mark.parametrize("e", [0, 11, 20])
@pytest.mark.parametrize("dim,vdim", [(128, 64), (64, 64), (100, 33)])
def test_decayed_scan_over_channels_far_apart(ctx, ops, dim, vdim, e, fixed):
    n, H, G = 77, 2, 1
    g = torch.Generator().manual_seed(dim + e)
    f = spread(dim, e, g)
    q, k, v = rows([n], g, G, dim) * dim ** -0.5 * f, rows([n], g, G, dim) * dim ** -0.5 / f, rows([n], g, H, vdim)
    ld, decay = -rows([n], g, H).abs() * 0.1, torch.tensor([0.9, 0.99], device=DEV)
    state = torch.randn(1, H, dim, vdim, generator=g).to(DEV) / f[:, None]
    S = state[0].to(F64)
    o = ops.decay_scan(ctx, q.view(-1, G * dim), k.view(-1, G * dim), v.view(-1, H * vdim), state, i32([0]), i32([0, n]), i32(list(range(3, 3 + n))), H, G, dim, vdim,
                       decay=decay if fixed else None, log_decay=None if fixed else ld, max_qlen=n)
    keep, want = decay.to(F64).expand(n, H) if fixed else ld.to(F64).exp(), []
    for t in range(n):
        S = S * keep[t][:, None, None] + k[t].to(F64).expand(H, dim)[:, :, None] * v[t].to(F64)[:, None]
        want.append(torch.einsum("hdv,hd->hv", S, q[t].to(F64).expand(H, dim)))
    assert off(state[0], S, -1) <= 2e-6
    assert off(o.view(n, H, vdim), torch.stack(want), -1) <= 2e-6


@pytest.mark.parametrize("e", [0, 11, 20])
@pytest.mark.parametrize("dim,vdim", [(128, 64), (64, 64), (100, 33)])
def test_delta_rule_over_channels_far_apart(ctx, ops, dim, vdim, e):
    n, H, G, taps = 77, 2, 1, 2
    g = torch.Generator().manual_seed(dim + e)
    C = 2 * G * dim + H * vdim
    f = spread(dim, e, g)
    w = torch.randn(taps, C, generator=g).to(DEV)
    w[:, :dim] *= f
    w[:, dim:2 * dim] /= f
    state = torch.randn(1, H, dim, vdim, generator=g).to(DEV) / f[:, None] * float(f.min())
    S = state[0].to(F64)
    o, q, k, v, gb = ops.delta_rule(ctx, rows([n], g, C + 2 * H), (0, G * dim, 2 * G * dim, C, C + H), H, G, dim, vdim, taps, w, torch.zeros(1, taps - 1, C, device=DEV),
                                    state, i32([0]), i32([0, n]), i32(list(range(3, 3 + n))), torch.full((H,), -2.0, device=DEV), torch.full((H,), -1.0, device=DEV),
                                    max_qlen=n)
    q, k, v = q.to(F64).view(-1, G, dim).expand(-1, H, dim), k.to(F64).view(-1, G, dim).expand(-1, H, dim), v.to(F64).view(-1, H, vdim)
    gb, want = gb.to(F64).view(-1, H, 2), []
    for t in range(n):
        S = S * gb[t, :, 0].exp()[:, None, None]
        u = gb[t, :, 1][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None]
        want.append(torch.einsum("hdv,hd->hv", S, q[t]))
    assert off(state[0], S, -1) <= 2e-6
    assert off(o.view(n, H, vdim), torch.stack(want), -1) <= 2e-6
