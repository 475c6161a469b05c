"""Performance cases: the work that a serving process has this framework do, block by block, through the public entry points
(`ops`, and the step runner of `engine` for the whole call).

A case names a block ("kind"), its sizes and its number of tokens; every block exists for prompts (many tokens of several sequences, ragged
lengths) and for a decode step (one token per sequence on top of a paged cache or a recurrent state).  Layer sizes are those of the
Qwen3 configurations and of the equal-size family comparison (`bench.py --compare-families`).  Decode blocks of the dense layers are
captured in a CUDA graph once, as the step executor does it: what a pass costs is then the replay of the kernels and not the Python
calls.  Weights differ from layer to layer, so that a pass streams them from memory as a model's step does."""
import importlib
import math

import numpy as np
import torch

ops = importlib.import_module("nano-vllm-candle_b200.ops")
engine = importlib.import_module("nano-vllm-candle_b200.engine")

DEV = "cuda:0"
BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
EPS = 1e-6


# ------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the feed-forward half of eight layers of the 0.6B model in a decode step of 64 sequences: small products whose weights are new
        {"name": "mlp decode 64", "kind": "mlp", "tokens": 64, "width": 1024, "ff": 3072, "layers": 8, "captured": True},
        # the feed-forward half of one 8B layer over a prompt batch of odd length: the largest products
        {"name": "mlp prefill 3977", "kind": "mlp", "tokens": 3977, "width": 4096, "ff": 12288, "layers": 1, "captured": False},
        # the attention half of two 8B layers in a decode step: norm, projection, rotation, cache store, paged attention, output
        {"name": "attention decode 64", "kind": "attention", "decode": True, "seqs": 64, "short": 200, "long": 1500, "width": 4096,
         "heads": 32, "kv_heads": 8, "layers": 2, "block": 256, "captured": True},
        # the attention half of a 0.6B layer over prompts of mixed lengths
        {"name": "attention prefill 16", "kind": "attention", "decode": False, "seqs": 16, "short": 90, "long": 1100, "width": 1024,
         "heads": 16, "kv_heads": 8, "layers": 1, "block": 256, "captured": False},
        # the end of a decode step: last norm, vocabulary product, greedy choice
        {"name": "head 64", "kind": "head", "tokens": 64, "width": 1024, "vocab": 151936, "sampled": False},
        # whole decode steps of a small model through the step runner, host inputs to host logits
        {"name": "runner decode 8", "kind": "runner", "prefill": False, "seqs": 8, "short": 60, "long": 400, "layers": 4, "vocab": 32768},
        # routed experts behind a mixer, prompt batch and decode step
        {"name": "experts prefill 4000", "kind": "experts", "tokens": 4000, "width": 1024, "ff": 1536, "experts": 16, "top": 2, "captured": False},
        {"name": "experts decode 64", "kind": "experts", "tokens": 64, "width": 1024, "ff": 1536, "experts": 16, "top": 2, "captured": True},
        # latent attention in a decode step: one shared cache row per token for all heads
        {"name": "latent decode 64", "kind": "latent", "decode": True, "seqs": 64, "short": 200, "long": 1500, "heads": 16, "rank": 96,
         "rot": 32, "q_rank": 512, "window": 0, "sink": True, "block": 64, "captured": True},
        # window attention with head norms, rotation, sink and gate over prompts
        {"name": "window prefill 8", "kind": "window", "decode": False, "seqs": 8, "short": 200, "long": 1100, "heads": 16, "kv_heads": 8,
         "dim": 128, "window": 256, "block": 64, "float32": False, "captured": False},
        # the gated delta rule over prompts: convolutions, recurrence, head norm and gate
        {"name": "delta prefill 8", "kind": "delta", "decode": False, "seqs": 8, "short": 200, "long": 1100, "heads": 16, "kv_heads": 8,
         "dim": 128, "vdim": 128, "taps": 4, "channels": False},
        # a selective state space layer over prompts: convolution, recurrence, gated norm
        {"name": "ssm prefill 8", "kind": "ssm", "decode": False, "seqs": 8, "short": 200, "long": 1100, "heads": 32, "vdim": 64,
         "groups": 2, "state": 128, "taps": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mlp", "attention", "head", "runner", "experts", "latent", "window", "delta", "ssm"])
    if kind == "mlp":
        width, ff = rng.choice([(1024, 3072), (2048, 6144), (4096, 12288)])
        if rng.random() < 0.5:
            return {"kind": kind, "tokens": _log(rng, 1, 256), "width": width, "ff": ff, "layers": {1024: 8, 2048: 4, 4096: 2}[width], "captured": True}
        return {"kind": kind, "tokens": _log(rng, 300, {1024: 16000, 2048: 8000, 4096: 3900}[width]), "width": width, "ff": ff, "layers": 1, "captured": False}
    if kind == "head":
        return {"kind": kind, "tokens": _log(rng, 1, 200), "width": 1024, "vocab": 151936, "sampled": rng.random() < 0.3}
    if kind == "runner":
        return {"kind": kind, "prefill": rng.random() < 0.4, "seqs": _log(rng, 1, 12), "short": 20, "long": _log(rng, 100, 500), "layers": 4, "vocab": 32768}
    if kind == "experts":
        decode = rng.random() < 0.5
        return {"kind": kind, "tokens": _log(rng, 4, 256) if decode else _log(rng, 500, 4000), "width": rng.choice([1024, 2048]), "ff": rng.choice([768, 1536]),
                "experts": rng.choice([8, 16, 24]), "top": rng.choice([1, 2, 3]), "captured": decode}
    decode = rng.random() < 0.5
    seqs = _log(rng, 1, 64) if decode else _log(rng, 1, 10)
    short = rng.randint(17, 200)
    long = short + _log(rng, 50, 1200 if decode else 900)
    case = {"kind": kind, "decode": decode, "seqs": seqs, "short": short, "long": long}
    if kind == "attention":
        width, heads = rng.choice([(1024, 16), (2048, 16), (4096, 32)])
        case.update(width=width, heads=heads, kv_heads=8, layers=2 if decode else 1, block=rng.choice([16, 64, 256]), captured=decode)
    elif kind == "latent":
        rank, rot = rng.choice([(96, 32), (96, 32), (64, 64), (112, 16)])
        case.update(heads=rng.choice([8, 16, 24]), rank=rank, rot=rot, q_rank=rng.choice([256, 512]), window=rng.choice([0, 0, 300]),
                    sink=rng.random() < 0.5, block=rng.choice([16, 64]), captured=decode)
        if not decode:
            case["short"], case["long"] = max(64, short), max(64, short) + long - short
    elif kind == "window":
        heads, kv = rng.choice([(16, 8), (16, 4), (8, 8)])
        case.update(heads=heads, kv_heads=kv, dim=rng.choice([128, 128, 64]), window=rng.choice([0, 128, 256, 700]), block=rng.choice([16, 64]),
                    float32=rng.random() < 0.2, captured=decode)
    elif kind == "delta":
        heads, kv = rng.choice([(16, 8), (16, 16), (8, 4)])
        case.update(heads=heads, kv_heads=kv, dim=rng.choice([128, 128, 64]), vdim=128, taps=rng.choice([2, 4]), channels=rng.random() < 0.4)
    else:
        heads, vdim = rng.choice([(32, 64), (16, 128), (64, 64)])
        case.update(heads=heads, vdim=vdim, groups=rng.choice([1, 2]), state=rng.choice([64, 128]), taps=rng.choice([2, 4]))
        if heads * vdim > 2048 and not decode:
            case["seqs"] = min(seqs, 4)
    return case


# ------------------------------------------------------------------------------------------ helpers
def _lens(case):
    """Ragged lengths between case["short"] and case["long"], the same for every seed."""
    n, lo, hi = case["seqs"], case["short"], case["long"]
    return [int(round(lo * (hi / lo) ** ((0.5 + 0.6180339887 * i) % 1.0))) for i in range(n)]


class _Rand:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed))

    def __call__(self, *shape, scale=1.0, mean=0.0, dtype=F32):
        t = torch.randn(*shape, generator=self.g, device=DEV, dtype=F32)
        return t.mul_(scale).add_(mean).to(dtype)

    def perm(self, n):
        return torch.randperm(n, generator=self.g, device=DEV)

    def ints(self, hi, n):
        return torch.randint(0, hi, (n,), generator=self.g, device=DEV, dtype=torch.int32)


def _i32(v):
    return torch.as_tensor(v, dtype=torch.int32).to(DEV)


def _layout(rand, ctx_lens, q_lens, block):
    """Paged layout of sequences with ctx_lens tokens in the cache, the last q_lens of them new: shuffled pages, slots and positions of the
    new tokens, their first rows."""
    need = [(n + block - 1) // block for n in ctx_lens]
    pages = rand.perm(sum(need)).to(torch.int32)
    tables = torch.full((len(need), max(need)), -1, dtype=torch.int32, device=DEV)
    at = 0
    for b, n in enumerate(need):
        tables[b, :n] = pages[at:at + n]
        at += n
    q = torch.tensor(q_lens, device=DEV)
    cu = torch.cat([torch.zeros(1, dtype=torch.int64, device=DEV), q.cumsum(0)])
    seq = torch.arange(len(q_lens), device=DEV).repeat_interleave(q)
    pos = torch.arange(int(sum(q_lens)), device=DEV) - cu[seq] + (torch.tensor(ctx_lens, device=DEV) - q)[seq]
    slots = tables[seq, pos // block].long() * block + pos % block
    return {"tables": tables, "context": _i32(ctx_lens), "cu": cu.to(torch.int32), "positions": pos.to(torch.int32), "slots": slots.to(torch.int32),
            "blocks": sum(need), "longest": max(q_lens), "ctx_lens": list(ctx_lens), "q_lens": list(q_lens)}


def _rows_of(layout, b, block):
    """Cache rows of sequence b, oldest first."""
    n = layout["ctx_lens"][b]
    j = torch.arange(n, device=DEV)
    return layout["tables"][b, j // block].long() * block + j % block


def _finish(state, case, fn):
    """The call of a pass: captured in a CUDA graph where the case says so."""
    state["call"] = fn
    if case.get("captured"):
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            fn()
        torch.cuda.current_stream().wait_stream(side)
        state["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state["graph"]):
            state["out"] = fn()
    return state


def run(state):
    if "graph" in state:
        state["graph"].replay()
        return state["out"]
    return state["call"]()


def _rms(x, w, eps):
    x = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return x if w is None else x * w


def _silu(x):
    return x * torch.sigmoid(x)


# ------------------------------------------------------------------------------------------ feed-forward half
def _mlp_inputs(case, seed):
    r = _Rand(seed)
    M, W, F = case["tokens"], case["width"], case["ff"]
    x, res = r(M, W, dtype=BF16), r(M, W)
    layers = [(r(W, scale=0.1, mean=1.0, dtype=BF16), r(2 * F, W, scale=W ** -0.5, dtype=BF16), r(W, F, scale=F ** -0.5, dtype=BF16)) for _ in range(case["layers"])]
    return x, res, layers


def _mlp_prepare(case, seed):
    x, res, layers = _mlp_inputs(case, seed)
    ctx = ops.Context(0)
    layers = [(n, ctx.interleave_gate_up(gu), d) for n, gu, d in layers]

    def fn():
        h, s = x, res
        for norm, gu, down in layers:
            t = torch.empty_like(s)
            a = ctx.fused_add_rmsnorm(h, norm, EPS, residual_in=s, residual_out=t)
            h, s = ctx.gemm(ctx.gemm_silu_mul(a, gu), down), t
        return {"x": h, "residual": s}
    return _finish({"ctx": ctx}, case, fn)


def _mlp_exact(case, seed):
    x, res, layers = _mlp_inputs(case, seed)
    h, s, F = x.to(F64), res.to(F64), case["ff"]
    for norm, gu, down in layers:
        s = s + h
        z = _rms(s, norm.to(F64), EPS) @ gu.to(F64).T
        h = (_silu(z[:, :F]) * z[:, F:]) @ down.to(F64).T
    return {"x": h, "residual": s}


def _mlp_work(case):
    M, W, F, L = case["tokens"], case["width"], case["ff"], case["layers"]
    return {"bytes": L * (6 * F * W + 2 * W) + M * W * (2 + 4 + 2 + 4), "flops": L * 6 * M * F * W}


# ------------------------------------------------------------------------------------------ attention half
def _attention_inputs(case, seed):
    r = _Rand(seed)
    W, nh, kv = case["width"], case["heads"], case["kv_heads"]
    lens = _lens(case)
    lay = _layout(r, lens, [1] * len(lens) if case["decode"] else lens, case["block"])
    N = sum(lay["q_lens"])
    x, res = r(N, W, dtype=BF16), r(N, W)
    layers = []
    for _ in range(case["layers"]):
        layers.append({"norm": r(W, scale=0.1, mean=1.0, dtype=BF16), "qkv": r((nh + 2 * kv) * 128, W, scale=W ** -0.5, dtype=BF16),
                       "qn": r(128, scale=0.1, mean=1.0, dtype=BF16), "kn": r(128, scale=0.1, mean=1.0, dtype=BF16),
                       "o": r(W, nh * 128, scale=(nh * 128) ** -0.5, dtype=BF16),
                       "k": r(lay["blocks"], case["block"], kv, 128, dtype=BF16), "v": r(lay["blocks"], case["block"], kv, 128, dtype=BF16)})
    return x, res, layers, lay


def _attention_prepare(case, seed):
    x, res, layers, lay = _attention_inputs(case, seed)
    ctx = ops.Context(0)
    nh, kv, scale = case["heads"], case["kv_heads"], 128 ** -0.5
    table = ctx.rope_table(1e6, 128, case["long"] + 1)

    def fn():
        h, s = x, res
        for p in layers:
            t = torch.empty_like(s)
            a = ctx.fused_add_rmsnorm(h, p["norm"], EPS, residual_in=s, residual_out=t)
            qkv = ctx.qkv_proj_norm_rope(a, p["qkv"], p["qn"], p["kn"], EPS, table, lay["positions"], nh, kv, 128, lay["slots"], p["k"], p["v"])
            q, k, v = qkv[:, :nh * 128], qkv[:, nh * 128:(nh + kv) * 128], qkv[:, (nh + kv) * 128:]
            if case["decode"]:
                o = ctx.paged_decode_attn(q, p["k"], p["v"], lay["tables"], lay["context"], nh, kv, 128, case["block"], scale)
            else:
                o = ctx.prefill_attn(q, k, v, lay["cu"], lay["longest"], nh, kv, 128, scale)
            h, s = ctx.gemm(o, p["o"]), t
        return {"x": h, "residual": s, "caches": [c for p in layers for c in (p["k"], p["v"])]}
    return _finish({"ctx": ctx}, case, fn)


def _rope64(x, pos, theta):
    """x [N, heads, 128], pairs (i, i + 64)."""
    f = theta ** (-torch.arange(64, device=DEV, dtype=F64) / 64)
    a = pos.to(F64)[:, None, None] * f
    u, w = x[..., :64], x[..., 64:]
    return torch.cat([u * a.cos() - w * a.sin(), w * a.cos() + u * a.sin()], -1)


def _attend(q, k, v, scale, first, window=0, sink=None):
    """q [T, H, d] at positions first .. of keys k [n, G, d] and values v [n, G, vd]: causal softmax attention."""
    T, H, _ = q.shape
    n, G, vd = v.shape
    s = torch.einsum("tgrd,ngd->grtn", q.view(T, G, H // G, -1), k) * scale
    i, j = first + torch.arange(T, device=DEV)[:, None], torch.arange(n, device=DEV)[None]
    hide = (j > i) | (j <= i - window if window else j < 0)
    s = s.masked_fill(hide, -math.inf)
    if sink is not None:
        s = torch.cat([s, sink.view(G, H // G, 1, 1).expand(-1, -1, T, 1)], -1)
    w = torch.softmax(s, -1)[..., :n]
    return torch.einsum("grtn,ngd->tgrd", w, v).reshape(T, H * vd)


def _attention_exact(case, seed):
    x, res, layers, lay = _attention_inputs(case, seed)
    nh, kv, bs = case["heads"], case["kv_heads"], case["block"]
    h, s, N = x.to(F64), res.to(F64), x.shape[0]
    cu = lay["cu"].tolist()
    for p in layers:
        s = s + h
        z = (_rms(s, p["norm"].to(F64), EPS) @ p["qkv"].to(F64).T).view(N, nh + 2 * kv, 128)
        q = _rope64(_rms(z[:, :nh], p["qn"].to(F64), EPS), lay["positions"], 1e6)
        k = _rope64(_rms(z[:, nh:nh + kv], p["kn"].to(F64), EPS), lay["positions"], 1e6)
        v, out = z[:, nh + kv:], []
        for b, n in enumerate(lay["ctx_lens"]):
            rows, a, e = _rows_of(lay, b, bs), cu[b], cu[b + 1]
            old = n - (e - a)
            kk = torch.cat([p["k"].view(-1, kv, 128)[rows[:old]].to(F64), k[a:e]])
            vv = torch.cat([p["v"].view(-1, kv, 128)[rows[:old]].to(F64), v[a:e]])
            out.append(_attend(q[a:e], kk, vv, 128 ** -0.5, old))
        h = torch.cat(out) @ p["o"].to(F64).T
    return {"x": h, "residual": s, "caches": None}


def _pairs(lay_q, lay_ctx, window=0):
    total = 0
    for q, c in zip(lay_q, lay_ctx):
        i = np.arange(c - q, c) + 1
        total += int(np.minimum(i, window).sum() if window else i.sum())
    return total


def _attention_work(case):
    lens = _lens(case)
    q = [1] * len(lens) if case["decode"] else lens
    N, W, nh, kv, L = sum(q), case["width"], case["heads"], case["kv_heads"], case["layers"]
    weights = 2 * W * ((nh + 2 * kv) + nh) * 128
    cache = sum(lens) * kv * 512
    return {"bytes": L * (weights + cache) + N * W * 12, "flops": L * (N * weights + 4 * 128 * nh * _pairs(q, lens))}


# ------------------------------------------------------------------------------------------ head
def _head_inputs(case, seed):
    r = _Rand(seed)
    B, W, V = case["tokens"], case["width"], case["vocab"]
    return r(B, W, dtype=BF16), r(B, W), r(W, scale=0.1, mean=1.0, dtype=BF16), r(V, W, scale=W ** -0.5, dtype=BF16), torch.rand(B, generator=r.g, device=DEV) + 0.5


def _head_prepare(case, seed):
    x, res, norm, w, temps = _head_inputs(case, seed)
    ctx = ops.Context(0)
    streams = torch.arange(x.shape[0], device=DEV, dtype=torch.int64) * 1000 + 7

    def fn():
        logits = ctx.gemm(ctx.fused_add_rmsnorm(x, norm, EPS, residual_in=res), w, out_dtype=F32)
        idx, val = ctx.sample_gumbel(logits, temps, streams, 11) if case["sampled"] else ctx.argmax_last(logits)
        return {"logits": logits, "token": idx, "score": val}
    return _finish({"ctx": ctx}, case, fn)


def _head_exact(case, seed):
    x, res, norm, w, _ = _head_inputs(case, seed)
    a = _rms(x.to(F64) + res.to(F64), norm.to(F64), EPS)
    logits = torch.cat([a @ c.to(F64).T for c in w.split(16384)], 1)
    return {"logits": logits, "token": None, "score": None if case["sampled"] else logits.max(-1).values}


def _head_work(case):
    B, W, V = case["tokens"], case["width"], case["vocab"]
    return {"bytes": 2 * V * W + 6 * B * W + 4 * B * V, "flops": 2 * B * V * W}


# ------------------------------------------------------------------------------------------ the step runner
_RUNNER = {"width": 1024, "heads": 16, "kv_heads": 8, "ff": 3072, "block": 64}


def _runner_inputs(case, seed):
    r = _Rand(seed)
    W, nh, kv, F, V = _RUNNER["width"], _RUNNER["heads"], _RUNNER["kv_heads"], _RUNNER["ff"], case["vocab"]
    w = {"model.embed_tokens.weight": r(V, W, dtype=BF16), "model.norm.weight": r(W, scale=0.1, mean=1.0, dtype=BF16),
         "lm_head.weight": r(V, W, scale=W ** -0.5, dtype=BF16)}
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        for n, rows, cols in (("self_attn.q_proj", nh * 128, W), ("self_attn.k_proj", kv * 128, W), ("self_attn.v_proj", kv * 128, W),
                              ("self_attn.o_proj", W, nh * 128), ("mlp.gate_proj", F, W), ("mlp.up_proj", F, W), ("mlp.down_proj", W, F)):
            w[p + n + ".weight"] = r(rows, cols, scale=cols ** -0.5, dtype=BF16)
        for n, size in (("input_layernorm", W), ("post_attention_layernorm", W), ("self_attn.q_norm", 128), ("self_attn.k_norm", 128)):
            w[p + n + ".weight"] = r(size, scale=0.1, mean=1.0, dtype=BF16)
    lens = _lens(case)
    ids = r.ints(V, sum(lens) + len(lens)).cpu().numpy()
    return w, lens, ids


def _runner_prepare(case, seed):
    w, lens, ids = _runner_inputs(case, seed)
    B, bs = len(lens), _RUNNER["block"]
    cfg = engine.Qwen3Config(vocab_size=case["vocab"], hidden_size=_RUNNER["width"], head_dim=128, num_hidden_layers=case["layers"],
                             num_attention_heads=_RUNNER["heads"], num_key_value_heads=_RUNNER["kv_heads"], intermediate_size=_RUNNER["ff"],
                             max_position_embeddings=4096)
    need = [n // bs + 1 for n in lens]
    tables = np.full((B, max(need)), -1, np.int32)
    at = 0
    for b, n in enumerate(need):
        tables[b, :n] = np.arange(at, at + n)[::-1]
        at += n
    ctx = ops.Context(0)
    runner = engine.Qwen3ModelRunner.from_weights(ctx, cfg, w.items(), num_kvcache_blocks=at, kvcache_block_size=bs, max_num_seqs=B,
                                                  max_num_batched_tokens=sum(lens), max_model_len=(max(lens) // bs + 1) * bs)
    cu = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    pos = np.concatenate([np.arange(n) for n in lens]).astype(np.int32)
    seq = np.repeat(np.arange(B), lens)
    slots = (tables[seq, pos // bs] * bs + pos % bs).astype(np.int32)
    prompt = (ids[:cu[-1]], pos, cu, slots)
    if case["prefill"]:
        def fn():
            tok = runner.prefill(*prompt)
            return {"token": tok, "logits": runner.last_logits(B)}
        return _finish({"runner": runner}, case, fn)
    runner.prefill(*prompt)
    p = np.array(lens, np.int32)
    step = (ids[cu[-1]:], p, (tables[np.arange(B), p // bs] * bs + p % bs).astype(np.int32), tables, p + 1)

    def fn():
        tok = runner.decode(*step)
        return {"token": tok, "logits": runner.last_logits(B)}
    return _finish({"runner": runner}, case, fn)


def _runner_exact(case, seed):
    w, lens, ids = _runner_inputs(case, seed)
    nh, kv, F = _RUNNER["heads"], _RUNNER["kv_heads"], _RUNNER["ff"]
    w = {k: v.to(F64) for k, v in w.items()}
    B, at, out = len(lens), 0, []
    for b, n in enumerate(lens):
        t = ids[at:at + n]
        at += n
        if not case["prefill"]:
            t, n = np.concatenate([t, ids[sum(lens) + b:sum(lens) + b + 1]]), n + 1
        x, pos = w["model.embed_tokens.weight"][torch.from_numpy(t).long().to(DEV)], torch.arange(n, device=DEV)
        for i in range(case["layers"]):
            g = lambda name: w[f"model.layers.{i}.{name}.weight"]  # noqa: E731
            a = _rms(x, g("input_layernorm"), EPS)
            q = _rope64(_rms((a @ g("self_attn.q_proj").T).view(n, nh, 128), g("self_attn.q_norm"), EPS), pos, 1e6)
            k = _rope64(_rms((a @ g("self_attn.k_proj").T).view(n, kv, 128), g("self_attn.k_norm"), EPS), pos, 1e6)
            x = x + _attend(q, k, (a @ g("self_attn.v_proj").T).view(n, kv, 128), 128 ** -0.5, 0) @ g("self_attn.o_proj").T
            a = _rms(x, g("post_attention_layernorm"), EPS)
            x = x + (_silu(a @ g("mlp.gate_proj").T) * (a @ g("mlp.up_proj").T)) @ g("mlp.down_proj").T
        out.append(_rms(x[-1:], w["model.norm.weight"], EPS) @ w["lm_head.weight"].T)
    return {"token": None, "logits": torch.cat(out)}


def _runner_work(case):
    lens = _lens(case)
    W, nh, kv, F, V, L = _RUNNER["width"], _RUNNER["heads"], _RUNNER["kv_heads"], _RUNNER["ff"], case["vocab"], case["layers"]
    per = W * (2 * nh + 2 * kv) * 128 + 3 * W * F
    q = lens if case["prefill"] else [1] * len(lens)
    cache = 0 if case["prefill"] else L * sum(lens) * kv * 512
    return {"bytes": 2 * (L * per + V * W) + cache + 4 * len(lens) * V,
            "flops": 2 * (sum(q) * L * per + len(lens) * V * W) + L * 4 * 128 * nh * _pairs(q, lens)}


# ------------------------------------------------------------------------------------------ routed experts
def _experts_inputs(case, seed):
    r = _Rand(seed)
    N, W, F, E = case["tokens"], case["width"], case["ff"], case["experts"]
    router = torch.zeros(64, W, dtype=BF16, device=DEV)
    router[:E] = r(E, W, scale=W ** -0.5, dtype=BF16)
    return r(N, W, dtype=BF16), router, r(E, 2 * F, W, scale=W ** -0.5, dtype=BF16), r(E, W, F, scale=F ** -0.5, dtype=BF16)


def _experts_prepare(case, seed):
    h, router, gate_up, down = _experts_inputs(case, seed)
    ctx = ops.Context(0)
    E, top, F = case["experts"], case["top"], case["ff"]
    correction = torch.zeros(E, device=DEV)

    def fn():
        z = ctx.gemm(h, router, out_dtype=F32)
        idx, w = ops.moe_route_logits_ex(ctx, z, correction, E, top, 1.0, ops.ROUTE_SOFTMAX, True)
        offsets, src, pos, groups = ops.moe_sort_padded(ctx, idx, E)
        rows = ops.gather_rows(ctx, h, src, offsets[E:])
        hid = ops.act_mul_p(ctx, ops.gemm_grouped(ctx, rows, gate_up, groups), F, F, ops.ACT_SILU_MUL)
        y = ops.gemm_grouped(ctx, hid, down, groups, out_dtype=F32)
        return {"y": ops.moe_combine(ctx, y, pos, w), "experts": idx, "weights": w}
    return _finish({"ctx": ctx}, case, fn)


def _experts_exact(case, seed):
    h, router, gate_up, down = _experts_inputs(case, seed)
    E, F = case["experts"], case["ff"]
    x = h.to(F64)
    z = x @ router[:E].to(F64).T
    w, idx = torch.topk(torch.softmax(z, -1), case["top"], -1)
    w = w / w.sum(-1, keepdim=True)
    y = torch.zeros_like(x)
    for e in range(E):
        tok, t = torch.nonzero(idx == e, as_tuple=True)
        if tok.numel():
            u = x[tok] @ gate_up[e].to(F64).T
            y.index_add_(0, tok, w[tok, t][:, None] * ((_silu(u[:, :F]) * u[:, F:]) @ down[e].to(F64).T))
    return {"y": y, "experts": None, "weights": w}


def _experts_work(case):
    N, W, F, E, top = case["tokens"], case["width"], case["ff"], case["experts"], case["top"]
    used = E * (1 - (1 - top / E) ** N)
    return {"bytes": used * 6 * F * W + 2 * E * W + 6 * N * W, "flops": 6 * N * top * F * W + 2 * N * E * W}


# ------------------------------------------------------------------------------------------ latent attention
def _latent_inputs(case, seed):
    r = _Rand(seed)
    H, D, R, qr = case["heads"], case["rank"] + case["rot"], case["rank"], case["q_rank"]
    lens = _lens(case)
    lay = _layout(r, lens, [1] * len(lens) if case["decode"] else lens, case["block"])
    N = sum(lay["q_lens"])
    return {"rows": r(N, qr + D), "w0": r(qr, scale=0.1, mean=1.0), "w1": r(R, scale=0.1, mean=1.0), "q": r(N, H, D, dtype=BF16),
            "cache": r(lay["blocks"] * case["block"], D, dtype=BF16), "sink": r(H) if case["sink"] else None}, lay


def _latent_prepare(case, seed):
    t, lay = _latent_inputs(case, seed)
    ctx = ops.Context(0)
    H, R, rot, D, qr, scale = case["heads"], case["rank"], case["rot"], case["rank"] + case["rot"], case["q_rank"], 0.7 * 128 ** -0.5
    table = ops.rotary_table(ctx, 10000.0, rot, case["long"] + 1)

    def fn():
        latent = ops.latent_norm_store_rot(ctx, t["rows"], qr, qr, R, t["w0"], t["w1"], EPS, t["cache"], lay["slots"], rot, rot, True, table,
                                           lay["positions"], BF16)
        q = t["q"].view(-1, H * D)
        if case["decode"]:
            o = ops.attn_paged_wide(ctx, q, t["cache"], t["cache"], lay["tables"], lay["context"], None, 1, case["block"], H, 1, D, R, scale,
                                    window=case["window"], sink=t["sink"])
        else:   # the value columns behind the latent are a by-product here
            o = ops.prefill_attn_shared(ctx, q, t["cache"], lay["tables"], lay["context"], lay["cu"], lay["longest"], case["block"], H, 1, scale,
                                        window=case["window"], sink=t["sink"])
        return {"latent": latent, "out": o, "cache": t["cache"]}
    return _finish({"ctx": ctx}, case, fn)


def _rotate_half(x, pos, dims, base):
    h = dims // 2
    a = pos.to(F64)[:, None] * base ** (-2.0 * torch.arange(h, device=DEV, dtype=F64) / dims)
    a = a.view(a.shape[0], *([1] * (x.dim() - 2)), h)
    u, w = x[..., :h], x[..., h:dims]
    return torch.cat([u * a.cos() - w * a.sin(), w * a.cos() + u * a.sin(), x[..., dims:]], -1)


def _latent_exact(case, seed):
    t, lay = _latent_inputs(case, seed)
    H, R, rot, D, qr, scale = case["heads"], case["rank"], case["rot"], case["rank"] + case["rot"], case["q_rank"], 0.7 * 128 ** -0.5
    rows, cache, cu = t["rows"].to(F64), t["cache"].to(F64), lay["cu"].tolist()
    new = torch.cat([_rms(rows[:, qr:qr + R], t["w1"].to(F64), EPS), _rotate_half(rows[:, qr + R:], lay["positions"], rot, 10000.0)], -1)
    cache[lay["slots"].long()] = new
    sink, out = None if t["sink"] is None else t["sink"].to(F64), []
    for b, n in enumerate(lay["ctx_lens"]):
        kk = cache[_rows_of(lay, b, case["block"])][:, None]
        out.append(_attend(t["q"][cu[b]:cu[b + 1]].to(F64), kk, kk[..., :R] if case["decode"] else kk, scale, n - lay["q_lens"][b], case["window"], sink))
    return {"latent": _rms(rows[:, :qr], t["w0"].to(F64), EPS), "out": torch.cat(out), "cache": cache}


def _seen(case, lens, q):
    w = case["window"]
    return sum(min(n, m + w - 1) if w else n for n, m in zip(lens, q))


def _latent_work(case):
    lens = _lens(case)
    q = [1] * len(lens) if case["decode"] else lens
    N, H, D, R, qr = sum(q), case["heads"], case["rank"] + case["rot"], case["rank"], case["q_rank"]
    vd = R if case["decode"] else D
    return {"bytes": N * (4 * (qr + D) + 2 * qr + 2 * D + 2 * H * (D + vd)) + 2 * D * _seen(case, lens, q),
            "flops": 2 * H * (D + vd) * _pairs(q, lens, case["window"])}


# ------------------------------------------------------------------------------------------ window attention
def _window_inputs(case, seed):
    r = _Rand(seed)
    H, G, d, dt = case["heads"], case["kv_heads"], case["dim"], F32 if case["float32"] else BF16
    lens = _lens(case)
    lay = _layout(r, lens, [1] * len(lens) if case["decode"] else lens, case["block"])
    N, cols = sum(lay["q_lens"]), (2 * H + 2 * G) * d
    return {"rows": r(N, cols), "bias": r(cols, scale=0.1), "qn": r(d, scale=0.1, mean=1.0), "kn": r(d, scale=0.1, mean=1.0),
            "k": r(lay["blocks"] * case["block"], G * d, dtype=dt), "v": r(lay["blocks"] * case["block"], G * d, dtype=dt), "sink": r(H)}, lay, dt


def _window_prepare(case, seed):
    t, lay, dt = _window_inputs(case, seed)
    ctx = ops.Context(0)
    H, G, d = case["heads"], case["kv_heads"], case["dim"]
    table = ops.rotary_table(ctx, 10000.0, 64, case["long"] + 1)
    gate = t["rows"][:, (H + 2 * G) * d:]
    cu = None if case["decode"] else lay["cu"]

    def fn():
        q = torch.empty(t["rows"].shape[0], H * d, dtype=dt, device=DEV)
        ops.qkv_prep(ctx, t["rows"], 0, H * d, (H + G) * d, H, G, d, d, q, t["k"], t["v"], bias=t["bias"], q_norm=t["qn"], k_norm=t["kn"], eps=EPS,
                     rot_dims=64, rot_table=table, positions=lay["positions"], slot_mapping=lay["slots"])
        o = ops.attn_paged_wide(ctx, q, t["k"], t["v"], lay["tables"], lay["context"], cu, lay["longest"], case["block"], H, G, d, d, d ** -0.5,
                                window=case["window"], sink=t["sink"], gate=gate)
        return {"out": o, "k": t["k"], "v": t["v"]}
    return _finish({"ctx": ctx}, case, fn)


def _rotate_pairs(x, pos, dims, base):
    a = pos.to(F64)[:, None, None] * base ** (-2.0 * torch.arange(dims // 2, device=DEV, dtype=F64) / dims)
    y, u, w = x.clone(), x[..., 0:dims:2], x[..., 1:dims:2]
    y[..., 0:dims:2], y[..., 1:dims:2] = u * a.cos() - w * a.sin(), w * a.cos() + u * a.sin()
    return y


def _window_exact(case, seed):
    t, lay, _ = _window_inputs(case, seed)
    H, G, d, N = case["heads"], case["kv_heads"], case["dim"], t["rows"].shape[0]
    x = t["rows"].to(F64) + t["bias"].to(F64)
    q = _rotate_pairs(_rms(x[:, :H * d].view(N, H, d), t["qn"].to(F64), EPS), lay["positions"], 64, 10000.0)
    k = _rotate_pairs(_rms(x[:, H * d:(H + G) * d].view(N, G, d), t["kn"].to(F64), EPS), lay["positions"], 64, 10000.0)
    kc, vc, at, cu, out = t["k"].to(F64).view(-1, G, d), t["v"].to(F64).view(-1, G, d), lay["slots"].long(), lay["cu"].tolist(), []
    kc[at], vc[at] = k, x[:, (H + G) * d:(H + 2 * G) * d].view(N, G, d)
    for b, n in enumerate(lay["ctx_lens"]):
        rows = _rows_of(lay, b, case["block"])
        out.append(_attend(q[cu[b]:cu[b + 1]], kc[rows], vc[rows], d ** -0.5, n - lay["q_lens"][b], case["window"], t["sink"].to(F64)))
    o = torch.cat(out) * torch.sigmoid(t["rows"][:, (H + 2 * G) * d:].to(F64))
    return {"out": o, "k": kc.view(-1, G * d), "v": vc.view(-1, G * d)}


def _window_work(case):
    lens = _lens(case)
    q = [1] * len(lens) if case["decode"] else lens
    N, H, G, d, e = sum(q), case["heads"], case["kv_heads"], case["dim"], 4 if case["float32"] else 2
    return {"bytes": N * (4 * (2 * H + 2 * G) * d + e * (H + 2 * G) * d) + 2 * e * G * d * _seen(case, lens, q), "flops": 4 * H * d * _pairs(q, lens, case["window"])}


# ------------------------------------------------------------------------------------------ recurrences
def _steps(case):
    """(tokens per sequence, first rows or None, positions): prompts start at position 0, decode steps go on from a state."""
    q = [1] * case["seqs"] if case["decode"] else _lens(case)
    pos = [n for n in _lens(case)] if case["decode"] else [i for n in q for i in range(n)]
    cu = None if case["decode"] else _i32(np.concatenate([[0], np.cumsum(q)]))
    return q, cu, _i32(pos)


def _delta_inputs(case, seed):
    r = _Rand(seed)
    H, G, d, vd, taps = case["heads"], case["kv_heads"], case["dim"], case["vdim"], case["taps"]
    q, cu, pos = _steps(case)
    N, B, C = sum(q), len(q), 2 * G * d + H * vd
    ch = case["channels"]
    return {"rows": r(N, C + 2 * H + H * vd), "conv": r(taps, C, scale=0.5), "conv_state": r(B, taps - 1, C), "state": r(B, H, d, vd, scale=0.1),
            "slots": r.perm(B).to(torch.int32), "A_log": r(H, scale=0.3), "dt_bias": r(H * d if ch else H, mean=-1.0),
            "channel_a": r(N, H * d) if ch else None, "norm": r(vd, scale=0.1, mean=1.0)}, q, cu, pos


def _delta_prepare(case, seed):
    t, q, cu, pos = _delta_inputs(case, seed)
    ctx = ops.Context(0)
    H, G, d, vd = case["heads"], case["kv_heads"], case["dim"], case["vdim"]
    C = 2 * G * d + H * vd
    offs, gate, longest = (0, G * d, 2 * G * d, C, C + H), t["rows"][:, C + 2 * H:], max(q)

    def fn():
        o = ops.delta_rule(ctx, t["rows"], offs, H, G, d, vd, case["taps"], t["conv"], t["conv_state"], t["state"], t["slots"], cu, pos,
                           t["A_log"], t["dt_bias"], max_qlen=longest, channel_a=t["channel_a"])[0]
        return {"out": ops.head_gate_w(ctx, o, gate, t["norm"], H, vd, True, 1e-5, "silu", 1.0, out_dtype=BF16), "state": t["state"], "conv": t["conv_state"]}
    return _finish({"ctx": ctx}, case, fn)


def _padded(rows, q):
    """[N, c] -> [B, longest, c], zeros behind a sequence's end."""
    return torch.nn.utils.rnn.pad_sequence(list(rows.split(q)), batch_first=True)


def _unpadded(rows, q):
    return torch.cat([rows[b, :n] for b, n in enumerate(q)])


def _short_conv(x, w, before, q):
    """Causal convolution of x [B, T, C] behind before [B, taps - 1, C]; also every sequence's last taps - 1 inputs."""
    taps, T = w.shape[0], x.shape[1]
    full = torch.cat([before, x], 1)
    y = sum(full[:, j:j + T] * w[j] for j in range(taps))
    return y, torch.stack([full[b, n:n + taps - 1] for b, n in enumerate(q)])


def _delta_exact(case, seed):
    t, q, _, _ = _delta_inputs(case, seed)
    H, G, d, vd, B = case["heads"], case["kv_heads"], case["dim"], case["vdim"], len(q)
    C, slots, rows = 2 * G * d + H * vd, t["slots"].long(), t["rows"].to(F64)
    before = t["conv_state"].to(F64)[slots] if case["decode"] else torch.zeros(B, case["taps"] - 1, C, dtype=F64, device=DEV)
    S = t["state"].to(F64)[slots] if case["decode"] else torch.zeros(B, H, d, vd, dtype=F64, device=DEV)
    y, conv = _short_conv(_padded(rows[:, :C], q), t["conv"].to(F64), before, q)
    y, T = _silu(y), max(q)

    def unit(x):
        return (x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 2)
    qq = unit(y[..., :G * d].view(B, T, G, d)) * d ** -0.5
    kk, vv = unit(y[..., G * d:2 * G * d].view(B, T, G, d)), y[..., 2 * G * d:].view(B, T, H, vd)
    beta = torch.sigmoid(_padded(rows[:, C:C + H], q))
    a = _padded((t["channel_a"] if case["channels"] else t["rows"][:, C + H:C + 2 * H]).to(F64), q) + t["dt_bias"].to(F64)
    rate = t["A_log"].to(F64).exp()
    g = torch.exp(-rate[:, None] * torch.nn.functional.softplus(a).view(B, T, H, d)) if case["channels"] else \
        torch.exp(-rate * torch.nn.functional.softplus(a))[..., None].expand(B, T, H, d)
    live = torch.arange(T, device=DEV)[None] < torch.tensor(q, device=DEV)[:, None]
    beta, g = beta * live[..., None], torch.where(live[..., None, None], g, torch.ones_like(g))
    out = torch.empty(B, T, H, vd, dtype=F64, device=DEV)
    for i in range(T):
        S = S * g[:, i, :, :, None]
        u = beta[:, i, :, None] * (vv[:, i] - torch.einsum("bhdv,bhd->bhv", S, kk[:, i]))
        S = S + kk[:, i, :, :, None] * u[:, :, None]
        out[:, i] = torch.einsum("bhdv,bhd->bhv", S, qq[:, i])
    o = _rms(_unpadded(out, q), t["norm"].to(F64), 1e-5).reshape(-1, H * vd) * _silu(rows[:, C + 2 * H:])
    state, cs = torch.empty_like(S), torch.empty_like(conv)
    state[slots], cs[slots] = S, conv
    return {"out": o, "state": state, "conv": cs}


def _delta_work(case):
    q, B = [1] * case["seqs"] if case["decode"] else _lens(case), case["seqs"]
    N, H, G, d, vd = sum(q), case["heads"], case["kv_heads"], case["dim"], case["vdim"]
    C = 2 * G * d + H * vd
    states = B * (H * d * vd + (case["taps"] - 1) * C) * (2 if case["decode"] else 1)
    return {"bytes": 4 * (N * (C + 2 * H + H * vd + (H * d if case["channels"] else 0)) + states) + 2 * N * H * vd, "flops": 6 * N * H * d * vd}


def _ssm_inputs(case, seed):
    r = _Rand(seed)
    H, vd, G, S, taps = case["heads"], case["vdim"], case["groups"], case["state"], case["taps"]
    q, cu, pos = _steps(case)
    N, B, inner = sum(q), len(q), H * vd
    C = inner + 2 * G * S
    return {"rows": r(N, inner + C + H), "conv": r(taps, C, scale=0.5), "conv_b": r(C, scale=0.1), "conv_state": r(B, taps - 1, C),
            "state": r(B, H, S, vd, scale=0.1), "slots": r.perm(B).to(torch.int32), "A_log": r(H, scale=0.5), "dt_bias": r(H, mean=-2.0), "D": r(H),
            "norm": r(inner, scale=0.1, mean=1.0)}, q, cu, pos


def _ssm_prepare(case, seed):
    t, q, cu, pos = _ssm_inputs(case, seed)
    ctx = ops.Context(0)
    H, vd, G, S = case["heads"], case["vdim"], case["groups"], case["state"]
    inner, longest = H * vd, max(q)
    dt_off = 2 * inner + 2 * G * S

    def fn():
        x, v, b, c, decay = ops.ssd_prep(ctx, t["rows"], inner, dt_off, H, vd, G, S, case["taps"], t["conv"], t["conv_b"], t["conv_state"], t["slots"], cu,
                                         pos, t["A_log"], t["dt_bias"])
        y = ops.decay_scan(ctx, c, b, v, t["state"], t["slots"], cu, pos, H, G, S, vd, log_decay=decay, skip=x, skip_w=t["D"], max_qlen=longest)
        o = ops.group_norm_gate(ctx, y, t["rows"][:, :inner], t["norm"], G, inner // G, True, 1e-5, "silu", out_dtype=BF16)
        return {"out": o, "state": t["state"], "conv": t["conv_state"]}
    return _finish({"ctx": ctx}, case, fn)


def _ssm_exact(case, seed):
    t, q, _, _ = _ssm_inputs(case, seed)
    H, vd, G, n, B = case["heads"], case["vdim"], case["groups"], case["state"], len(q)
    inner = H * vd
    C, slots, rows, T = inner + 2 * G * n, t["slots"].long(), t["rows"].to(F64), max(q)
    before = t["conv_state"].to(F64)[slots] if case["decode"] else torch.zeros(B, case["taps"] - 1, C, dtype=F64, device=DEV)
    S = t["state"].to(F64)[slots] if case["decode"] else torch.zeros(B, H, n, vd, dtype=F64, device=DEV)
    y, conv = _short_conv(_padded(rows[:, inner:inner + C], q), t["conv"].to(F64), before, q)
    y = _silu(y + t["conv_b"].to(F64))
    x = y[..., :inner].view(B, T, H, vd)
    bb = y[..., inner:inner + G * n].view(B, T, G, n).repeat_interleave(H // G, 2)
    cc = y[..., inner + G * n:].view(B, T, G, n).repeat_interleave(H // G, 2)
    live = torch.arange(T, device=DEV)[None] < torch.tensor(q, device=DEV)[:, None]
    dt = torch.nn.functional.softplus(_padded(rows[:, inner + C:], q) + t["dt_bias"].to(F64)) * live[..., None]
    keep = torch.exp(-t["A_log"].to(F64).exp() * dt)
    out = torch.empty(B, T, H, vd, dtype=F64, device=DEV)
    for i in range(T):
        S = S * keep[:, i, :, None, None] + bb[:, i, :, :, None] * (dt[:, i, :, None] * x[:, i])[:, :, None]
        out[:, i] = torch.einsum("bhnv,bhn->bhv", S, cc[:, i])
    o = _unpadded((out + t["D"].to(F64)[:, None] * x).reshape(B, T, inner), q) * _silu(rows[:, :inner])
    o = _rms(o.view(-1, G, inner // G), None, 1e-5).reshape(-1, inner) * t["norm"].to(F64)
    state, cs = torch.empty_like(S), torch.empty_like(conv)
    state[slots], cs[slots] = S, conv
    return {"out": o, "state": state, "conv": cs}


def _ssm_work(case):
    q, B = [1] * case["seqs"] if case["decode"] else _lens(case), case["seqs"]
    N, H, vd, G, n = sum(q), case["heads"], case["vdim"], case["groups"], case["state"]
    inner = H * vd
    C = inner + 2 * G * n
    states = B * (H * n * vd + (case["taps"] - 1) * C) * (2 if case["decode"] else 1)
    return {"bytes": 4 * (N * (inner + C + H) + states) + 2 * N * inner, "flops": 4 * N * H * n * vd}


# ------------------------------------------------------------------------------------------ the interface
def prepare(case, seed):
    return globals()[f"_{case['kind']}_prepare"](case, seed)


def work(case):
    return globals()[f"_{case['kind']}_work"](case)


def exact(case, seed):
    return globals()[f"_{case['kind']}_exact"](case, seed)


def tolerance(case):
    """About four times what one bf16 pass of a block is off its 64-bit value (0.002 - 0.005, 0.006 behind eight layers; a float32 block 4e-7);
    whole numbers (tokens, experts) only differ where two of them tie."""
    if case.get("float32"):
        return {"rel": 1e-5, "differ": 0.01}
    return {"rel": {"mlp": 2.5e-2, "attention": 2e-2, "runner": 2e-2, "experts": 1.5e-2}.get(case["kind"], 1e-2), "differ": 0.01}
