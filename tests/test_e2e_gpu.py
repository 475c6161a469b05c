"""End-to-end GPU parity: the whole hot path (runner + engine through the C ABI) against the
oracle's full-recompute fp32 forward on the same synthetic checkpoints.

Tolerances: logits max-abs <= 2e-2 and cosine >= 0.999 against the
fp32 reference; greedy tokens identical.  Token identity between a bf16 path and an fp32
reference is only decidable where the reference's top-2 logit gap exceeds the bf16 path's
logit error, so a mismatch is accepted ONLY at a step whose recorded fp32 gap is below
4x the measured max-abs logit error, and must then agree with the bf16-storage-emulating
oracle mode instead (see oracle/qwen3_oracle.py, mode="bf16")."""
import importlib
import json
import os

import numpy as np
import pytest
import torch

from oracle import engine_oracle as E
from oracle import qwen3_oracle as O
from oracle import synth
from conftest import diag

pytestmark = pytest.mark.gpu
eng = importlib.import_module("nano-vllm-candle_b200.engine")
GOLD = os.path.join(os.path.dirname(__file__), "golden")


def _oracle_last_logits(model, prompts):
    out = []
    for p in prompts:
        ids = torch.tensor([p])
        out.append(model.compute_logits(model.forward(ids))[0, -1])
    return torch.stack(out)


def _teacher_forced_check(model, prompt, got, tol, name):
    """Greedy identity up to numerical ties: feed the oracle the CUDA path's own sequence (one
    full-recompute forward, logits at every position) and require every generated token to be
    within `tol` of the oracle's maximum logit at its step.  Also verifies that incremental
    paged-KV decode equals the reference's recompute-everything semantics."""
    ids = torch.tensor([list(prompt) + list(got[:-1])])
    logits = model.compute_logits(model.forward(ids))[0]
    exact, worst = 0, 0.0
    for i, t in enumerate(got):
        row = logits[len(prompt) - 1 + i]
        deficit = float(row.max() - row[t])
        worst = max(worst, deficit)
        exact += int(O.argmax_last(row.numpy()) == t)
        assert deficit <= tol, f"{name}: step {i} token {t} is {deficit:.4f} below the oracle's best logit (tol {tol})"
    diag(f"[{name}] {exact}/{len(got)} tokens are the fp32 oracle's exact argmax; worst logit deficit {worst:.4e}")
    return exact


@pytest.fixture(scope="module")
def tiny(ctx):
    cfg = O.MODEL_CONFIGS["qwen3-tiny"]
    w = synth.make_weights(cfg, seed=0, norm_jitter=0.1)
    runner = eng.Qwen3ModelRunner.from_weights(ctx, cfg, w.items(), num_kvcache_blocks=64, kvcache_block_size=16,
                                               max_num_seqs=16, max_num_batched_tokens=2048, max_model_len=1024)
    wf = {k: v.float() for k, v in w.items()}
    yield cfg, runner, O.Qwen3Oracle(cfg, wf, "fp32"), O.Qwen3Oracle(cfg, wf, "bf16")
    runner.close()


def test_prefill_logits_within_tolerance(tiny):
    cfg, runner, fp32, bf16 = tiny
    lens = [1, 5, 16, 17, 130, 257, 64]
    prompts = [synth.make_prompts(1, n, cfg.vocab_size, 10 + n)[0] for n in lens]
    sch = eng.Scheduler(eng.SchedulerConfig(16, 2048, cfg.eos_token_id, 64, 16))
    e = eng.LLMEngine(sch, runner, greedy=True)
    for p in prompts:
        e.add_request(p, eng.SamplingParams(1.0, 2, True))
    si = e.schedule()
    assert si.is_prefill and len(si.seq_ids) == len(prompts)
    toks = runner.prefill(si.ids, si.positions, si.cu_seqlens, si.slot_mapping)
    got = torch.from_numpy(runner.last_logits(len(prompts)))
    ref = _oracle_last_logits(fp32, prompts)
    ref16 = _oracle_last_logits(bf16, prompts)
    err = (got - ref).abs().max().item()
    err16 = (got - ref16).abs().max().item()
    cos = torch.nn.functional.cosine_similarity(got, ref, dim=1).min().item()
    diag(f"[e2e tiny prefill] logits max-abs vs fp32 {err:.4e} vs bf16-mode {err16:.4e} min cosine {cos:.6f}")
    assert err <= 2e-2 and cos >= 0.999
    want = [O.argmax_last(r.numpy()) for r in ref]
    gaps = [float(torch.topk(r, 2).values.diff().abs()) for r in ref]
    for b, (t, w_, g) in enumerate(zip(toks.tolist(), want, gaps)):
        assert t == w_ or g < 4 * err, f"seq {b}: token {t} != {w_} with top-2 gap {g:.4f} (logit err {err:.4f})"
    e.post_process(toks)


def _generate_cuda(runner, cfg, prompts, max_tokens, max_num_seqs, nblocks, bs):
    sch = eng.Scheduler(eng.SchedulerConfig(max_num_seqs, 2048, cfg.eos_token_id, nblocks, bs))
    e = eng.LLMEngine(sch, runner, greedy=True)
    outs = e.generate(prompts, eng.SamplingParams(1.0, max_tokens, True))
    return [o.token_ids for o in outs], e


def _generate_oracle(model, cfg, prompts, max_tokens, max_num_seqs, nblocks, bs):
    E.Sequence._counter = 0
    runner = E.OracleModelRunner(model, cfg.eos_token_id)
    sch = E.Scheduler(E.SchedulerConfig(max_num_seqs, 2048, cfg.eos_token_id, nblocks, bs), E.BlockManager(nblocks, bs))
    e = E.LLMEngine(sch, runner, block_size=bs)
    return [t for _, t in e.generate(prompts, E.SamplingParams(1.0, max_tokens, True))]


def test_greedy_generation_matches_oracle_tiny(tiny):
    """Paged-KV decode (incremental) == the reference's full recompute, token for token; a small
    KV pool forces preemption + re-prefill on the way (scheduler.rs:188-211)."""
    cfg, runner, fp32, bf16 = tiny
    prompts = [synth.make_prompts(1, n, cfg.vocab_size, 100 + n)[0] for n in (7, 33, 16, 50)]
    got, e = _generate_cuda(runner, cfg, prompts, 40, 4, 64, 16)
    want16 = _generate_oracle(bf16, cfg, prompts, 40, 4, 64, 16)
    want32 = _generate_oracle(fp32, cfg, prompts, 40, 4, 64, 16)
    agree16 = [next((i for i, (a, b) in enumerate(zip(g, w)) if a != b), len(g)) for g, w in zip(got, want16)]
    agree32 = [next((i for i, (a, b) in enumerate(zip(g, w)) if a != b), len(g)) for g, w in zip(got, want32)]
    diag(f"[e2e tiny generate] tokens agreeing with bf16-mode oracle {agree16}, with fp32 oracle {agree32} of 40")
    assert e.decode_tokens == 4 * 39 and e.prefill_tokens >= sum(len(p) + 1 for p in prompts)
    for b, (p, g) in enumerate(zip(prompts, got)):
        _teacher_forced_check(fp32, p, g, 4e-2, f"e2e tiny generate seq {b}")


def test_greedy_generation_with_preemption_tiny(tiny):
    cfg, runner, fp32, bf16 = tiny
    prompts = [synth.make_prompts(1, n, cfg.vocab_size, 200 + n)[0] for n in (40, 33, 47, 20)]
    got, e = _generate_cuda(runner, cfg, prompts, 30, 8, 12, 16)       # 12 blocks of 16: must preempt
    assert e.prefill_tokens > sum(len(p) + 1 for p in prompts), "the small pool must have forced a re-prefill"
    for b, (p, g) in enumerate(zip(prompts, got)):
        assert len(g) == 30
        _teacher_forced_check(fp32, p, g, 4e-2, f"e2e tiny preemption seq {b}")


def test_prefix_caching_generation_matches_oracle_tiny(tiny):
    """With prefix caching on, sequences that share full KV blocks skip them in
    prefill (paged K4 reads the prefix through block_tables); every token must still be the
    oracle's full-recompute greedy choice up to numerical ties, and the cache must have hit."""
    cfg, runner, fp32, _ = tiny
    bs = 16
    base = synth.make_prompts(1, 5 * bs + 3, cfg.vocab_size, 900)[0]
    prompts = [base[:3 * bs + 5] + synth.make_prompts(1, 9, cfg.vocab_size, 901)[0],      # shares 3 blocks
               base,                                                                       # shares 3 blocks, longer
               base[:2 * bs],                                                              # exactly 2 full blocks: last one recomputed
               base + synth.make_prompts(1, 40, cfg.vocab_size, 902)[0],                   # shares 5 blocks with `base`
               synth.make_prompts(1, 21, cfg.vocab_size, 903)[0]]                          # unrelated
    sch = eng.Scheduler(eng.SchedulerConfig(2, 2048, cfg.eos_token_id, 64, bs, enable_prefix_caching=True))
    e = eng.LLMEngine(sch, runner, greedy=True)        # max_num_seqs 2: later prompts arrive when earlier ones have finished or are running
    outs = e.generate(prompts, eng.SamplingParams(1.0, 20, True))
    hit, queried = e.prefix_cache_stats()
    diag(f"[e2e tiny prefix caching] cache hits {hit} of {queried} full blocks; prefill tokens {e.prefill_tokens}")
    assert hit >= 3 + 1 + 5 - 2, "shared prefixes must have been served from the cache"
    for b, (p, o) in enumerate(zip(prompts, outs)):
        assert len(o.token_ids) == 20
        _teacher_forced_check(fp32, p, o.token_ids, 4e-2, f"e2e tiny prefix caching seq {b}")


def test_prefix_cached_prefill_logits_match_uncached(tiny):
    """The same prompt prefilled twice, the second time with its first blocks served from the
    cache: last-token logits agree with the uncached run to bf16 rounding and with the oracle
    within the logit tolerance."""
    cfg, runner, fp32, _ = tiny
    bs = 16
    prompt = synth.make_prompts(1, 4 * bs + 7, cfg.vocab_size, 950)[0]
    sch = eng.Scheduler(eng.SchedulerConfig(1, 2048, cfg.eos_token_id, 64, bs, enable_prefix_caching=True))
    e = eng.LLMEngine(sch, runner, greedy=True)
    logits = []
    for rnd in range(2):
        e.add_request(prompt, eng.SamplingParams(1.0, 1, True))
        si = e.schedule()
        assert si.is_prefill and len(si.ids) == (len(prompt) if rnd == 0 else 7)
        if rnd == 0:
            toks = runner.prefill(si.ids, si.positions, si.cu_seqlens, si.slot_mapping)
        else:
            st = runner.l.nvc_runner_prefill_paged(
                runner.handle, eng._p(si.ids), eng._p(si.positions), eng._p(si.cu_seqlens), eng._p(si.slot_mapping),
                eng._p(np.ascontiguousarray(si.block_tables)), si.block_tables.shape[1], eng._p(si.context_lens), 1,
                len(si.ids), len(si.ids), eng._p(np.empty(1, np.int32)))
            assert st == 0, runner.l.nvc_last_error(runner.ctx.h).decode()
            toks = np.asarray([0], np.int32)
        logits.append(torch.from_numpy(runner.last_logits(1))[0].clone())
        e.post_process(toks)
    ref = _oracle_last_logits(fp32, [prompt])[0]
    d01 = (logits[0] - logits[1]).abs().max().item()
    err = (logits[1] - ref).abs().max().item()
    diag(f"[e2e tiny prefix logits] cached vs uncached max-abs {d01:.4e}; cached vs fp32 oracle {err:.4e}")
    assert err <= 2e-2 and d01 <= 2e-2


def test_chunked_prefill_generation_matches_oracle_tiny(tiny):
    """Mixed steps (decode tokens through paged decode attention next to prompt chunks
    through paged prefill attention, one pass of everything else over all tokens).  Prompts longer
    than the 24-token budget are split over steps while earlier sequences keep decoding; every
    token must be the fp32 oracle's full-recompute greedy choice up to numerical ties."""
    cfg, runner, fp32, _ = tiny
    prompts = [synth.make_prompts(1, n, cfg.vocab_size, 700 + n)[0] for n in (9, 70, 33, 100, 5, 48)]
    sch = eng.Scheduler(eng.SchedulerConfig(4, 24, cfg.eos_token_id, 64, 16, enable_chunked_prefill=True))
    e = eng.LLMEngine(sch, runner, greedy=True)
    for p in prompts:
        e.add_request(p, eng.SamplingParams(1.0, 20, True))
    mixed = steps = 0
    while not e.is_finished():
        s = e.step()
        assert s.num_query_tokens <= 24
        mixed += int(s.num_decode_seqs > 0 and s.num_query_tokens > s.num_decode_seqs)
        steps += 1
    diag(f"[e2e tiny chunked prefill] {steps} steps, {mixed} of them mixed decode + prompt chunk")
    assert mixed >= 5
    for b, p in enumerate(prompts):
        got, fin = e.output_of(b)
        assert fin and len(got) == 20
        _teacher_forced_check(fp32, p, got, 4e-2, f"e2e tiny chunked prefill seq {b}")


def test_mixed_step_logits_match_whole_prompt_prefill(tiny):
    """One prompt prefilled whole (K4 varlen) and again in three chunks riding along with two
    decoding sequences (nvc_runner_step_mixed): last-token logits agree to bf16 rounding and with
    the fp32 oracle within the logit tolerance; the decode rows of the mixed step equal a
    plain decode step's logits for the same state within the same tolerance."""
    cfg, runner, fp32, _ = tiny
    bs = 16
    prompt = synth.make_prompts(1, 3 * bs + 11, cfg.vocab_size, 990)[0]
    others = [synth.make_prompts(1, n, cfg.vocab_size, 991 + n)[0] for n in (21, 40)]
    # whole-prompt reference on the CUDA path
    e0 = eng.LLMEngine(eng.Scheduler(eng.SchedulerConfig(4, 2048, cfg.eos_token_id, 64, bs)), runner, greedy=True)
    e0.add_request(prompt, eng.SamplingParams(1.0, 1, True))
    si = e0.schedule()
    runner.prefill(si.ids, si.positions, si.cu_seqlens, si.slot_mapping)
    whole = torch.from_numpy(runner.last_logits(1))[0].clone()
    # chunked, 27-token budget: two sequences prefilled first, then the long prompt arrives (25 tokens per step are left)
    e = eng.LLMEngine(eng.Scheduler(eng.SchedulerConfig(4, 27, cfg.eos_token_id, 64, bs, enable_chunked_prefill=True)), runner, greedy=True)
    for p in others:
        e.add_request(p, eng.SamplingParams(1.0, 8, True))
    gen = [list(p) for p in others]
    while True:                                                # prefill the two short prompts (27-token budget: 2 steps)
        si = e.schedule()
        toks = runner.step_mixed(si.ids, si.positions, si.cu_seqlens, si.slot_mapping, si.block_tables, si.context_lens,
                                 si.num_decode_seqs)
        for sid, t, m in zip(si.seq_ids.tolist(), toks.tolist(), si.emit.tolist()):
            if m:
                gen[sid].append(t)
        e.post_process(toks)
        if all(len(g) > len(p) for g, p in zip(gen, others)):
            break
    e.add_request(prompt, eng.SamplingParams(1.0, 1, True))
    chunks = []
    for _ in range(3):
        si = e.schedule()
        assert si.num_decode_seqs == 2 and si.seq_ids.tolist() == [0, 1, 2]
        chunks.append(int(si.cu_seqlens[3] - si.cu_seqlens[2]))
        toks = runner.step_mixed(si.ids, si.positions, si.cu_seqlens, si.slot_mapping, si.block_tables, si.context_lens,
                                 si.num_decode_seqs)
        lg = torch.from_numpy(runner.last_logits(3)).clone()
        # decode rows against the oracle's full recompute of the same sequences
        ref_dec = _oracle_last_logits(fp32, gen)
        err_dec = (lg[:2] - ref_dec).abs().max().item()
        assert err_dec <= 2e-2, f"decode rows of a mixed step: max-abs {err_dec:.4e}"
        for sid in (0, 1):
            gen[sid].append(int(toks[sid]))
        e.post_process(toks)
    assert chunks == [25, 25, 9] and si.emit.tolist() == [1, 1, 1]
    ref = _oracle_last_logits(fp32, [prompt])[0]
    d = (lg[2] - whole).abs().max().item()
    err = (lg[2] - ref).abs().max().item()
    diag(f"[e2e tiny mixed step] chunked vs whole-prompt logits max-abs {d:.4e}; chunked vs fp32 oracle {err:.4e}; "
         f"decode rows vs oracle {err_dec:.4e}")
    assert err <= 2e-2 and d <= 2e-2


def test_mixed_step_rejects_inconsistent_inputs(tiny):
    """nvc_runner_step_mixed reports bad arguments as status codes (never aborts, never guesses)."""
    cfg, runner, _, _ = tiny
    bs = 16
    e = eng.LLMEngine(eng.Scheduler(eng.SchedulerConfig(4, 64, cfg.eos_token_id, 64, bs, enable_chunked_prefill=True)), runner, greedy=True)
    e.add_request(synth.make_prompts(1, 20, cfg.vocab_size, 5)[0], eng.SamplingParams(1.0, 2, True))
    si = e.schedule()
    args = (si.ids, si.positions, si.cu_seqlens, si.slot_mapping, si.block_tables, si.context_lens)
    with pytest.raises(eng.NvcError):        # the first "decode" sequence has 20 query tokens
        runner.step_mixed(*args, 1)
    with pytest.raises(eng.NvcError):        # more decode sequences than sequences
        runner.step_mixed(*args, 2)
    bad_ctx = si.context_lens.copy(); bad_ctx[0] = 5          # context shorter than the query
    with pytest.raises(eng.NvcError):
        runner.step_mixed(si.ids, si.positions, si.cu_seqlens, si.slot_mapping, si.block_tables, bad_ctx, 0)
    toks = runner.step_mixed(*args, 0)        # the well-formed step still runs afterwards
    assert len(toks) == 1
    e.post_process(toks)


def test_on_device_sampling_is_reproducible_and_follows_the_oracle(tiny):
    """Temperature sampling on device (seeded Gumbel-max).  Same seed -> same tokens;
    every sampled token, teacher-forced through the fp32 oracle with the same Philox stream
    (seq_id, step), must be within tolerance of the oracle's best perturbed score."""
    from oracle import sampling_oracle as S
    cfg, runner, fp32, _ = tiny
    prompts = [synth.make_prompts(1, n, cfg.vocab_size, 300 + n)[0] for n in (9, 40, 17)]
    seed, T, steps = 20261104, 0.8, 12

    def run(sd):
        e = eng.LLMEngine(eng.Scheduler(eng.SchedulerConfig(4, 2048, cfg.eos_token_id, 64, 16)), runner, seed=sd)   # default: sampling
        return [o.token_ids for o in e.generate(prompts, eng.SamplingParams(T, steps, True))]

    a, b, c = run(seed), run(seed), run(seed + 1)
    assert a == b, "same seed must reproduce the same tokens"
    assert a != c, "a different seed must change the draws"
    greedy = [o.token_ids for o in eng.LLMEngine(eng.Scheduler(eng.SchedulerConfig(4, 2048, cfg.eos_token_id, 64, 16)),
                                                 runner, greedy=True).generate(prompts, eng.SamplingParams(T, steps, True))]
    assert a != greedy, "sampling at T = 0.8 over a flat random-init distribution must leave the greedy path"
    exact = total = 0
    for sid, (p, toks) in enumerate(zip(prompts, a)):
        ids = torch.tensor([list(p) + list(toks[:-1])])
        logits = fp32.compute_logits(fp32.forward(ids))[0]
        for i, t in enumerate(toks):
            row = logits[len(p) - 1 + i].numpy()
            sc = S.gumbel_scores(row, T, seed, S.stream_id(sid, i))
            # logits within 2e-2 of the oracle -> scores within 2e-2 / T, both sides
            assert sc.max() - sc[t] <= 2 * 2e-2 / T + 1e-4, f"seq {sid} step {i}: token {t} is {sc.max() - sc[t]:.4f} below the best draw"
            exact += int(S.sample(row, T, seed, S.stream_id(sid, i)) == t)
            total += 1
    diag(f"[e2e tiny sampling] {exact}/{total} sampled tokens identical to the fp32 oracle's draw")
    assert exact >= total * 0.8


def test_causality_property(tiny):
    """tests/layer_test.rs:164-202: logits of a prefix do not depend on later tokens -
    here: last-token logits of [a] equal position-0 logits of [a, b] in the oracle, and the
    CUDA path reproduces the 1-token logits."""
    cfg, runner, fp32, _ = tiny
    e = eng.LLMEngine(eng.Scheduler(eng.SchedulerConfig(4, 2048, cfg.eos_token_id, 64, 16)), runner, greedy=True)
    e.add_request([971], eng.SamplingParams(1.0, 1, True))
    si = e.schedule()
    runner.prefill(si.ids, si.positions, si.cu_seqlens, si.slot_mapping)
    got = torch.from_numpy(runner.last_logits(1))[0]
    two = fp32.compute_logits(fp32.forward(torch.tensor([[971, 11]])))[0, 0]
    assert (got - two).abs().mean().item() < 0.01


@pytest.mark.parametrize("name", ["qwen3-0.6b_cfg0.json"])
def test_config0_golden_tokens(ctx, name):
    """The golden workload (Qwen3-0.6B shapes, 1 seq, 32-token prompt, 64 greedy tokens): tokens and
    top logits committed by oracle/make_goldens.py from the fp32 full-recompute oracle."""
    path = os.path.join(GOLD, name)
    if not os.path.exists(path):
        pytest.skip("golden fixture not generated")
    g = json.load(open(path))
    cfg = O.MODEL_CONFIGS[g["model"]]
    w = synth.make_weights(cfg, g["weight_seed"], norm_jitter=g["norm_jitter"])
    runner = eng.Qwen3ModelRunner.from_weights(
        ctx, cfg, w.items(),
        num_kvcache_blocks=8, kvcache_block_size=256, max_num_seqs=4, max_num_batched_tokens=1024, max_model_len=2048)
    fp32 = O.Qwen3Oracle(cfg, {k: v.float() for k, v in w.items()}, "fp32")
    del w
    try:
        for case in g["cases"]:
            sch = eng.Scheduler(eng.SchedulerConfig(1, 4096, cfg.eos_token_id, 8, 256))
            e = eng.LLMEngine(sch, runner, greedy=True)
            e.add_request(case["prompt"], eng.SamplingParams(1.0, g["max_tokens"], True))
            si = e.schedule()
            tok0 = runner.prefill(si.ids, si.positions, si.cu_seqlens, si.slot_mapping)
            lg = runner.last_logits(1)[0]
            idx, val = case["top8_step0"]["idx"], np.asarray(case["top8_step0"]["val"], np.float32)
            err = float(np.abs(lg[idx] - val).max())
            e.post_process(tok0)
            toks = [int(tok0[0])]
            while not e.is_finished():
                e.step()
            toks, _ = e.output_of(0)
            n32 = next((i for i, (a, b) in enumerate(zip(toks, case["tokens_fp32"])) if a != b), len(toks))
            n16 = next((i for i, (a, b) in enumerate(zip(toks, case["tokens_bf16_mode"])) if a != b), len(toks))
            diag(f"[golden {g['model']} prompt seed {case['prompt_seed']}] top-8 logit max-abs err {err:.4e}; tokens equal to "
                 f"fp32 oracle for {n32}/{len(toks)}, to bf16-mode oracle for {n16}/{len(toks)}; min fp32 gap {case['min_gap_fp32']:.4f}")
            assert err <= 2e-2, "step-0 logits outside the logit tolerance"
            _teacher_forced_check(fp32, case["prompt"], toks, 4e-2, f"golden {g['model']} seed {case['prompt_seed']}")
            if n32 < len(toks):
                gap = case["gaps_fp32"][n32]
                assert gap < 4 * max(err, 5e-3), f"token {n32} differs although the fp32 top-2 gap is {gap:.4f}"
            if case["prompt_seed"] == g["asserted_prompt_seed"]:
                assert toks == case["tokens_fp32"], "greedy tokens differ from the fp32 reference on the asserted prompt"
    finally:
        runner.close()
