"""Generates tests/golden/*.json from the fp32 oracle (TEST INFRASTRUCTURE).

    python -m oracle.make_goldens [--model qwen3-0.6b] [--prompt-seeds 1 2 3 ...]

The golden workload: Qwen3-0.6B shapes, synthetic checkpoint seed 0, ONE sequence, 32-token
prompt (uniform ids, seed = prompt seed), 64 greedy tokens, ignore_eos, run with the
reference's algorithm (full recompute every step, all-position logits, host argmax with the
last-maximum tie rule).  For every step the top-2 logit gap is recorded: greedy identity
between a bf16 path and the fp32 reference is only meaningful on prompts whose minimum gap is
well above the bf16 path's logit error.  The first prompt
seed whose minimum gap is >= --min-gap becomes the asserted fixture; the others are recorded
with their gaps.
"""
from __future__ import annotations

import argparse
import json
import os
import time

import numpy as np
import torch

from .engine_oracle import (BlockManager, LLMEngine, OracleModelRunner, SamplingParams, Scheduler, SchedulerConfig,
                            Sequence)
from .qwen3_oracle import MODEL_CONFIGS, Qwen3Oracle
from .synth import make_prompts, make_weights

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


class _GapRunner(OracleModelRunner):
    def __init__(self, model, eos):
        super().__init__(model, eos)
        self.gaps, self.top = [], []

    def run(self, seqs, is_prefill):
        toks = super().run(seqs, is_prefill)
        for lg in self.last_logits:
            v, i = torch.topk(lg, 8)
            self.gaps.append(float(v[0] - v[1]))
            self.top.append((i.tolist(), [float(x) for x in v]))
        return toks


def generate(model, cfg, prompt, max_tokens):
    Sequence._counter = 0
    runner = _GapRunner(model, cfg.eos_token_id)
    sch = Scheduler(SchedulerConfig(max_num_seqs=1, max_num_batched_tokens=4096, eos=cfg.eos_token_id,
                                    num_kvcache_blocks=16, kvcache_block_size=256), BlockManager(16, 256))
    eng = LLMEngine(sch, runner)
    out = eng.generate([prompt], SamplingParams(1.0, max_tokens, True))
    return out[0][1], runner


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--model", default="qwen3-0.6b")
    ap.add_argument("--weight-seed", type=int, default=0)
    ap.add_argument("--prompt-seeds", type=int, nargs="+", default=[1, 2, 3, 4])
    ap.add_argument("--prompt-len", type=int, default=32)
    ap.add_argument("--max-tokens", type=int, default=64)
    ap.add_argument("--min-gap", type=float, default=0.05)
    ap.add_argument("--norm-jitter", type=float, default=0.0)
    ap.add_argument("--out", default=None)
    a = ap.parse_args()
    cfg = MODEL_CONFIGS[a.model]
    torch.manual_seed(0)
    t0 = time.time()
    w = {k: v.float() for k, v in make_weights(cfg, a.weight_seed, norm_jitter=a.norm_jitter).items()}
    fp32 = Qwen3Oracle(cfg, w, "fp32")
    bf16 = Qwen3Oracle(cfg, w, "bf16")
    print(f"weights ready in {time.time() - t0:.1f}s", flush=True)
    cases, chosen = [], None
    for ps in a.prompt_seeds:
        prompt = make_prompts(1, a.prompt_len, cfg.vocab_size, ps)[0]
        t0 = time.time()
        toks32, r32 = generate(fp32, cfg, prompt, a.max_tokens)
        t32 = time.time() - t0
        toks16, r16 = generate(bf16, cfg, prompt, a.max_tokens)
        agree = next((i for i, (x, y) in enumerate(zip(toks32, toks16)) if x != y), len(toks32))
        case = dict(prompt_seed=ps, prompt=prompt, tokens_fp32=toks32, tokens_bf16_mode=toks16,
                    gaps_fp32=r32.gaps, min_gap_fp32=min(r32.gaps), first_disagreement_bf16_mode=agree,
                    top8_step0=dict(idx=r32.top[0][0], val=r32.top[0][1]),
                    top8_last=dict(idx=r32.top[-1][0], val=r32.top[-1][1]),
                    cpu_seconds_fp32=t32, cpu_threads=torch.get_num_threads())
        cases.append(case)
        print(f"prompt seed {ps}: min gap {case['min_gap_fp32']:.4f}, bf16-mode agrees for {agree}/{len(toks32)} tokens, "
              f"{t32:.1f}s on {torch.get_num_threads()} threads", flush=True)
        if chosen is None and case["min_gap_fp32"] >= a.min_gap:
            chosen = ps
            if len(cases) >= 2:
                break
    out = a.out or os.path.join(ROOT, "tests", "golden", f"{a.model}_cfg0.json")
    os.makedirs(os.path.dirname(out), exist_ok=True)
    with open(out, "w") as f:
        json.dump(dict(model=a.model, weight_seed=a.weight_seed, norm_jitter=a.norm_jitter, prompt_len=a.prompt_len,
                       max_tokens=a.max_tokens, min_gap_required=a.min_gap, asserted_prompt_seed=chosen, cases=cases,
                       generator="python -m oracle.make_goldens", oracle="oracle/qwen3_oracle.py (fp32, full recompute)"),
                  f, indent=1)
    print("wrote", out, "asserted seed:", chosen)


if __name__ == "__main__":
    main()
