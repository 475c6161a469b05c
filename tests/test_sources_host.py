"""What the kernel sources must not hold: a TMA or bulk load that one CTA sends to several of its cluster.  The library runs on several GPUs too,
and such a load must never see a peer's memory."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_load_with_cluster_multicast():
    found = []
    for top in ("nano-vllm-candle_b200", "include", "tools"):
        for d, _, files in os.walk(os.path.join(ROOT, top)):
            for f in files:
                if f.endswith((".cu", ".cuh", ".h", ".hpp", ".cpp", ".py")):
                    src = open(os.path.join(d, f), encoding="utf-8").read()
                    found += [f for m in re.finditer(r"cp\.async\.bulk[\w.:]*", src) if "multicast" in m.group()]
    assert not found


# What no kernel of a step writes: weights, norm vectors, tables, positions, slots, block tables, lengths (launch order, nvc_b200.h)
STATIC = set("table w w0 w1 wy wgt weight b bias alpha qw kw cos_sin cs tab rot_table positions slot_mapping slots block_tables bt context_lens cu_seqlens W corr wr wsg wqk peers "
             "sink A_log dt_bias conv_w conv_b wp decay skip_w i_bias f_bias mix out_w in_w lambda q_norm k_norm nw norm".split())


def test_reads_of_data_that_never_changes_are_of_static_operands():
    """A load through `const T* __restrict__` or __ldg may move in front of the wait for the previous kernel, so neither stands for what a kernel writes."""
    found = []
    for f in sorted(os.listdir(os.path.join(ROOT, "nano-vllm-candle_b200", "csrc"))):
        if not f.endswith((".cu", ".cuh")):
            continue
        src = re.sub(r"//[^\n]*", "", open(os.path.join(ROOT, "nano-vllm-candle_b200", "csrc", f), encoding="utf-8").read())
        for m in re.finditer(r"__global__\b[^;{]*\{", src):
            found += [(f, p) for p in re.findall(r"const\s+[\w:]+\s*\*(?:\s*const\s*\*)?\s*__restrict__\s+(\w+)", m.group()) if p not in STATIC]
        for m in re.finditer(r"__ldg\(", src):
            base = re.match(r"(?:reinterpret_cast<[^>]*>\()?\s*(?:\w+\.)*(\w+)", src[m.end():]).group(1)
            if base not in STATIC:
                found.append((f, src[m.start():m.end() + 40]))
    assert not found, found
