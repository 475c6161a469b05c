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
