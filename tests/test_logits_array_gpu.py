"""Arrays for logits: page-locked between 64 KiB and 32 MiB, plain outside, and always the caller's own."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(1, 7), (1, 16384), (3, 32768), (64, 131072), (65, 131073)])
def test_logits_arrays_are_the_callers_own(ctx, rows, cols):
    engine = importlib.import_module("nano-vllm-candle_b200.engine")
    torch.zeros(1, device="cuda:0")
    a, b = engine._logits_array(rows, cols), engine._logits_array(rows, cols)
    for x in (a, b):
        assert x.shape == (rows, cols) and x.dtype == np.float32 and x.flags.c_contiguous and x.flags.writeable
        assert torch.from_numpy(x).is_pinned() == ((1 << 16) <= rows * cols * 4 <= (1 << 25))
    assert not np.shares_memory(a, b)
    a[:], b[:] = 1.0, 2.0
    assert a[0, 0] == 1.0 and a[-1, -1] == 1.0


def test_a_default_device_does_not_matter(ctx):
    engine = importlib.import_module("nano-vllm-candle_b200.engine")
    torch.zeros(1, device="cuda:0")
    with torch.device("cuda:0"):
        x = engine._logits_array(1, 16384)
    assert x.shape == (1, 16384) and torch.from_numpy(x).is_pinned()


def test_arrays_that_are_kept_are_page_locked_up_to_four(ctx):
    engine = importlib.import_module("nano-vllm-candle_b200.engine")
    torch.zeros(1, device="cuda:0")
    kept = [engine._logits_array(1, 16384) for _ in range(7)]
    assert [torch.from_numpy(x).is_pinned() for x in kept] == [True] * 4 + [False] * 3
    row = kept[0][0]                          # a view keeps its array, and the array its place
    del kept[:2]
    x = engine._logits_array(1, 16384)
    assert torch.from_numpy(x).is_pinned() and not torch.from_numpy(engine._logits_array(1, 16384)).is_pinned()
    del row
    assert torch.from_numpy(engine._logits_array(1, 16384)).is_pinned()
