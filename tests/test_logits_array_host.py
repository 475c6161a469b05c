"""Arrays for logits where page-locked memory cannot be had: plain ones, and nothing is lost for later."""
import importlib

import numpy as np
import torch

engine = importlib.import_module("nano-vllm-candle_b200.engine")


def test_plain_memory_without_a_gpu():
    assert engine._logits_array(2, 16384).shape == (2, 16384)


def test_plain_memory_where_no_page_locked_memory_is_left(monkeypatch):
    def empty(*shape, **kw):
        assert kw["device"] == "cpu" and kw["pin_memory"]
        raise RuntimeError("CUDA error: out of memory")
    monkeypatch.setattr(torch.cuda, "is_initialized", lambda: True)
    monkeypatch.setattr(torch, "empty", empty)
    before = len(engine._pinned_permits)
    for _ in range(10):
        x = engine._logits_array(2, 16384)
        assert x.shape == (2, 16384) and x.dtype == np.float32 and x.flags.writeable
    assert len(engine._pinned_permits) == before


def test_at_most_four_page_locked_arrays_at_a_time(monkeypatch):
    made = []

    class Tensor:
        def __init__(self, shape, **kw):
            made.append(shape)
            self.memory = np.zeros(shape, dtype=np.float32)
            self.__array_interface__ = self.memory.__array_interface__

        def numpy(self):
            return np.asarray(self)           # the array holds on to the tensor, as a real one does
    monkeypatch.setattr(torch.cuda, "is_initialized", lambda: True)
    monkeypatch.setattr(torch, "empty", Tensor)
    kept = [engine._logits_array(2, 16384) for _ in range(9)]
    assert len(made) == 4
    row = kept[1][0]
    del kept[:2]
    kept.append(engine._logits_array(2, 16384))
    kept.append(engine._logits_array(2, 16384))
    assert len(made) == 5                     # the second one's row is still held
    del row, kept
    assert len(engine._pinned_permits) == 4
