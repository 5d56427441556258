"""The block of memory a pass takes its intermediate tensors from: a stack with marks, aligned pieces, growth
after a pass that did not fit."""
import pytest
import torch

from gpullama3.java_b200.engine.workspace import Workspace


def test_pieces_are_aligned_disjoint_and_given_back_in_stack_order():
    ws = Workspace("cpu", 64 * 1024)
    a = ws.take((3, 5), torch.float32)
    b = ws.take((7,), torch.bfloat16)
    assert a.shape == (3, 5) and a.dtype == torch.float32 and b.dtype == torch.bfloat16
    assert a.data_ptr() % 256 == 0 and b.data_ptr() % 256 == 0 and b.data_ptr() >= a.data_ptr() + 60
    a.fill_(1.0)
    b.fill_(2.0)
    assert float(a.sum()) == 15.0                      # writing one piece leaves the other alone
    mark = ws.mark()
    c = ws.take((100,), torch.float32)
    ws.release(mark)
    d = ws.take((50,), torch.int32)
    assert d.data_ptr() == c.data_ptr()                # the same memory again after the release
    ws.release(0)
    with pytest.raises(ValueError):
        ws.release(10)                                 # beyond what is taken
    assert ws.overflowed == 0


def test_a_pass_that_does_not_fit_is_served_and_the_block_grows_for_the_next():
    ws = Workspace("cpu")                               # starts empty
    x = ws.take((1000,), torch.float32)
    y = ws.take((10, 10), torch.float32)
    assert x.numel() == 1000 and y.shape == (10, 10) and ws.overflowed == 2
    ws.reset()
    assert ws.capacity >= 4000 + 400
    z = ws.take((1000,), torch.float32)
    assert ws.overflowed == 2 and z.data_ptr() % 256 == 0
    ws.reset()
    big = ws.take((ws.capacity,), torch.float32)        # four times the block: from the allocator this once
    assert big.numel() == ws.capacity and ws.overflowed == 3
    assert ws.take((0, 4), torch.float32).numel() == 0


def test_spare_memory_is_handed_out_again_unless_it_is_kept():
    ws = Workspace("cpu", 64 * 1024)
    a = ws.take((100,), torch.float32)
    b = ws.spare((1000,), torch.bfloat16)
    assert b.data_ptr() >= a.data_ptr() + 400 and ws.take((10,), torch.float32).data_ptr() == b.data_ptr()
    c = ws.spare((1000,), torch.float32, keep=True)
    assert ws.take((10,), torch.float32).data_ptr() >= c.data_ptr() + 4000
    big = ws.spare((ws.capacity,), torch.float32)        # more than the block: from the allocator this once, and wanted from then on
    assert big.numel() == ws.capacity and ws.overflowed == 1
    capacity = ws.capacity
    ws.reset()
    assert ws.capacity > 4 * capacity


def _no_memory_above(limit, monkeypatch):
    empty = torch.empty

    def limited(shape, *args, **kwargs):
        n = 1
        for s in shape if isinstance(shape, (tuple, list)) else (shape,):
            n *= int(s)
        if n * empty((), dtype=kwargs.get("dtype", torch.float32)).element_size() > limit:
            raise torch.OutOfMemoryError("no memory")
        return empty(shape, *args, **kwargs)

    monkeypatch.setattr(torch, "empty", limited)


def test_without_memory_to_spare_there_is_none_and_nothing_more_is_wanted(monkeypatch):
    ws = Workspace("cpu", 64 * 1024)
    _no_memory_above(100 * 1024, monkeypatch)
    a = ws.take((100,), torch.float32)
    assert ws.spare((100 * 1024,), torch.float32) is None
    assert ws.take((10,), torch.float32).data_ptr() == a.data_ptr() + 512
    ws.reset()
    assert ws.capacity == 64 * 1024


def test_a_block_that_cannot_grow_stays_as_large_as_it_was(monkeypatch):
    ws = Workspace("cpu", 64 * 1024)
    ws.take((90 * 1024,), torch.uint8)                   # from the allocator
    _no_memory_above(100 * 1024, monkeypatch)            # (the block would be 112 KB)
    ws.reset()
    assert ws.capacity == 64 * 1024
    inside = ws.take((1000,), torch.float32)
    assert ws.overflowed == 1 and inside.numel() == 1000


def test_scratch_of_a_step_without_a_workspace(monkeypatch):
    from types import SimpleNamespace

    from gpullama3.java_b200.parts.base import StepContext

    step = SimpleNamespace(workspace=None, device=torch.device("cpu"))
    assert StepContext.scratch(step, (3, 4), torch.float32).shape == (3, 4)
    _no_memory_above(1024, monkeypatch)
    assert StepContext.scratch(step, (1024,), torch.float32) is None
