"""Scratch by name: tensors of one name and type share memory, the tensor objects are their callers' own, and a buffer that
grows takes every shape of its name along."""
import pytest
import torch

from test_engine_host_logic import build
from zlm_b200 import StepEntry
from zlm_b200.parts.base import Workspace

CHANGES = ["squeeze_(0)", "unsqueeze_(0)", "t_()", "requires_grad_()", "resize_(3)", "set_(torch.zeros(2))"]


@pytest.mark.parametrize("change", CHANGES)
def test_what_is_done_to_a_tensor_stays_with_its_holder(change):
    ws = Workspace("cpu")
    first, other = ws.get("a", (1, 7), torch.float32), ws.get("a", (1, 7), torch.float32)
    at = first.data_ptr()
    eval("first." + change, {"first": first, "torch": torch})
    for t in (other, ws.get("a", (1, 7), torch.float32)):
        assert t.shape == (1, 7) and t.is_contiguous() and not t.requires_grad and t.data_ptr() == at


@pytest.mark.parametrize("change", CHANGES)
def test_what_is_done_to_a_steps_logits_does_not_reach_the_next_step(change):
    eng, cfg, _ = build("A")
    s = eng.new_sequence()
    eng.step([StepEntry(s, [1], [0])])
    want = eng.step([StepEntry(s, [2], [0])]).clone()
    eng.release(s)
    s = eng.new_sequence()
    logits = eng.step([StepEntry(s, [1], [0])])
    eval("logits." + change, {"logits": logits, "torch": torch})
    assert torch.equal(eng.step([StepEntry(s, [2], [0])]), want)


def test_a_buffer_that_grows_takes_all_shapes_of_its_name_along():
    ws = Workspace("cpu")
    ws.get("a", (4,), torch.float32)
    moved = ws.generation
    big = ws.get("a", (100,), torch.float32)
    assert ws.generation == moved + 1
    small = ws.get("a", (4,), torch.float32)
    assert small.data_ptr() == big.data_ptr() and ws.generation == moved + 1
    small.fill_(5.0)
    assert big[:4].tolist() == [5.0] * 4


def test_types_and_shapes_of_one_name():
    ws = Workspace("cpu")
    a, b = ws.get("a", (2, 6), torch.float32), ws.get("a", (3, 4), torch.float32)
    c = ws.get("a", (2, 6), torch.int32)
    assert a.data_ptr() == b.data_ptr() != c.data_ptr()
    assert (a.shape, b.shape, c.dtype) == ((2, 6), (3, 4), torch.int32)
    assert ws.get("b", (2, 6), torch.float32).data_ptr() != a.data_ptr()


def test_more_shapes_than_are_kept():
    ws = Workspace("cpu")
    at = ws.get("a", (3000,), torch.float32).data_ptr()
    moved = ws.generation
    for n in range(1, 2100):
        t = ws.get("a", (n,), torch.float32)
        assert t.shape == (n,) and t.data_ptr() == at
    assert ws.generation == moved and len(ws._views) <= 1024
