"""What the step function leaves under way when it returns: steps from several streams, and the word of a kernel that gave up."""
from types import SimpleNamespace

import pytest
import torch

from fakes import fake_blocks
from sharpinference_b200.cache import CacheManager
from sharpinference_b200.engine.step import StepEntry, StepRunner
from sharpinference_b200.models.model import ScheduleEntry
from sharpinference_b200.parts.base import CacheSpec, StateSpec


class FakeStream:
    """A stream as a list of what was launched on it."""
    def __init__(self):
        self.work = []

    def wait_stream(self, other):
        self.work.append(("behind", other, len(other.work)))


def host_runner(monkeypatch, forward):
    """A runner whose cache goes by (fake) streams, without a device."""
    blocks = fake_blocks([CacheSpec("full", 0, 1, 8)])
    blocks[0].mixer.state_spec = StateSpec((3,), torch.float32)
    cache = CacheManager([ScheduleEntry(0)], blocks, page_size=4, num_pages=16, max_requests=4, dtype=torch.float32, device="cpu")
    runner = StepRunner(SimpleNamespace(vocab_size=100, blocks=blocks, forward=forward), cache)
    runner.use_graphs = False
    cache.ordered = True
    here = SimpleNamespace(stream=None)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: here.stream)
    return runner, cache, here


def test_work_from_another_stream_goes_behind_the_work_before_it(monkeypatch):
    """Steps and the clearing of a new request's states, on alternating streams: whatever comes from another stream than the work
    before it waits for that work's end, and work of one stream waits for nothing."""
    def forward(ctx):
        here.stream.work.append("step")
    runner, cache, here = host_runner(monkeypatch, forward)
    a, b = FakeStream(), FakeStream()
    here.stream = a
    cache.add_request("x")
    runner.run([StepEntry("x", [1, 2, 3], [])])
    assert a.work == ["step"]
    here.stream = b
    runner.run([StepEntry("x", [4], [0])])
    runner.run([StepEntry("x", [5], [0])])
    assert b.work == [("behind", a, 1), "step", "step"]
    here.stream = a
    cache.add_request("y")
    assert a.work[1:] == [("behind", b, 3)]
    runner.run([StepEntry("y", [1], [])])
    here.stream = b
    runner.run([StepEntry("x", [6], [])])
    assert b.work[3:] == [("behind", a, 3), "step"]


def test_a_step_that_raised_is_waited_for_too(monkeypatch):
    def forward(ctx):
        here.stream.work.append("part of a step")
        raise RuntimeError("in the middle of the step")
    runner, cache, here = host_runner(monkeypatch, forward)
    a, b = FakeStream(), FakeStream()
    here.stream = a
    cache.add_request("x")
    with pytest.raises(RuntimeError, match="in the middle"):
        runner.run([StepEntry("x", [1], [])])
    here.stream = b
    cache.add_request("y")
    assert b.work == [("behind", a, 1)]
