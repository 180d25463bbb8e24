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


class Word:
    """The device word, its copies to the host (made when the step before them ends) and the events behind them."""
    def __init__(self, monkeypatch, runner):
        self.now, self.under_way, self.waits = torch.zeros(1, dtype=torch.int32), [], 0
        runner.device = torch.device("cuda")
        runner.build_context = lambda entries: SimpleNamespace(extras={})
        runner._status_host = torch.zeros(runner.STEPS_AHEAD + 1, dtype=torch.int32)
        runner._status_events = [self.Event(self) for _ in range(runner.STEPS_AHEAD + 1)]
        self.runner = runner
        monkeypatch.setattr("sharpinference_b200.engine.step.ops.status_word", lambda device: self.now)
        monkeypatch.setattr("sharpinference_b200.engine.step.ops.check_status", self.check)
        monkeypatch.setattr(torch.cuda, "synchronize", lambda device=None: self.end_steps())

    class Event:
        def __init__(self, word):
            self.word, self.ended = word, True

        def record(self, stream=None):
            self.ended = False
            self.word.under_way.append(self)

        def query(self):
            return self.ended

        def synchronize(self):
            self.word.waits += not self.ended
            self.word.end_steps(self)

    def end_steps(self, upto=None):
        while self.under_way:
            event = self.under_way.pop(0)
            event.ended = True
            if event is upto:
                return

    def check(self, device):
        if int(self.now):
            self.now.zero_()
            raise RuntimeError("gave up")


def status_runner(monkeypatch):
    runner, cache, here = host_runner(monkeypatch, lambda ctx: None)
    here.stream = FakeStream()
    word = Word(monkeypatch, runner)
    cache.add_request("x")
    return runner, word, lambda: runner.run([StepEntry("x", [1], [])])


def test_one_step_runs_ahead_of_the_status_and_no_more(monkeypatch):
    runner, word, step = status_runner(monkeypatch)
    step()
    step()                                               # beside the first
    assert word.waits == 0 and len(word.under_way) == 2
    step()                                               # waits for the first
    assert word.waits == 1 and len(word.under_way) == 2
    word.end_steps()
    step()
    step()
    assert word.waits == 1 and len(runner._status_pending) == 2
    runner.flush_status()
    assert word.waits == 3 and not runner._status_pending and not word.under_way
    runner.flush_status()


@pytest.mark.parametrize("ended", [True, False])
def test_a_kernel_that_gave_up_raises_at_the_next_step_or_the_one_after(monkeypatch, ended):
    """A step that has ended (its result was read) raises before anything of the next one runs; one that is under way then, as soon
    as the step after that begins.  Behind the error both places are free and no old word is read."""
    runner, word, step = status_runner(monkeypatch)
    step()
    runner._status_host[runner._status_pending[0]] = word.now[0] = 3
    if ended:
        word.end_steps()
    else:
        step()
    run = runner.steps_run
    with pytest.raises(RuntimeError, match="gave up"):
        step()
    assert runner.steps_run == run and not runner._status_pending
    for _ in range(4):
        step()
    runner.flush_status()


def test_the_word_is_reset_behind_a_step_on_another_stream(monkeypatch):
    """The status that raises is read on the stream of whoever flushes: behind the steps on others."""
    runner, word, step = status_runner(monkeypatch)
    step()
    runner._status_host[runner._status_pending[0]] = word.now[0] = 3
    first = runner.cache._last_stream
    other = FakeStream()
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: other)
    with pytest.raises(RuntimeError, match="gave up"):
        runner.flush_status()
    assert other.work == [("behind", first, 0)]


def test_a_flush_or_a_reset_leaves_no_old_word_behind(monkeypatch):
    runner, word, step = status_runner(monkeypatch)
    step()
    step()
    runner._status_host[runner._status_pending[1]] = word.now[0] = 3
    with pytest.raises(RuntimeError, match="gave up"):
        runner.flush_status()
    assert not runner._status_pending
    step()
    runner._status_host[runner._status_pending[0]] = word.now[0] = 3
    runner.reset_after_failure()
    assert int(word.now) == 0 and not runner._status_pending
    for _ in range(4):
        step()
    runner.flush_status()
