"""Work areas of the stage executor and the streams that use them, with stand-ins for buffers, events and streams."""
import pytest
import torch

from diloco_swarm_b200.models.stage_exec import KEEP_AREA_BYTES, SavedArea, StageExec


class Stream:
    def __init__(self):
        self.waited = []

    def wait_event(self, event):
        self.waited.append(event)

    def wait_stream(self, other):
        self.waited.append(other)


class Event:
    def record(self, stream):
        self.on = stream


class Buffer:
    def __init__(self, nbytes):
        self.nbytes, self.recorded = nbytes, []

    def numel(self):
        return self.nbytes

    def record_stream(self, stream):
        self.recorded.append(stream)


@pytest.fixture
def executor(monkeypatch):
    monkeypatch.setattr(torch.cuda, "Event", Event)
    ex = StageExec.__new__(StageExec)
    ex.side, ex._idle, ex._alloc, ex.capturing = Stream(), [], Buffer, False
    return ex


def test_an_area_is_recorded_on_every_stream_but_its_own(executor):
    """Taken by a pass on another stream than the one it was allocated on, an area is dropped when a pass of another
    size comes: the allocator must not hand it out again on the first stream before the second is done with it."""
    a, b = Stream(), Stream()
    size = KEEP_AREA_BYTES - 100
    area = executor.take(size, a)
    executor.give(area, a)
    assert executor.take(size, a) is area and area.buf.recorded == []
    executor.give(area, a)
    assert executor.take(size, b) is area and a in b.waited and b in area.buf.recorded
    executor.give(area, b)
    other = executor.take(200, a)                      # another size, no room for both: the area is dropped, b still runs
    assert other is not area and executor._idle == [] and set(area.buf.recorded) == {b}


def test_a_backward_on_another_stream_is_recorded(executor):
    a, b = Stream(), Stream()
    area = executor.take(100, a)
    executor.give(area, b)
    assert area.buf.recorded == [b] and isinstance(area, SavedArea)


def test_a_capture_has_areas_of_its_own(executor, monkeypatch):
    """Under a capture of the caller's no kept area is used, none is kept, and no event from outside is waited for."""
    executor._scratch, a = {}, Stream()
    a.cuda_stream = 1
    area = executor.take(100, a)
    executor.give(area, a)
    scratch = executor.area("scratch", 100, a)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: a)
    assert executor.enter() is a
    mine = executor.take(100, a)
    assert mine is not area and executor.area("scratch", 100, a) is not scratch and a.waited == []
    executor.give(mine, a)
    assert executor._idle == [area] and list(executor._scratch.values()) == [scratch] and mine.free is None


def test_sizes_that_alternate_keep_their_areas(executor):
    """As many as fit: the areas of one microbatch size are not given back because another one comes."""
    a = Stream()
    first = {}
    for n in (100, 200, 100, 200):
        area = executor.take(n, a)
        assert area is first.setdefault(n, area)
        executor.give(area, a)
    large = executor.take(KEEP_AREA_BYTES, a)            # larger than all that may lie idle: the others go
    executor.give(large, a)
    assert executor._idle == [large]
    executor.give(executor.take(100, a), a)              # and it goes when another size comes
    assert [x.buf.numel() for x in executor._idle] == [100]


def test_a_pass_is_not_counted_on_top_of_its_launches(executor, monkeypatch):
    """The executor counts the kernels that it launches; the calls that queue them are no launches themselves."""
    from diloco_swarm_b200.models import stage_exec
    from diloco_swarm_b200.ops import _lib
    monkeypatch.setattr(stage_exec, "ptr", lambda t: None)
    executor.handle, executor.d, executor._sizes = 1, 64, {}

    class Library:
        def __getattr__(self, name):
            return lambda *a: 0
    executor.lib = Library()
    stream, t = Stream(), torch.zeros(1, dtype=torch.long)
    stream.cuda_stream = 1
    before = _lib.LAUNCHES
    executor.sizes(2, 3, True, True, 1)
    executor.forward(t, None, t, None, None, 2, 3, True, stream)
    executor.head(t, t, t, None, 1.0, t, 2, 3, True, True, 1, stream)
    executor.backward(1, 0, None, None, t, t, t, None, 2, 3, 1, stream)
    assert _lib.LAUNCHES == before
