"""engine.Workspace.turn on a fake of torch.cuda's streams: a pass waits on its
own stream for the pass before, whatever stream that ran on, and one thread's
launches are not queued between another's."""

import threading
import types

import pytest

from gkmsvm_lite_b200 import engine


class _Stream:
    def __init__(self, name, log):
        self.name, self.log = name, log

    def wait_event(self, ev):
        self.log.append((self.name, "waits for", ev.at))


@pytest.fixture
def cuda(monkeypatch):
    log, here = [], threading.local()

    class Event:
        def record(self, stream):
            self.at = stream.name
            log.append((stream.name, "done"))

    fake = types.SimpleNamespace(Event=Event, current_stream=lambda: here.stream,
                                 is_current_stream_capturing=lambda: getattr(here, "capturing", False))
    monkeypatch.setattr(engine.torch, "cuda", fake)
    return log, here


def test_a_pass_waits_for_the_one_before(cuda):
    log, here = cuda
    w = engine.Workspace()
    for name in "aba":
        here.stream = _Stream(name, log)
        with w.turn():
            log.append((name, "pass"))
    assert log == [("a", "pass"), ("a", "done"), ("b", "waits for", "a"), ("b", "pass"), ("b", "done"),
                   ("a", "waits for", "b"), ("a", "pass"), ("a", "done")]


def test_a_pass_that_fails_is_waited_for(cuda):
    log, here = cuda
    w = engine.Workspace()
    here.stream = _Stream("a", log)
    with pytest.raises(ValueError):
        with w.turn():
            raise ValueError
    here.stream = _Stream("b", log)
    with w.turn():
        pass
    assert log == [("a", "done"), ("b", "waits for", "a"), ("b", "done")]


def test_a_capture_neither_waits_nor_records(cuda):
    log, here = cuda
    w = engine.Workspace()
    here.stream = _Stream("a", log)
    with w.turn():
        pass
    here.capturing = True
    with w.turn():
        pass
    assert log == [("a", "done")]


def test_threads_take_turns(cuda):
    log, here = cuda
    w = engine.Workspace()

    def passes(name):
        here.stream = _Stream(name, log)
        for _ in range(200):
            with w.turn():
                for _ in range(5):
                    log.append((name, "launch"))

    ts = [threading.Thread(target=passes, args=(n,)) for n in "abc"]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    launches = [e[0] for e in log if e[1] == "launch"]
    assert len(launches) == 3000
    assert all(len(set(launches[i:i + 5])) == 1 for i in range(0, 3000, 5))


def test_growth_is_bounded():
    """Requests that rise a little at a time, as a server's buckets do."""
    w = engine.Workspace()
    sizes = [1000 + 37 * k for k in range(60)]
    for n in sizes:
        assert w.get(n, "cpu").numel() == n
    assert sum(b.numel() for b in w._buffers) <= 3 * sizes[-1]
    assert len(w._buffers) <= 5
    before = len(w._buffers)
    for n in (0, 10, sizes[-1]):
        assert w.get(n, "cpu").numel() == n
    assert len(w._buffers) == before
