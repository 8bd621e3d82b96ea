"""The second stream of a step, on the CPU with stand-ins for the runtime: where a thread's launches go inside and behind
on_side_stream(), also when something inside it fails."""
import threading

import pytest

from microllm_rocm_b200.kernels import ops

MAIN, SIDE = 100, 200


@pytest.fixture
def events(monkeypatch):
    seen = []
    monkeypatch.setattr(ops, "side_stream", lambda: SIDE)
    monkeypatch.setattr(ops, "fork", lambda side: seen.append(("fork", side, ops._stream())))
    monkeypatch.setattr(ops, "join", lambda side: seen.append(("join", side, ops._stream())))
    monkeypatch.setattr(ops, "_raw_stream", lambda device: MAIN)
    monkeypatch.setattr(ops, "_current_device", lambda: 0)
    return seen


def test_launches_go_to_the_side_stream_inside_only(events):
    with ops.on_side_stream() as side:
        assert side == SIDE and ops._stream() == SIDE
        other = []
        thread = threading.Thread(target=lambda: other.append(ops._stream()))
        thread.start()
        thread.join()
        assert other == [MAIN]                          # another thread's launches stay where they were
    assert ops._stream() == MAIN and events == [("fork", SIDE, MAIN)]


def test_a_failure_inside_is_joined_before_it_leaves(events):
    """Whoever catches it lets go of tensors that the side stream's kernels may still use, and may be capturing."""
    with pytest.raises(ValueError):
        with ops.on_side_stream():
            raise ValueError("a launcher refused")
    assert ops._stream() == MAIN and events == [("fork", SIDE, MAIN), ("join", SIDE, MAIN)]


def test_one_inside_another_returns_to_the_outer(events):
    with ops.on_side_stream():
        with ops.on_side_stream():
            assert ops._stream() == SIDE
        assert ops._stream() == SIDE
    assert ops._stream() == MAIN
