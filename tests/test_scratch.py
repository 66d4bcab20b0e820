"""Whose scratch a call gets: an engine's steps share their own, every other call has its stream's, and nobody shares with a
line of work that may run at the same time. Streams, captures and the device are stood in for here; the kernels' side is in
test_kernels_gpu.py."""
import ctypes
import sys
import threading

import pytest
import torch

from llm_b200 import ops
from llm_b200.ops import scratch


class Device:
    """A CUDA device as far as scratch is concerned: the current stream, and whether it is being captured."""

    def __init__(self, monkeypatch):
        self.local = threading.local()
        self.capturing = False
        empty, zeros = torch.empty, torch.zeros
        monkeypatch.setattr(torch, "empty", lambda n, dtype, device: empty(n, dtype=dtype))
        monkeypatch.setattr(torch, "zeros", lambda n, dtype, device: zeros(n, dtype=dtype))
        monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: self.capturing)
        monkeypatch.setattr(ops, "_stream", lambda: ctypes.c_void_p(getattr(self.local, "stream", 1)))

    def on(self, stream, floats=1 << 10, counters=16):
        self.local.stream = stream
        return ops._split_scratch(torch.device("cuda:0"), floats, counters)


@pytest.fixture
def device(monkeypatch):
    scratch._of_stream.clear()
    yield Device(monkeypatch)
    scratch._of_stream.clear()


def address(pair):
    return pair[0].data_ptr(), pair[1].data_ptr()


def test_no_two_streams_share(device):
    pairs = [device.on(stream) for stream in range(1, 20)]
    assert len({address(p) for p in pairs}) == len(pairs)
    assert len(scratch._of_stream) == scratch.STREAMS                     # what older streams held was given back
    assert address(device.on(19)) == address(pairs[-1])                   # a stream's calls share


def test_a_capture_has_its_own(device):
    eager = device.on(1)
    device.capturing = True
    captured = [device.on(1), device.on(1), device.on(0)]
    device.capturing = False
    assert len({address(p) for p in [eager] + captured}) == 4             # (and each call its own)
    assert address(device.on(1)) == address(eager)
    assert all(int(p[1].abs().sum()) == 0 for p in captured)


def test_an_engine_s_steps_have_one_on_every_stream_and_under_capture(device):
    scope, other = ops.StepScope(), ops.StepScope()
    eager = device.on(1)
    with scope:
        first = device.on(1)
        assert address(device.on(2)) == address(first)
        device.capturing = True
        assert address(device.on(3)) == address(first)
        large = device.on(3, floats=first[0].numel() + 1)                 # more than there is: the capture's own
        device.capturing = False
        assert address(large) != address(first) and address(device.on(1)) == address(first) and scope.generation == 0
        with other:
            assert address(device.on(1)) not in (address(first), address(eager))
        grown = device.on(1, floats=first[0].numel() + 1)
        assert scope.generation == 1 and address(grown) != address(first) and address(device.on(2)) == address(grown)
        assert any(held is first for held in scope._outgrown)             # captured steps still point at it
    assert address(device.on(1)) == address(eager)


def test_a_scope_holds_for_the_thread_that_entered_it(device):
    seen = []
    with ops.StepScope():
        inside = device.on(1)
        thread = threading.Thread(target=lambda: seen.append(device.on(1)))
        thread.start()
        thread.join()
    assert address(seen[0]) != address(inside)


def test_first_calls_of_many_threads(device):
    """Streams that ask for the first time while others look theirs up."""
    device.on(1)
    failures, old = [], sys.getswitchinterval()
    sys.setswitchinterval(1e-6)

    def work(base):
        try:
            for i in range(200):
                device.on(base + i % 40, floats=8, counters=1)
        except Exception as error:                                        # noqa: BLE001
            failures.append(error)
    try:
        threads = [threading.Thread(target=work, args=(100 * (t + 1),)) for t in range(6)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        sys.setswitchinterval(old)
    assert not failures and len(scratch._of_stream) <= scratch.STREAMS


def test_a_record_keeps_the_scratch_it_points_at(device):
    recording = ops.begin_recording()
    try:
        pair = device.on(5)
        ops._scratch_arguments(*pair)
    finally:
        ops.end_recording()
    for stream in range(10, 30):
        device.on(stream)
    assert any(t is pair[0] for t in recording.keep) and any(t is pair[1] for t in recording.keep)
