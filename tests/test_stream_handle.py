"""The stream handle that launches go to: of a CUDA device only, so that a call
given host tensors stops there and no kernel gets their addresses (CPU: the
runtime's two calls are replaced)."""
import pytest
import torch

from diver_gb300 import _native as N


@pytest.fixture(autouse=True)
def runtime(monkeypatch):
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda index: 100 + index)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 7)


@pytest.mark.parametrize("device", ["cpu", torch.device("cpu"), torch.device("meta")])
def test_a_host_device_has_no_stream(device):
    with pytest.raises(ValueError, match="cuda device"):
        N.stream(device)


@pytest.mark.parametrize("device,handle", [(None, 107), (2, 102), ("cuda", 107), ("cuda:3", 103),
                                           (torch.device("cuda"), 107), (torch.device("cuda", 1), 101)])
def test_stream_of_a_cuda_device(device, handle):
    assert N.stream(device) == handle


def test_device_rays_refuse_a_host_device(monkeypatch):
    """dv_camera_rays writes where it is told: host buffers never reach it."""
    from diver_gb300 import scenes

    def call(name, *args):
        raise AssertionError(f"{name} launched on host memory")

    monkeypatch.setattr(N, "call", call)
    with pytest.raises(ValueError, match="cuda device"):
        scenes.camera_rays_device(torch.eye(3, 4), 4, 4, 5.0, device="cpu")


class FakeStream:
    """A stream that logs what it waits for."""

    def __init__(self, handle, log):
        self.cuda_stream, self.log = handle, log

    def wait_event(self, event):
        self.log.append((self.cuda_stream, event.number))

    def wait_stream(self, other):
        self.log.append((self.cuda_stream, other))


@pytest.fixture
def cuda(monkeypatch):
    """Streams, events and captures of a device: .on(handle) makes a stream current."""

    class Cuda:
        log, events, capturing = [], 0, False

        def on(self, handle):
            self.current = FakeStream(handle, self.log)
            return self.current

    c = Cuda()
    c.log = []

    class Event:
        def __init__(self):
            c.events += 1
            self.number = c.events

        def record(self, stream):
            pass

    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: c.current)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: c.capturing)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda index: c.current.cuda_stream)
    return c


DEV = torch.device("cuda", 0)


def test_each_stream_waits_for_a_write_once(cuda):
    w = N.LastWrite()
    cuda.on(10)
    w.wait(DEV)  # nothing written
    w.done(DEV)
    w.wait(DEV)  # the writing stream itself
    for h in (11, 12, 11, 10, 12):
        cuda.on(h)
        w.wait(DEV)
    assert cuda.log == [(11, 1), (12, 1)]
    cuda.on(11)
    w.done(DEV)  # the next write: everyone else waits again
    for h in (10, 11, 12, 10):
        cuda.on(h)
        w.wait(DEV)
    assert cuda.log[2:] == [(10, 2), (12, 2)]


def test_join_covers_the_write_on_the_side_stream_only(cuda):
    w, v = N.LastWrite(), N.LastWrite()
    side, main = cuda.on(21), FakeStream(20, cuda.log)
    w.done(DEV)
    cuda.on(22)
    v.done(DEV)  # on a third stream: waiting for the side stream says nothing about it
    for x in (w, v):
        x.join(main, side)
    cuda.current = main
    cuda.log.clear()
    w.wait(DEV)
    v.wait(DEV)
    assert cuda.log == [(20, 2)]


def test_a_write_during_a_join_is_not_covered(cuda):
    """Another thread's refresh, on the side stream and after the wait for it."""
    w = N.LastWrite()
    side = cuda.on(21)
    w.done(DEV)

    class Main(FakeStream):
        def wait_stream(self, other):
            cuda.current = side
            w.done(DEV)

    main = Main(20, cuda.log)
    w.join(main, side)
    cuda.current = main
    w.wait(DEV)
    assert cuda.log == [(20, 2)]


def test_the_per_thread_stream_always_waits(cuda):
    w = N.LastWrite()
    cuda.on(2)
    w.done(DEV)
    w.wait(DEV)
    w.wait(DEV)
    w.join(cuda.on(2), FakeStream(2, cuda.log))
    w.wait(DEV)
    assert [x for x in cuda.log if x == (2, 1)] == [(2, 1)] * 3


def test_nothing_crosses_a_capture(cuda):
    w = N.LastWrite()
    cuda.on(10)
    w.done(DEV)
    cuda.on(11)
    cuda.capturing = True
    w.wait(DEV)
    w.done(DEV)
    assert cuda.log == [] and cuda.events == 1
    cuda.capturing = False
    w.wait(DEV)
    assert cuda.log == [(11, 1)]


def test_last_write_is_not_copied():
    """A field's copy (copy.deepcopy) holds no event of the original's."""
    import copy
    import pickle

    w = N.LastWrite()
    w.state = (object(), {1})
    assert copy.deepcopy(w).state == pickle.loads(pickle.dumps(w)).state == (None, set())
