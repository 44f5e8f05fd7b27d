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


def test_last_write_is_not_copied():
    """A field's copy (copy.deepcopy) holds no event of the original's."""
    import copy
    import pickle

    w = N.LastWrite()
    w.event = object()
    assert copy.deepcopy(w).event is None and pickle.loads(pickle.dumps(w)).event is None
