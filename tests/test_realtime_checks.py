"""What a real-time frame refuses before anything is launched (CPU: the launches
and the device checks are replaced, so a call that passes its checks shows)."""
import pytest
import torch

N_CELLS = 64


class Launched(Exception):
    pass


@pytest.fixture
def model(monkeypatch):
    from diver_gb300 import _native as N
    from diver_gb300.realtime import RealtimeModel

    def call(name, *args):
        raise Launched(name)

    monkeypatch.setattr(N, "need_cuda", lambda name, t, dtype=None: None)
    monkeypatch.setattr(N, "stream", lambda device=None: 0)
    monkeypatch.setattr(N, "call", call)
    z = torch.zeros
    m = RealtimeModel(z(8, 32), z(N_CELLS + 1, 1, 1, dtype=torch.int32), z((N_CELLS,) * 3, dtype=torch.bool),
                      z(1 + 64 + 4096, dtype=torch.bool), z(8), 32, N_CELLS, -1.0, 2.0 / N_CELLS)
    m._tc_blob = m.tc_err = z(1)  # made already
    return m


EYE = torch.tensor([0.0, 0.0, 4.0])


@pytest.mark.parametrize("shape", [(4, 5, 3), (5, 2), (5, 1), (6,), (3,), (5, 4), (3, 5)])
def test_frame_refuses_directions_of_another_shape(model, shape):
    """Directions that do not hold one (x, y, z) per ray: reading three floats a
    ray would leave the buffer, or render the first rays only."""
    with pytest.raises(ValueError, match="dirs"):
        model.render_frame(EYE, torch.ones(shape))


@pytest.mark.parametrize("shape", [(5, 3), (1, 3), (5, 1, 3)])
def test_frame_takes_one_direction_per_ray(model, shape):
    with pytest.raises(Launched, match="dv_realtime_begin"):
        model.render_frame(EYE, torch.ones(shape))


@pytest.mark.parametrize("rounds", [0, 1, 2.0, 2.5, 1e9, float("inf"), torch.tensor(3), -1, True])
def test_frame_takes_any_number_of_rounds(model, rounds):
    """max_rounds is compared with the rounds done, so any number will do."""
    with pytest.raises(Launched, match="dv_realtime_begin"):
        model.render_frame(EYE, torch.ones(5, 3), max_rounds=rounds)


@pytest.mark.parametrize("mode", ["tc", "fused", "loop"])
@pytest.mark.parametrize("eye,shape", [((3,), (5, 2)), ((3,), (6,)), ((2,), (5, 3)), ((0,), (5, 3))])
def test_no_mode_reads_past_its_inputs(model, mode, eye, shape):
    """A camera centre or directions with less than the kernels read, in any mode."""
    with pytest.raises(ValueError, match="eye|dirs|v must"):
        model.render_frame(torch.ones(eye), torch.ones(shape), mode=mode)


def test_one_launch_frame_refuses_short_types(model):
    with pytest.raises(ValueError, match="dirs"):
        model.render_frame(EYE, torch.ones(5, 3, dtype=torch.float16), mode="fused")


@pytest.mark.parametrize("shape", [(5, 3), (4, 5, 3), (5, 1, 3)])  # (rays in the first dimension)
def test_one_launch_frame_takes_what_it_took(model, shape):
    with pytest.raises(Launched, match="dv_realtime_frame"):
        model.render_frame(EYE, torch.ones(shape), mode="fused")
