"""GPU: one field or model used from several streams.  What a call keeps for the
next ones is written on the stream (or side stream) of the call that needed it
first; a call on another stream that finds it must wait for that write.  The
write is held back for about a tenth of a second by torch's bounded spin, so an
unordered reader would read what was there before."""
import pytest
import torch

pytestmark = pytest.mark.gpu
HOLD = 200_000_000  # clocks


def rays(n, seed=3):
    from diver_gb300 import scenes

    c2w = scenes.sphere_cameras(1, 4.0, seed)[0]
    o, d = scenes.camera_rays(c2w, 40, 40, 50.0, "cuda")
    return o[:n].contiguous(), d[:n].contiguous()


def small_field():
    from diver_gb300 import scenes
    from diver_gb300.renderer import DIVeRField

    return DIVeRField.from_scene(scenes.small_scene("cpu"), "cuda")


@pytest.mark.parametrize("form", ["bf16", "fp16", "bf16s"])
@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("capacity", [False, True])
def test_images_refreshed_on_another_stream(form, grad, capacity):
    """The first call after a change of the decoder refreshes its images on the
    field's side stream; a second one, on another stream and small enough to
    stay on it, decodes with the new images."""
    field, want = small_field(), small_field()
    o, d = rays(1500)
    cap = field.segment_capacity(o.shape[0]) if capacity else None
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.set_grad_enabled(grad):
        field(o, d, form=form, capacity=cap)  # images of the first decoder
        with torch.no_grad():
            for f in (field, want):
                f.params.mul_(0.5)
        ref = want(o, d, form=form, capacity=cap)[0].detach()
        torch.cuda.synchronize()
        with torch.cuda.stream(field._side_stream(field.voxels.device)):
            torch.cuda._sleep(HOLD)
        got = []
        for s in (a, b):
            with torch.cuda.stream(s):
                got.append(field(o, d, form=form, capacity=cap)[0].detach())
    torch.cuda.synchronize()
    assert torch.equal(got[0], ref) and torch.equal(got[1], ref)


@pytest.mark.parametrize("form", ["bf16", "fp16"])
def test_grid_copy_made_on_another_stream(form):
    """A render on another stream than the one that makes the 16-bit copy of the grid."""
    field, want = small_field(), small_field()
    o, d = rays(1500)
    cap = field.segment_capacity(o.shape[0])
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.no_grad():
        field(o, d, form=form, capacity=cap)
        for f in (field, want):
            f.voxels.mul_(0.5)
        ref = want(o, d, form=form, capacity=cap)[0]
        torch.cuda.synchronize()
        got = []
        for s in (a, b):
            with torch.cuda.stream(s):
                if s is a:
                    torch.cuda._sleep(HOLD)
                got.append(field(o, d, form=form, capacity=cap)[0])
    torch.cuda.synchronize()
    assert torch.equal(got[0], ref) and torch.equal(got[1], ref)


def realtime_model():
    from tests.test_realtime import small_realtime

    return small_realtime("diver32", "cuda", bias=0.2)[2]


def test_realtime_images_made_on_another_stream():
    """A frame on another stream than the one that makes the model's tensor-core images."""
    from diver_gb300 import scenes

    c2w = scenes.sphere_cameras(1, 4.0, 3)[0]
    _, v = scenes.camera_rays(c2w, 40, 40, 50.0, "cuda")
    want = realtime_model().render_frame(c2w[:, 3], v)[0]
    model = realtime_model()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        torch.cuda._sleep(HOLD)
        model.tc_blob()
    with torch.cuda.stream(b):
        got = model.render_frame(c2w[:, 3], v)[0]
    torch.cuda.synchronize()
    assert torch.equal(got, want) and int(model.tc_err.item()) == 0


def test_frames_of_one_model_on_several_threads():
    """Each thread renders its own view on its own stream; a frame's round counts
    come back to that frame alone, so every one equals the frame rendered by
    itself.  Frames one after the other on two streams share nothing either."""
    from concurrent.futures import ThreadPoolExecutor

    from diver_gb300 import scenes

    model = realtime_model()
    eyes, dirs, want = [], [], []
    for seed in range(4):
        c2w = scenes.sphere_cameras(1, 4.0, seed)[0]
        eyes.append(c2w[:, 3])
        dirs.append(scenes.camera_rays(c2w, 20 * (seed + 1), 30, 45.0, "cuda")[1])
        want.append(model.render_frame(eyes[-1], dirs[-1])[0])
    torch.cuda.synchronize()

    def frames(i):
        s, out = torch.cuda.Stream(), []
        with torch.cuda.stream(s):
            for _ in range(10):
                out.append(model.render_frame(eyes[i], dirs[i])[0])
        s.synchronize()
        return out

    with ThreadPoolExecutor(4) as pool:
        for i, out in enumerate(pool.map(frames, range(4))):
            assert all(torch.equal(x, want[i]) for x in out)
    streams, got = [torch.cuda.Stream() for _ in range(2)], []
    for k in range(20):
        with torch.cuda.stream(streams[k % 2]):
            got.append(model.render_frame(eyes[k % 4], dirs[k % 4])[0])
    torch.cuda.synchronize()
    assert all(torch.equal(x, want[k % 4]) for k, x in enumerate(got))
    # nothing that the host waits on stays with the model for another frame to share
    kept = [y for x in vars(model).values() for y in (x if isinstance(x, (tuple, list)) else [x])]
    assert not any(isinstance(y, torch.Tensor) and y.is_pinned() for y in kept)
    assert int(model.tc_err.item()) == 0


@pytest.mark.parametrize("form", ["bf16", "fp16", "bf16s"])
def test_images_belong_to_the_calling_stream(form):
    """The refresh runs on the side stream, but the images' memory is the calling
    stream's: freed there, it is used again behind the decode that read it."""
    field = small_field()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s), torch.no_grad():
        field(*rays(1500), form=form)
    torch.cuda.synchronize()
    tw = field.tc_weights(form)
    kept = [tw.blob, tw.bias, tw.err] + ([tw.bwd[0]] if tw.bwd else []) + ([tw._folded] if tw._folded is not None else [])
    for t in kept:
        owner = [g["stream"] for g in torch.cuda.memory_snapshot()
                 if g["address"] <= t.data_ptr() < g["address"] + g["total_size"]]
        assert owner == [s.cuda_stream]
