"""The plain FP32 form's record of a training forward's activations: how much of
it is held at a time, when it is given back, and what happens where there is no
room for it.  The accounting on the CPU; the steps on the GPU, with failed
allocations made on the host."""
import pytest
import torch

from diver_gb300 import _native as N
from diver_gb300 import renderer

CPU = torch.device("cpu")
SEGS = 1000


@pytest.fixture
def one(monkeypatch):
    """Bytes of one record, with room for two and a half on the CPU 'device'."""
    n = int(N.lib().dv_decode_save_bytes(32, 32, SEGS))
    monkeypatch.setattr(renderer, "PLAIN_SAVE", 2 * n + n // 2)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    return n


def test_records_are_bounded_together(one):
    """Forwards whose backward is still to run share the limit; a smaller one may
    still fit, and what is dropped makes room."""
    a, b = (renderer._plain_save(32, 32, SEGS, CPU) for _ in range(2))
    assert a.data.numel() == b.data.numel() == one
    assert renderer._plain_save(32, 32, SEGS, CPU) is None
    small = renderer._plain_save(32, 32, SEGS // 4, CPU)
    assert small is not None
    del small, a
    assert renderer._plain_save(32, 32, SEGS, CPU) is not None


def test_no_record_of_nothing_or_of_too_much(one):
    assert renderer._plain_save(32, 32, 0, CPU) is None
    assert renderer._plain_save(32, 32, 3 * SEGS, CPU) is None
    assert renderer._plain_save(32, 64, SEGS, CPU) is None  # no such decoder


def test_no_room_for_a_record(one, monkeypatch):
    def full(*args, **kw):
        raise torch.cuda.OutOfMemoryError("full")

    empty = torch.empty
    monkeypatch.setattr(torch, "empty", full)
    assert renderer._plain_save(32, 32, SEGS, CPU) is None
    monkeypatch.setattr(torch, "empty", empty)
    assert renderer._plain_save(32, 32, 2 * SEGS, CPU) is not None  # nothing was counted


@pytest.mark.parametrize("eighths,kept", [(7, False), (8, True), (80, True)])
def test_captured_step_takes_an_eighth_of_the_free_memory(one, monkeypatch, eighths, kept):
    """A graph keeps the record for good and cannot make up for a failed
    allocation, so it looks at the free memory instead of trying."""
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device=None: (eighths * one, 100 * one))
    assert (renderer._plain_save(32, 32, SEGS, CPU) is not None) == kept


# ---- on the GPU --------------------------------------------------------------

def step_of(field, o, d):
    rgb, reg = field(o, d)
    return (rgb * torch.arange(1.0, 4.0, device="cuda")).mean() + 1e-3 * reg


@pytest.fixture
def field():
    from diver_gb300 import scenes
    from diver_gb300.renderer import DIVeRField

    return DIVeRField.from_scene(scenes.small_scene("cpu"), "cuda")


@pytest.fixture
def launches(monkeypatch):
    """Names of the entry points launched since."""
    seen = []
    call = N.call
    monkeypatch.setattr(N, "call", lambda name, *a: (seen.append(name), call(name, *a))[1])
    return seen


def views(n):
    from diver_gb300 import scenes

    out = []
    for seed in range(n):
        o, d = scenes.camera_rays(scenes.sphere_cameras(1, 4.0, seed)[0], 30, 30, 40.0, "cuda")
        out.append((o.contiguous(), d.contiguous()))
    return out


def same(a, b):
    """Equal up to the order of the atomic sums, which 1e-5 relative L2 covers (a
    sum of n FP32 terms is off by n 2^-24 of their magnitudes at most, by some
    sqrt(n) 2^-24 in fact, and n is some ten thousand for a weight)."""
    return all(bool((x - y).norm() <= 1e-5 * y.norm()) for x, y in zip(a, b))


@pytest.mark.gpu
def test_several_renders_in_one_loss(field, launches, monkeypatch):
    """With room for the first records only the rest recompute; the gradients are
    those of the renders one by one, and nothing is held afterwards."""
    params = [field.voxels, field.params]
    vs = views(3)
    want = [torch.zeros_like(p) for p in params]
    for v in vs:
        for w, g in zip(want, torch.autograd.grad(step_of(field, *v), params)):
            w += g
    total = [field.segments(*v).total for v in vs]
    room = sum(int(N.lib().dv_decode_save_bytes(32, 32, t)) for t in total[:2])
    monkeypatch.setattr(renderer, "PLAIN_SAVE", room)
    launches.clear()
    loss = sum(step_of(field, *v) for v in vs)
    assert launches.count("dv_decode_fwd_save") == 2 and launches.count("dv_decode_fwd") == 1
    got = torch.autograd.grad(loss, params)
    assert launches.count("dv_decode_bwd_saved") == 2 and launches.count("dv_decode_bwd") == 1
    assert same(got, want)
    assert len(renderer._records) == 0  # although `loss` and its graph are still there


@pytest.mark.gpu
def test_backward_of_a_retained_graph(field, launches):
    """The first backward reads the record and gives it back, a second recomputes."""
    params = [field.voxels, field.params]
    loss = step_of(field, *views(1)[0])
    a = torch.autograd.grad(loss, params, retain_graph=True)
    b = torch.autograd.grad(loss, params)
    assert launches.count("dv_decode_bwd_saved") == 1 and launches.count("dv_decode_bwd") == 1
    assert same(b, a)


@pytest.mark.gpu
@pytest.mark.parametrize("name,which", [("empty_like", 0), ("zeros_like", 0), ("zeros_like", 1)])
def test_no_room_in_the_backward(field, launches, monkeypatch, name, which):
    """An allocation of the backward that fails while the record is held is made
    again without it; one that fails without it is the caller's error."""
    params = [field.voxels, field.params]
    v = views(1)[0]
    want = torch.autograd.grad(step_of(field, *v), params)
    make, calls = getattr(torch, name), []

    def tight(*args, **kw):
        calls.append(len(renderer._records))
        if calls[-1] > 0 and len(calls) > which:
            raise torch.cuda.OutOfMemoryError("full")
        return make(*args, **kw)

    loss = step_of(field, *v)
    launches.clear()
    with monkeypatch.context() as m:
        m.setattr(torch, name, tight)
        got = torch.autograd.grad(loss, params)
    assert "dv_decode_bwd" in launches and "dv_decode_bwd_saved" not in launches
    assert same(got, want)

    def full(*args, **kw):
        raise torch.cuda.OutOfMemoryError("full")

    loss = step_of(field, *v)
    with monkeypatch.context() as m:
        m.setattr(torch, name, full)
        with pytest.raises(torch.cuda.OutOfMemoryError):
            torch.autograd.grad(loss, params)


@pytest.mark.gpu
@pytest.mark.parametrize("room", [False, True])
def test_captured_step_with_and_without_room(field, launches, monkeypatch, room):
    from diver_gb300.graphs import TrainStepGraph

    o, d = views(1)[0]
    target = torch.rand(o.shape[0], 3, device="cuda")
    if not room:
        monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device=None: (1 << 20, 1 << 30))
    step = TrainStepGraph(field, o, d, target, form="fp32", warmup=1)
    assert ("dv_decode_bwd" in launches) == (not room)  # the warm-up's always read theirs
    loss, gv, gp = (x.clone() for x in step(o, d, target))
    rgb, reg = field(o, d)
    ref = renderer.l2_loss(rgb, reg, target, 1e-5)
    want = torch.autograd.grad(ref, [field.voxels, field.params])
    ref = ref.detach()
    assert abs(float(loss - ref)) <= 1e-6 * abs(float(ref)) and same((gv, gp), want)
