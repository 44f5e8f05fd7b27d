"""GPU: the frame loop over its live pixels against the reference's loop
(aabb_intersect, then ray_march and the tensor-core decoder over every pixel),
bit for bit, at sizes around a tile of pixels and with the rounds cut short."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["diver32", "diver64"])
@pytest.mark.parametrize("pixels", [1, 127, 128, 129, 5000])
@pytest.mark.parametrize("max_rounds", [None, 1, 2])
def test_live_loop_is_the_full_loop(kind, pixels, max_rounds):
    from diver_gb300 import aabb_intersect, ray_march, scenes
    from tests.test_realtime import small_realtime

    sc, _, model = small_realtime(kind, "cuda", bias=0.2)
    c2w = scenes.sphere_cameras(1, 4.0, 3)[0]
    _, v = scenes.camera_rays(c2w, 100, 100, 120.0, "cuda")
    v = v[torch.randperm(v.shape[0], generator=torch.Generator().manual_seed(pixels))[:pixels].cuda()].contiguous()
    got, _ = model.render_frame(c2w[:, 3], v, max_rounds=max_rounds)

    center = ((c2w[:, 3] - model.xyzmin) / model.voxel_size).cuda()
    coords = torch.zeros(8, pixels, 6, device="cuda")
    rgba = torch.zeros(pixels, 4, device="cuda")
    finish = torch.zeros(pixels, dtype=torch.bool, device="cuda")
    aabb_intersect(coords, v, center, finish, rgba, model.octrees, 64)
    rounds = 0
    while rounds < (192 if max_rounds is None else max_rounds) and not bool(finish.all()):
        ray_march(coords, v, model.voxel_masks, finish, 64)
        model.mlp_eval(rgba, coords, v, finish, True)
        rounds += 1
    assert torch.equal(got, rgba[:, :3] + rgba[:, 3:])
    assert int(model.tc_err.item()) == 0
