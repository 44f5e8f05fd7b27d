"""GPU: the masked walk's walker / consumer split at its edges, bit-exact
against the C oracle: batches around a warp and around the launch rule's
change, warps that mix ordinary rays with axis-parallel and extreme
directions (the plain step) and with misses, rays through grid corners and
along grid planes (ties), and per-axis extents."""
import numpy as np
import pytest
import torch

from oracle import native as orc
from tests.test_traverse_oracle import same_bits

pytestmark = pytest.mark.gpu


def rays(n, seed, special):
    rng = np.random.default_rng(seed)
    o = rng.uniform(-3.0, 3.0, (n, 3)).astype(np.float32)
    o[::5] = rng.uniform(-1.0, 1.0, (len(o[::5]), 3))  # inside
    at = rng.uniform(-1.2, 1.2, (n, 3))
    v = (at - o).astype(np.float32)
    if special:
        v[1::7, 1:] = 0.0
        v[2::7, 2] = 1e-30
        v[3::7] = rng.choice([-1.0, 1.0], (len(v[3::7]), 3))  # diagonals from lattice points: ties on every axis
        o[3::7] = np.round(o[3::7] * 4) / 4
        v[4::7, 0] = 1e-6
        v[5::7] = o[5::7] - at[5::7]  # most of these miss
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    return o, v.astype(np.float32)


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("batch", [1, 31, 32, 33, 1000, 40000])
@pytest.mark.parametrize("n", [16, 65])
def test_masked_walk_edges(batch, n, special):
    from diver_gb300 import masked_intersect, masked_segments

    o, v = rays(batch, batch + n, special)
    rng = np.random.default_rng(n)
    mask = rng.random((n, n, n)) < 0.5
    x0, vs = -1.5, 3.0 / n
    wi, num, wt = orc.masked_walk(o, v, x0, n, vs, mask, 1.0)
    oi, on, ot = orc.trim(wi, num, wt)  # (a box behind the ray has negative distances: no hit there, segments all the same)
    seg, t = orc.csr_from_padded(wi, num), orc.csr_from_padded(wt, num)
    od, vd, md = torch.from_numpy(o).cuda(), torch.from_numpy(v).cuda(), torch.from_numpy(mask).cuda()
    inter, hit, tns = masked_intersect(od, vd, x0, -x0, n, vs, md, 1.0)
    assert np.array_equal(hit.cpu().numpy(), on)
    assert same_bits(inter.cpu().numpy(), oi) and same_bits(tns.cpu().numpy(), ot)
    for capacity in (None, batch * (3 * n + 3)):
        if capacity is not None and batch > 1000:
            continue
        sg = masked_segments(od, vd, x0, n, vs, md, 1.0, capacity)
        S = int(sg.offsets[-1])
        assert same_bits(sg.seg[:S].cpu().numpy(), seg) and same_bits(sg.t[:S].cpu().numpy(), t)
        assert np.array_equal(sg.ray[:S].cpu().numpy(), np.repeat(np.arange(batch), num))
        assert np.array_equal(sg.counts.cpu().numpy(), num)


def test_masked_walk_per_axis_extents():
    from diver_gb300.ray_voxel_intersection import masked_segments_grid

    dims, vs = (40, 9, 23), 0.05
    x0 = [-1.0, -0.25, -0.5]
    o, v = rays(3000, 5, True)
    rng = np.random.default_rng(1)
    mask = rng.random((dims[2], dims[1], dims[0])) < 0.6
    oi, num, ot = orc.masked_walk_grid(o, v, x0, dims, vs, mask)
    sg = masked_segments_grid(torch.from_numpy(o).cuda(), torch.from_numpy(v).cuda(), x0, dims, vs,
                              torch.from_numpy(mask).cuda())
    assert np.array_equal(sg.counts.cpu().numpy(), num)
    assert same_bits(sg.seg.cpu().numpy(), orc.csr_from_padded(oi, num))


@pytest.mark.parametrize("extra", [-1, 0, 33])
def test_masked_count_of_large_batches(extra):
    """Around 768 rays per SM, where a count goes from the ring to a thread per ray."""
    from diver_gb300 import masked_segments

    batch = 768 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    o, v = rays(batch, 11, True)
    n, x0 = 12, -1.5
    mask = np.random.default_rng(2).random((n, n, n)) < 0.5
    wi, num, wt = orc.masked_walk(o, v, x0, n, 3.0 / n, mask, 1.0)
    sg = masked_segments(torch.from_numpy(o).cuda(), torch.from_numpy(v).cuda(), x0, n, 3.0 / n,
                         torch.from_numpy(mask).cuda(), 1.0)
    assert np.array_equal(sg.counts.cpu().numpy(), num)
    assert same_bits(sg.seg.cpu().numpy(), orc.csr_from_padded(wi, num))
    assert same_bits(sg.t.cpu().numpy(), orc.csr_from_padded(wt, num))
