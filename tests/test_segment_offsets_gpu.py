"""GPU: dv_segment_offsets (offsets, total and largest count) at the sizes
where it changes form, exact."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 31, 1023, 1024, 1025, 2049, 16383, 16384, 16385, 18432, 18433, 700001])
@pytest.mark.parametrize("high", [1, 800])
def test_segment_offsets(n, high):
    from diver_gb300.ray_voxel_intersection import _offsets_totals

    c = np.random.default_rng(n + high).integers(0, high + 1, n).astype(np.int32)
    off, tot = _offsets_totals(torch.from_numpy(c).cuda())
    assert np.array_equal(off.cpu().numpy(), np.concatenate([[0], np.cumsum(c, dtype=np.int64)]))
    assert tot.tolist() == [int(c.sum()), int(c.max()) if n else 0]
