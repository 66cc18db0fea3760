"""A window whose rows may use no entry: caps at and below zero leave the poses as they are, whatever
the sizes of the edges whose rows are sorted side by side."""
import numpy as np
import pytest

from rkhs_ba_gb300 import CvoGPU, CvoParams, CvoPointCloud, params_path

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap", [0, -1, -8, -1000])
def test_no_entry_of_any_row(cuda_device, cap):
    rng = np.random.default_rng(1)
    sizes = (33, 400, 31, 2000, 129)
    clouds = [CvoPointCloud(rng.uniform(0, 1, (n, 3)) + 3, np.full((n, 5), 0.5)) for n in sizes]
    p = CvoParams(params_path("irls"))
    p.nearest_neighbors_max, p.multiframe_max_iters, p.multiframe_min_nonzeros = cap, 2, 1
    P0 = np.tile(np.eye(4)[:3].reshape(12), (len(sizes), 1))
    edges = [(3, 1), (0, 3), (2, 3), (4, 3), (1, 3)]
    P, _, _ = CvoGPU(params=p).align_multi(clouds, P0, [1] + [0] * 4, edges)
    assert np.array_equal(P, P0)
