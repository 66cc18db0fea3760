"""The window solve's normal equations where their tiling can go wrong (rows around the warp's
32 and the block's 128, entries per row around 32, edges of very different sizes) against the
oracle's FP64 solve: one outer iteration within 1e-5 rad / 1e-5 m, the bound of the window tests."""
import numpy as np
import pytest

from oracle import oracle as orc
from rkhs_ba_gb300 import CvoGPU, CvoParams, CvoPointCloud, params_path, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes, cap", [((31, 1025, 33), 512), ((1024, 1056, 1023), 31), ((2049, 64, 5000), 33), ((700, 700, 700), 1)])
def test_one_outer_iteration(cuda_device, sizes, cap):
    rng = np.random.default_rng(sum(sizes))
    gt = [scenes.make_T(scenes.random_rotation(rng, 0.4), rng.uniform(-1, 1, 3)) for _ in sizes]
    world = rng.uniform(0, 1.0, (6000, 3)) + np.array([4.0, -3.0, 6.0])
    clouds = []
    for T, n in zip(gt, sizes):
        w = world[rng.permutation(6000)[:n]] if n < 6000 else world
        clouds.append(CvoPointCloud((w + 0.01 * rng.normal(size=w.shape) - T[:3, 3]) @ T[:3, :3], np.full((n, 5), 0.5)))
    P0 = np.stack([(T @ scenes.make_T(scenes.rot_axis_angle(rng.normal(size=3), 0.002), 0.01 * rng.normal(size=3)) if k else T)[:3]
                   .reshape(12) for k, T in enumerate(gt)])
    p = CvoParams(params_path("irls"))
    p.multiframe_max_iters, p.multiframe_num_neighbors, p.multiframe_min_nonzeros = 1, cap, 1
    edges = [(0, 1), (2, 1), (0, 2)]
    Pg, _, it = CvoGPU(params=p).align_multi(clouds, P0, [1, 0, 0], edges)
    Po, it_o, steps = orc.align_multi(p, clouds, P0, [1, 0, 0], edges)
    assert it == it_o == 1 and steps > 0
    for a, b in zip(Pg.reshape(-1, 3, 4), np.asarray(Po).reshape(-1, 3, 4)):
        R = a[:, :3].T @ b[:, :3]
        assert np.linalg.norm(R - R.T) / 2 < 1e-5 and np.linalg.norm(a[:, 3] - b[:, 3]) < 1e-5
