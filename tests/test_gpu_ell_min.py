"""A lengthscale without a lower bound: ell_min at, below and far below zero against the oracle."""
import numpy as np
import pytest

from oracle import oracle as orc
from rkhs_ba_gb300 import CvoGPU, CvoParams, params_path, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ell_min", [0.0, -0.25, -1.0, -100.0])
def test_no_lower_bound(cuda_device, ell_min):
    src, tgt, _ = scenes.room_pair(n=1500, seed=4)
    p = CvoParams(params_path("geometric"))
    p.MAX_ITER, p.ell_min = 4, ell_min
    ret, T, _, _, it = CvoGPU(params=p).align(src, tgt, np.eye(4))
    ret_o, To, it_o, _ = orc.align(p, src, tgt, np.eye(4))
    assert (ret, it) == (ret_o, it_o)
    R = T[:3, :3].T.astype(np.float64) @ To[:3, :3].astype(np.float64)
    assert np.linalg.norm(R - R.T) / 2 < 1e-4 and np.linalg.norm(T[:3, 3] - To[:3, 3]) < 1e-4
