"""Calls that have to fit into what is left of the device's memory."""
import contextlib

import numpy as np
import pytest

from rkhs_ba_gb300 import CvoGPU, CvoParams, CvoPointCloud, params_path

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def _free_memory(size):
    """All but `size` bytes of the device's memory taken."""
    import torch

    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    if free < size:
        pytest.skip("less memory free than the test leaves")
    taken = torch.empty(free - size, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del taken
        torch.cuda.empty_cache()


def _uniform(rng, n, size, features=0):
    return CvoPointCloud(rng.uniform(0, size, (n, 3)), rng.uniform(0, 1, (n, features)) if features else None)


def test_align_with_long_rows_needs_one_kernel_matrix(cuda_device):
    """20,000 rows of up to 20,000 pairs are 3.2 GB; twice that, for the order of the rows, is not needed."""
    rng = np.random.default_rng(1)
    p = CvoParams(params_path("geometric"))
    p.nearest_neighbors_max, p.MAX_ITER = 20000, 2
    src, tgt = _uniform(rng, 20000, 4.0), _uniform(rng, 20000, 4.0)
    T0 = CvoGPU(params=p).align(src, tgt, np.eye(4))[1]
    cvo = CvoGPU(params=p)
    gs, gt = cvo.upload(src), cvo.upload(tgt)
    with _free_memory(6 << 30):
        T = cvo.align(gs, gt, np.eye(4))[1]
    assert np.array_equal(T, T0)
