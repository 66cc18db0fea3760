"""Calls that have to fit into what is left of the device's memory."""
import contextlib

import numpy as np
import pytest

from rkhs_ba_gb300 import CvoGPU, CvoParams, CvoPointCloud, params_path
from rkhs_ba_gb300._lib import CvoError

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


def test_inner_product_with_little_room_for_candidates(cuda_device):
    """A candidate entry per row and group of 32 targets would be 1 GB; rows that need more entries than
    there is room for scan the targets."""
    rng = np.random.default_rng(2)
    cvo = CvoGPU(params=CvoParams(params_path("geometric")))
    src, tgt = _uniform(rng, 20000, 20.0), _uniform(rng, 200000, 20.0)
    want = cvo.inner_product_gpu(src, tgt, np.eye(4), 0.25)
    for size in (1 << 30, 400 << 20, 100 << 20):
        small = CvoGPU(params=cvo.get_params())
        gs, gt = small.upload(src), small.upload(tgt)
        with _free_memory(size):
            got = small.inner_product_gpu(gs, gt, np.eye(4), 0.25)
        assert abs(got - want) <= 1e-6 * want


def test_clouds_of_a_refused_align_are_ready_on_another_stream(cuda_device):
    """A kernel matrix that no device holds: the align is refused after the targets' orders were built, and
    the next one, of another handle on a stream of its own, may use them at once."""
    rng = np.random.default_rng(3)
    p = CvoParams(params_path("geometric"))
    p.MAX_ITER = 3
    src, tgt = _uniform(rng, 300000, 30.0), _uniform(rng, 300000, 30.0)
    cvo = CvoGPU(params=p)
    want = cvo.align(src, tgt, np.eye(4))[1]
    greedy = p.copy()
    greedy.nearest_neighbors_max = 1 << 22
    first, second = CvoGPU(params=greedy), CvoGPU(params=p)
    for _ in range(3):
        gs, gt = first.upload(src), first.upload(tgt)
        with pytest.raises(CvoError):
            first.align(gs, gt, np.eye(4))
        assert np.array_equal(second.align(gs, gt, np.eye(4))[1], want)
