"""The association's candidate test and row pass at the sizes where their tiling can go
wrong, against the CPU oracle: identical columns per row, values within 1e-5 relative (FP32
exp against the oracle's double).  Sizes straddle the tile of 32 rows, the group of 32 and
the supergroup of 1,024 targets (the bitmap window of 20,480: test_gpu_long_rows.py); caps below and above the
rows' counts; tiles many lengthscales wide; and the kernels without a geometric term."""
import numpy as np
import pytest

from oracle import oracle as orc
from rkhs_ba_gb300 import CvoGPU, CvoParams, CvoPointCloud, params_path

pytestmark = pytest.mark.gpu


def _check(p, src, tgt, T, ell):
    a = CvoGPU(params=p).compute_association_gpu(src, tgt, T, ell)
    ind, val, nnz = orc.association(p, src, tgt, T, ell, cap=p.nearest_neighbors_max)
    assert a.rows == src.num_points() and int(a.row_ptr[-1]) == int(nnz.sum())
    for i in range(a.rows):
        lo, hi = a.row_ptr[i], a.row_ptr[i + 1]
        assert np.array_equal(a.col[lo:hi], ind[i, :nnz[i]]), i
        assert np.allclose(a.val[lo:hi], val[i, :nnz[i]], rtol=1e-5, atol=0), i
    return int(nnz.sum()), int(nnz.max(initial=0))


def _cloud(rng, n, size, features=True):
    return CvoPointCloud(rng.uniform(0, size, (n, 3)), rng.uniform(0.3, 0.7, (n, 5)) if features else None)


T = np.array([[0.9998, -0.02, 0, 0.03], [0.02, 0.9998, 0, -0.02], [0, 0, 1, 0.01], [0, 0, 0, 1]], np.float32)


@pytest.mark.parametrize("n, m, cap", [(1, 1, 4), (31, 33, 256), (32, 32, 5), (33, 1025, 64), (65, 1024, 256), (40, 66000, 300),
                                       (1030, 2049, 7)])
@pytest.mark.parametrize("kind", ["geometric", "color"])
def test_sizes(cuda_device, n, m, cap, kind):
    rng = np.random.default_rng(n * 1000 + m)
    p = CvoParams(params_path(kind))
    p.nearest_neighbors_max = cap
    src, tgt = (_cloud(rng, k, 1.2, kind == "color") for k in (n, m))
    total, most = _check(p, src, tgt, T, 0.3)
    assert m < 1000 or total > 0
    if (m, cap) in ((66000, 300), (2049, 7)):
        assert most == cap


@pytest.mark.parametrize("ell", [0.002, 0.05])
def test_tiles_wider_than_the_half_precision_range(cuda_device, ell):
    """Neighbours in clusters tens of metres apart: a tile spans up to 10^4 lengthscales."""
    rng = np.random.default_rng(7)
    c = rng.uniform(-40, 40, (150, 1, 3))
    src, tgt = (CvoPointCloud((c + ell * rng.normal(size=(150, 3, 3))).reshape(-1, 3), rng.uniform(0.4, 0.6, (450, 5)))
                for _ in range(2))
    p = CvoParams(params_path("color"))
    total, _ = _check(p, src, tgt, np.eye(4, dtype=np.float32), ell)
    assert total > 100


@pytest.mark.parametrize("geometry, intensity", [(0, 1), (0, 0), (1, 1)])
def test_terms_switched_off(cuda_device, geometry, intensity):
    rng = np.random.default_rng(3)
    p = CvoParams(params_path("color"))
    p.is_using_geometry, p.is_using_intensity, p.nearest_neighbors_max = geometry, intensity, 50
    total, _ = _check(p, _cloud(rng, 70, 3.0), _cloud(rng, 1500, 3.0), T, 0.4)
    assert total > 0


@pytest.mark.parametrize("n, m, cap", [(300, 8192, 64), (300, 8193, 64), (70, 20001, 200)])
def test_targets_that_take_a_launch_for_the_rows_of_few_candidates(cuda_device, n, m, cap):
    """Rows of 0 to thousands of candidates on both sides of the 8,192 targets."""
    rng = np.random.default_rng(m)
    p = CvoParams(params_path("geometric"))
    p.nearest_neighbors_max = cap
    src, tgt = (CvoPointCloud(np.abs(rng.normal(size=(k, 3))) ** 3) for k in (n, m))
    total, most = _check(p, src, tgt, T, 0.1)
    assert total > 0 and most == cap


@pytest.mark.parametrize("m, cap", [(4127, 32), (4128, 32), (4129, 32), (6000, 7), (9000, 300)])
def test_align_of_rows_longer_than_those_put_in_order(cuda_device, m, cap):
    """Every target lies within the radius of every source: rows that keep about 4,096 pairs
    more than cap.  Three iterations against the oracle's, 1e-5 rad / 1e-5 m (the kept pairs are
    the same, FP32 sums of them in another order: 1e-6 relative, steps of at most 1 cm)."""
    rng = np.random.default_rng(m)
    p = CvoParams(params_path("color"))
    p.nearest_neighbors_max, p.MAX_ITER = cap, 3
    src, tgt = (CvoPointCloud(rng.uniform(0, 1, (k, 3)) + 2, rng.uniform(0.49, 0.51, (k, 5))) for k in (65, m))
    ret, Tg, _, _, it = CvoGPU(params=p).align(src, tgt, T)
    ret_o, To, it_o, _ = orc.align(p, src, tgt, T)
    assert (ret, it) == (ret_o, it_o)
    R = Tg[:3, :3].T.astype(np.float64) @ To[:3, :3].astype(np.float64)
    assert np.linalg.norm(R - R.T) / 2 < 1e-5 and np.linalg.norm(Tg[:3, 3] - To[:3, 3]) < 1e-5
