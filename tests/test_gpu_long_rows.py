"""Rows of an align that keep more than 512 pairs, put in lattice order through a bitmap over the
ranks, and rows whose candidates cross the row pass's windows of 20,480 target indices."""
import numpy as np
import pytest

from oracle import oracle as orc
from rkhs_ba_gb300 import CvoGPU, CvoParams, CvoPointCloud, params_path

pytestmark = pytest.mark.gpu


def _params(cap, iters):
    p = CvoParams(params_path("color"))
    p.nearest_neighbors_max, p.MAX_ITER, p.ell_init = cap, iters, 0.1
    return p


def _against_oracle(p, src, tgt):
    """Within 1e-5 rad / 1e-5 m: the kept pairs are the same, FP32 sums of them in another order
    (1e-6 relative), steps of at most 1 cm."""
    T = np.eye(4, dtype=np.float32)
    ret, Tg, _, _, it = CvoGPU(params=p).align(src, tgt, T)
    ret_o, To, it_o, _ = orc.align(p, src, tgt, T)
    assert (ret, it) == (ret_o, it_o)
    R = Tg[:3, :3].T.astype(np.float64) @ To[:3, :3].astype(np.float64)
    assert np.linalg.norm(R - R.T) / 2 < 1e-5 and np.linalg.norm(Tg[:3, 3] - To[:3, 3]) < 1e-5
    return Tg


def _sites(n, m, middle):
    """m targets on a line of sites 0.2 m apart (wider than a lattice cell at this lengthscale) of
    equal points, 400 or so to a site, site by site or dealt out over the indices; n sources around
    site `middle`."""
    rng = np.random.default_rng(m)
    k = max(5, m // 400)
    feat = rng.uniform(0.49, 0.51, (k, 5))
    site = np.arange(m) % k
    src = np.array([0.2 * middle, 0, 3]) + rng.uniform(-0.06, 0.06, (n, 3))
    cloud = lambda s: CvoPointCloud(np.stack([0.2 * s, 0 * s, 3 + 0 * s], 1), feat[s])  # noqa: E731
    return CvoPointCloud(src, rng.uniform(0.49, 0.51, (n, 5))), cloud(site), cloud(np.sort(site))


@pytest.mark.parametrize("n, m, middle", [(70, 1601, 2), (40001, 4001, 5), (70, 20480, 25), (70, 20481, 25), (70, 45000, 51)])
def test_order_is_the_lattice_s(cuda_device, n, m, middle):
    """Rows of some 1,200 pairs: the sums of targets dealt out over the indices are those of targets
    in the order of the sites, to the bit, and the oracle's.  40,001 rows have their room per warp."""
    src, dealt, by_site = _sites(n, m, middle)
    p = _params(4000, 8)
    _, _, nnz = orc.association(p, src, dealt, np.eye(4, dtype=np.float32), p.ell_init, cap=4000)
    assert 512 < nnz.max() < 4000
    T = _against_oracle(p, src, dealt)
    assert np.array_equal(T, CvoGPU(params=p).align(src, by_site, np.eye(4, dtype=np.float32))[1])


@pytest.mark.parametrize("m, cap", [(600, 513), (2000, 1500), (20480, 1500), (20481, 513), (45000, 1500), (45000, 4000)])
def test_dense_rows(cuda_device, m, cap):
    """Rows that keep fewer pairs than cap, more than cap, and more than 4,096 beyond it."""
    rng = np.random.default_rng(m + cap)
    src, tgt = (CvoPointCloud(rng.uniform(0, 0.35, (n, 3)) + (0, 0, 3), rng.uniform(0.45, 0.55, (n, 5))) for n in (65, m))
    p = _params(cap, 3)
    _, _, nnz = orc.association(p, src, tgt, np.eye(4, dtype=np.float32), p.ell_init, cap=m)
    assert nnz.max() > 500
    _against_oracle(p, src, tgt)
