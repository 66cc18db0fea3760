"""A pair's result does not depend on the batch that it is in, to the bit: batches whose rows
take the gradient and step kernels with other blocks and lanes than a pair alone."""
import numpy as np
import pytest

from rkhs_ba_gb300 import CvoGPU, CvoParams, CvoPointCloud, params_path

pytestmark = pytest.mark.gpu


def _mirrored(rng, n, shift=0.0):
    """n points symmetric in y, two of them 10^7 m away: in the gradient's odd terms these cancel, and
    what is left shows in which groups the rows of the near points were added to them."""
    half = rng.uniform((-1, 0.01, 2), (1, 1, 4), (n // 2, 3))
    half[0] = 1e7 + shift, 1e7, 3
    return CvoPointCloud(np.concatenate([half, half * (1, -1, 1)]), np.tile(rng.uniform(0.45, 0.55, (n // 2, 5)), (2, 1)))


def _alone_and_in_batch(params, srcs, tgts, some):
    cvo = CvoGPU(params=params)
    gs, gt = [cvo.upload(s) for s in srcs], [cvo.upload(t) for t in tgts]
    eye = np.eye(4, dtype=np.float32)
    Ts, rets, its, _ = cvo.align_batch(gs, gt, [eye] * len(gs))
    for k in some:
        ret, T, _, _, it = cvo.align(gs[k], gt[k], eye)
        assert (ret, it) == (rets[k], its[k]) and np.array_equal(T, Ts[k]), k


@pytest.mark.parametrize("sizes", [(20000, 20000, 20000), (3002, 45000, 32), (1000, 40000, 130000, 70000)])
def test_batches_of_more_rows_than_their_pairs(cuda_device, sizes):
    rng = np.random.default_rng(len(sizes))
    p = CvoParams(params_path("color"))
    p.MAX_ITER, p.ell_init, p.nearest_neighbors_max = 5, 0.1, 24
    clouds = [(_mirrored(rng, n), _mirrored(rng, 4000, 1.0)) for n in sizes]
    _alone_and_in_batch(p, *zip(*clouds), range(len(sizes)))


def test_batch_of_more_than_half_a_million_rows(cuda_device):
    """Rows that keep 4,000 pairs at a cap of 200 are added up in the same order alone and beside a
    pair of 600,000 rows."""
    rng = np.random.default_rng(5)
    p = CvoParams(params_path("color"))
    p.MAX_ITER, p.nearest_neighbors_max = 20, 200
    src, tgt = (CvoPointCloud(rng.uniform(0, 1.6, (n, 3)) + 2, rng.uniform(0.495, 0.505, (n, 5))) for n in (300, 4000))
    many, one = (CvoPointCloud(rng.uniform(0, 30, (n, 3)), rng.uniform(0.4, 0.6, (n, 5))) for n in (600000, 1))
    _alone_and_in_batch(p, [src, many], [tgt, one], [0])
