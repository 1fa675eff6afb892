"""Far queries of the spatial search, whose boxes hold cells of many points: a row of cells of up to
32 points is one lane's, a longer one the whole warp's.  Clumps of 31 to 5,000 points in one cell and
lone points far from them and from each other, against the oracle."""
import numpy as np
import pytest

from oracle import spatial as osp
from msc_b200 import spatial as msp, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("clump,k", [(31, 4), (32, 9), (33, 20), (65, 33), (64, 65), (5_000, 2),
                                     (5_000, 65)])
def test_clumps_and_lone_points(clump, k, dims):
    import torch
    rng = np.random.default_rng(clump + k)
    P = [rng.normal(0, 0.01, (clump, dims))]
    P.append(rng.normal(0, 0.01, (max(clump // 2, 1), dims)) + 400.0)
    P.append(rng.uniform(-90_000, 90_000, (70, dims)))
    P = np.vstack(P).astype(np.float32)
    P[-1] = P[-2]                                        # and a coincident pair
    idx, dist, stats = msp.knn_grid_device(torch.from_numpy(P).cuda(), k)
    _lib.check_spatial_stats(stats.cpu().numpy())
    oi, od = osp.grid_knn(P, k)
    np.testing.assert_array_equal(idx.cpu().numpy(), oi)
    np.testing.assert_array_equal(dist.cpu().numpy(), od)


@pytest.mark.parametrize("dims,width", [(2, 1.0), (3, 1.0), (3, 0.0), (2, 40.0)])
@pytest.mark.parametrize("n,k", [(2_094, 45), (5_000, 9)])
def test_points_along_a_line_need_one_box(n, k, dims, width):
    import torch
    rng = np.random.default_rng(n + dims)
    P = rng.normal(0, 1, (n, dims)) * width
    P[:, 0] = rng.random(n) * 10_000
    P = P.astype(np.float32)
    idx, dist, stats = msp.knn_grid_device(torch.from_numpy(P).cuda(), k)
    oi, od = osp.grid_knn(P, k)
    np.testing.assert_array_equal(idx.cpu().numpy(), oi)
    np.testing.assert_array_equal(dist.cpu().numpy(), od)
    # most queries end in the first box of cells (in the plane and in space about one in four goes on)
    assert int(stats[_lib.SP_STAT_EXPANDED]) <= n // 3
