"""The per-query spatial search at its edges against the oracle: far outliers that leave the lane pass,
every list length's last k, empty regions between dense ones, 3-D, and fewer points than a warp."""
import numpy as np
import pytest

from oracle import spatial as osp
from msc_b200 import spatial as msp, _lib

pytestmark = pytest.mark.gpu


def points(name):
    rng = np.random.default_rng(17)
    if name == "outliers":              # a dense patch and lone points far from it and each other
        far = rng.uniform(-50_000, 50_000, (40, 2))
        return np.vstack([rng.normal(0, 40, (3_000, 2)), far]).astype(np.float32)
    if name == "two_patches":           # the nearest points of a sparse strip lie across a gap
        return np.vstack([rng.normal(0, 5, (2_000, 2)), rng.normal(0, 5, (2_000, 2)) + [9_000, 0],
                          np.c_[np.linspace(500, 8_500, 60), np.zeros(60)]]).astype(np.float32)
    if name == "line":                  # one effective axis
        return np.c_[rng.uniform(0, 1e5, 1_500), np.full(1_500, 3.0)].astype(np.float32)
    if name == "cloud3":
        return np.vstack([rng.normal(0, 10, (2_500, 3)),
                          rng.uniform(-2_000, 2_000, (30, 3))]).astype(np.float32)
    return rng.uniform(0, 10, (20, 2)).astype(np.float32)


@pytest.mark.parametrize("name,k", [("outliers", 9), ("outliers", 17), ("outliers", 65),
                                    ("two_patches", 7), ("two_patches", 33), ("line", 10),
                                    ("cloud3", 8), ("cloud3", 33), ("few", 20)])
def test_knn_equals_oracle(name, k):
    import torch
    X = points(name)
    idx, dist, stats = msp.knn_grid_device(torch.from_numpy(X).cuda(), k)
    torch.cuda.synchronize()
    _lib.check_spatial_stats(stats.cpu().numpy())
    oi, od = osp.grid_knn(X, k)
    np.testing.assert_array_equal(idx.cpu().numpy(), oi)
    np.testing.assert_array_equal(dist.cpu().numpy(), od)


@pytest.mark.parametrize("name,radius", [("outliers", 30.0), ("two_patches", 4.0), ("cloud3", 6.0)])
def test_radius_equals_oracle(name, radius):
    import torch
    X = points(name)                    # rows of up to a few hundred entries and empty ones
    ip, cols, dist, _ = msp.radius_grid_device(torch.from_numpy(X).cuda(), radius)
    oip, oc, od = osp.grid_radius(X, radius)
    np.testing.assert_array_equal(ip.cpu().numpy(), oip)
    np.testing.assert_array_equal(cols.cpu().numpy(), oc)
    np.testing.assert_array_equal(dist.cpu().numpy(), od)
