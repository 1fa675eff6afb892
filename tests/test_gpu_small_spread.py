"""Embeddings of so small a spread that the FP32 squares of their differences leave the normal range
(below about 1e-20): an FP32 distance is then off by more than its relative bound says, and only
what is decided in FP64 counts.  The scales run from where every square is normal to where all of
them vanish; the lists are the oracle's at each."""
import numpy as np
import pytest

import oracle
from msc_b200 import neighbors as nbm, synth, _lib

pytestmark = pytest.mark.gpu

SCALES = [1e-16, 1e-20, 3e-21, 1e-21, 1e-22, 1e-23]


def cells(scale, n=1_500, d=30):
    X = synth.gaussian_mixture(n, d, 3, seed=5, centre_scale=2.0)
    return (X.astype(np.float64) * scale).astype(np.float32)


def assert_lists(X, k, **kw):
    import torch
    idx, dist, st = nbm.knn_device(torch.from_numpy(X).cuda(), k, **kw)
    torch.cuda.synchronize()
    assert int(st[_lib.STAT_TIMEOUT]) == 0
    ri, _, rd = oracle.knn_exact(X, k)
    np.testing.assert_array_equal(idx.cpu().numpy(), ri.astype(np.int32))
    np.testing.assert_array_equal(dist.cpu().numpy(), rd)


@pytest.mark.parametrize("scale", SCALES)
@pytest.mark.parametrize("k", [83, 200])
def test_wide_lists(k, scale):
    assert_lists(cells(scale), k)
