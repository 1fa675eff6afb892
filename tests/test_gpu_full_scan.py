"""The full scan of small samples (no locality order, every query tile's keys split into ranges with
a candidate list each): the same lists as the ordered and pruned path and as the oracle, at the
edges of tiles, ranges and list lengths, for cells stored by cluster, and for every precision."""
import os

import numpy as np
import pytest

import oracle
from msc_b200 import neighbors as nbm, synth, _lib

pytestmark = pytest.mark.gpu


def _knn(X, k, dense, **kw):
    import torch
    os.environ["MSC_B200_DENSE"] = str(dense)
    try:
        idx, dist, stats = nbm.knn_device(torch.from_numpy(X).cuda(), k, **kw)
        torch.cuda.synchronize()
        s = stats.cpu().numpy()
        assert int(s[_lib.STAT_TIMEOUT]) == 0
        return idx.cpu().numpy(), dist.cpu().numpy()
    finally:
        del os.environ["MSC_B200_DENSE"]


CASES = [
    # n, d, k, metric, precision, kprime, sorted by cluster
    (256, 20, 15, "euclidean", "fp16", 0, False),       # one key tile: no split
    (257, 20, 15, "euclidean", "fp16", 0, False),       # two ranges, the second of one key
    (641, 50, 5, "euclidean", "fp16", 0, True),         # a last half tile without keys
    (2_049, 61, 10, "euclidean", "fp16", 0, False),     # widest one-atom row, eight key tiles + 1
    (3_000, 62, 15, "cosine", "fp16", 0, True),         # two atoms per row
    (5_001, 100, 30, "cosine", "fp16", 0, False),       # two ranges
    (4_500, 125, 16, "euclidean", "bf16x3", 0, True),
    (4_097, 50, 34, "euclidean", "bf16", 0, False),
    (4_000, 40, 50, "euclidean", "fp16", 0, False),     # wide lists: no split
    (3_001, 30, 65, "euclidean", "fp16", 0, True),
    (6_000, 30, 15, "euclidean", "fp16", 60, False),    # candidates asked for
    (20_011, 50, 15, "euclidean", "fp16", 0, True),
]


@pytest.mark.parametrize("n,d,k,metric,precision,kprime,by_cluster", CASES)
def test_full_scan_equals_ordered_path_and_oracle(n, d, k, metric, precision, kprime, by_cluster):
    X = synth.gaussian_mixture(n, d, 12, seed=n, sizes="lognormal", noise_frac=0.01,
                               shuffle=not by_cluster)
    fi, fd = _knn(X, k, 1 << 20, metric=metric, precision=precision, kprime=kprime)
    oi, od = _knn(X, k, 0, metric=metric, precision=precision, kprime=kprime)
    np.testing.assert_array_equal(fi, oi, err_msg="full scan vs ordered path: indices")
    np.testing.assert_array_equal(fd, od, err_msg="full scan vs ordered path: distances")
    rows = np.sort(np.random.default_rng(n).choice(n, min(n, 1000), replace=False))
    ri, _, rd = oracle.knn_exact(X, k, metric=metric, rows=rows)
    np.testing.assert_array_equal(fi[rows], ri.astype(np.int32))
    np.testing.assert_array_equal(fd[rows], rd)


def test_full_scan_of_coincident_and_non_finite_cells():
    rng = np.random.default_rng(3)
    X = rng.normal(size=(3_000, 30)).astype(np.float32)
    X[100:700] = X[100]                                  # 600 coincident cells: ties by index
    fi, fd = _knn(X, 15, 1 << 20)
    ri, _, rd = oracle.knn_exact(X, 15)
    np.testing.assert_array_equal(fi, ri.astype(np.int32))
    np.testing.assert_array_equal(fd, rd)
    import torch
    X[5, 3] = np.nan
    _, _, stats = nbm.knn_device(torch.from_numpy(X).cuda(), 15)
    with pytest.raises(ValueError):
        _lib.check_stats(stats.cpu().numpy())
