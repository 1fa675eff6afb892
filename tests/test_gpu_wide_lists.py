"""Lists wider than 65 neighbours (wide.cu: FP32 differences, FP64 around the k-th place) against the
oracle, at the edges of its tiles (8 rows, 64 to 256 keys), samples (1,024 keys and more) and lists (128,
256, 512), for odd and even widths, both metrics, coincident cells and several samples."""
import numpy as np
import pytest

import oracle
from msc_b200 import batch, neighbors as nbm, synth, _lib

pytestmark = pytest.mark.gpu

CASES = [
    # n, d, k, metric
    (66, 3, 66, "euclidean"),            # every other cell is a neighbour
    (129, 1, 70, "euclidean"),
    (1_024, 127, 129, "euclidean"),      # the sample is every key; 128-entry list
    (1_025, 128, 130, "cosine"),         # ... and one key more; 256-entry list
    (3_001, 30, 82, "euclidean"),
    (5_003, 50, 257, "cosine"),
    (9_000, 17, 513, "euclidean"),
    (20_000, 20, 100, "euclidean"),
]


@pytest.mark.parametrize("n,d,k,metric", CASES)
def test_wide_lists_equal_oracle(n, d, k, metric):
    import torch
    X = synth.gaussian_mixture(n, d, 7, seed=n + k, sizes="lognormal", noise_frac=0.01,
                               shuffle=n % 2 == 0)
    idx, dist, stats = nbm.knn_device(torch.from_numpy(X).cuda(), k, metric=metric)
    torch.cuda.synchronize()
    st = stats.cpu().numpy()
    assert int(st[_lib.STAT_RESCANNED]) == n
    rows = np.sort(np.random.default_rng(1).choice(n, min(n, 800), replace=False))
    ri, _, rd = oracle.knn_exact(X, k, metric=metric, rows=rows)
    np.testing.assert_array_equal(idx.cpu().numpy()[rows], ri.astype(np.int32))
    np.testing.assert_array_equal(dist.cpu().numpy()[rows], rd)


def test_coincident_cells_and_a_nan_row():
    import torch
    rng = np.random.default_rng(2)
    X = rng.normal(size=(2_500, 12)).astype(np.float32)
    X[300:900] = X[300]                                  # more coincident cells than the list holds
    idx, dist, _ = nbm.knn_device(torch.from_numpy(X).cuda(), 90)
    ri, _, rd = oracle.knn_exact(X, 90)
    np.testing.assert_array_equal(idx.cpu().numpy(), ri.astype(np.int32))
    np.testing.assert_array_equal(dist.cpu().numpy(), rd)
    X[7, 0] = np.nan                                     # its row takes the FP64 scan; others exact
    idx, dist, _ = nbm.knn_device(torch.from_numpy(X).cuda(), 90)
    assert int(idx.min()) >= 0 and int(idx.max()) < X.shape[0]


def test_several_samples():
    import torch
    X, off, _ = synth.batch_samples(3, seed=5, d=20, sizes=[700, 1_500, 3_100])
    Xd = torch.from_numpy(X).cuda()
    bk = batch.BatchedKnn(off, 20, 100)
    idx, dist = bk.run(Xd)
    bk.check()
    for a, b in zip(off[:-1], off[1:]):
        ri, _, rd = oracle.knn_exact(X[a:b], 100)
        np.testing.assert_array_equal(idx[a:b].cpu().numpy(), (ri + a).astype(np.int32))
        np.testing.assert_array_equal(dist[a:b].cpu().numpy(), rd)
