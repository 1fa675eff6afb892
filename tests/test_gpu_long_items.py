"""The main scan's longest work items, scanned in parts: samples whose outliers fill whole query
tiles that visit most of the keys.  The full scan of the same cells (no pruning, so no parts) gives
every index and distance; both are exact, so they agree bit for bit."""
import numpy as np
import pytest

from msc_b200 import neighbors as nbm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k,metric,outliers", [
    (60_000, 50, 15, "euclidean", 300),      # parts hold 32 of 48
    (60_000, 50, 50, "euclidean", 129),      # k' = 64, lists of the parts shorter than k - 1
    (60_000, 20, 5, "cosine", 1),            # one outlier in a padded tile
    (70_001, 33, 30, "cosine", 1500),        # odd dimension and size
    (60_000, 50, 15, "euclidean", 20_000),   # many outliers: nothing is long
])
def test_long_items_match_full_scan(n, d, k, metric, outliers, monkeypatch):
    import torch
    rng = np.random.default_rng(n + d + k)
    centres = rng.normal(0, 6, (40, d))
    X = centres[rng.integers(0, 40, n)] + rng.normal(0, 0.4, (n, d))
    X[rng.choice(n, outliers, replace=False)] = rng.normal(0, 7, (outliers, d))
    X = torch.from_numpy(X.astype(np.float32)).cuda()
    got_i, got_d, _ = nbm.knn_device(X, k, metric=metric)
    monkeypatch.setenv("MSC_B200_PRUNE", "0")
    monkeypatch.setenv("MSC_B200_DENSE", "0")
    ref_i, ref_d, _ = nbm.knn_device(X, k, metric=metric)
    assert torch.equal(got_d, ref_d)
    assert torch.equal(got_i, ref_i)
