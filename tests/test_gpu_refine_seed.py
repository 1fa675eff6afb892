"""The refine pass below the bounds that the main scan leaves: rows that the one-term candidates
cannot certify (neighbours closer together than the 16-bit operands tell), few enough to be split
and too many for it, with and without outlier tiles scanned in parts.  The full scan of the
same cells gives every index and distance; both are exact, so they agree bit for bit."""
import numpy as np
import pytest

from msc_b200 import _lib, neighbors as nbm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k,tight,outliers", [
    (60_000, 50, 15, 500, 200),        # a few hundred rows: split over eight parts
    (60_000, 50, 15, 40_000, 200),     # more than the parts' buffers take: not split
    (60_001, 31, 40, 3000, 0),         # odd dimension, k' = 64
])
def test_refine_rows_match_full_scan(n, d, k, tight, outliers, monkeypatch):
    import torch
    rng = np.random.default_rng(n + tight)
    centres = rng.normal(0, 8, (30, d))
    c = rng.integers(0, 30, n)
    X = centres[c] + rng.normal(0, 0.5, (n, d))
    X[:tight] = centres[c[:tight]] + rng.normal(0, 1e-3, (tight, d))   # closer than the operands tell
    if outliers:
        X[-outliers:] = rng.normal(0, 9, (outliers, d))
    X = torch.from_numpy(X.astype(np.float32)).cuda()
    got_i, got_d, st = nbm.knn_device(X, k)
    assert int(st[_lib.STAT_REFINED]) > 0
    monkeypatch.setenv("MSC_B200_PRUNE", "0")
    monkeypatch.setenv("MSC_B200_DENSE", "0")
    ref_i, ref_d, _ = nbm.knn_device(X, k)
    assert torch.equal(got_d, ref_d)
    assert torch.equal(got_i, ref_i)
