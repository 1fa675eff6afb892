"""Wide lists (k > 65) where many cells coincide, so that more keys than a row's buffer takes lie at
or below any threshold that keeps k: such rows take the FP64 scan, the others do not.  Ties go by index,
as in the oracle."""
import numpy as np
import pytest

import oracle
from msc_b200 import neighbors as nbm, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,n,k", [("all", 3_000, 83), ("most", 4_000, 83), ("half", 2_600, 130),
                                      ("some", 6_000, 83), ("lattice", 5_000, 70)])
def test_coincident_cells(name, n, k):
    import torch
    X = synth.gaussian_mixture(n, 6, 5, seed=n)
    share = {"all": n, "most": n * 9 // 10, "half": n // 2, "some": 1_000}.get(name, 0)
    X[:share] = X[0]
    if name == "lattice":
        X = np.round(X)
    X = X[np.random.default_rng(k).permutation(n)]
    idx, dist, _ = nbm.knn_device(torch.from_numpy(X).cuda(), k)
    rows = np.sort(np.random.default_rng(1).choice(n, 700, replace=False))
    ri, _, rd = oracle.knn_exact(X, k, rows=rows)
    np.testing.assert_array_equal(idx.cpu().numpy()[rows], ri.astype(np.int32))
    np.testing.assert_array_equal(dist.cpu().numpy()[rows], rd)
