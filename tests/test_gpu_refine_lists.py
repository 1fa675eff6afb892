"""The refine pass of the full scan keeps lists long enough for the rows that come to it, whose k-th
place is crowded (wide rows, many neighbours): they are certified there instead of each taking the
FP64 scan of every key.  k = 22 is the last with lists of 32, beyond 50 dimensions k = 17."""
import numpy as np
import pytest

import oracle
from msc_b200 import neighbors as nbm, synth, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k,precision", [
    (20_000, 128, 30, "fp16"), (20_506, 128, 25, "bf16"), (6_641, 128, 25, "bf16"),
    (12_000, 128, 33, "fp16"), (40_000, 128, 17, "bf16"), (40_000, 128, 18, "bf16"),
    (40_000, 128, 19, "bf16"), (40_000, 50, 22, "bf16"), (40_000, 50, 23, "bf16"),
    (15_000, 51, 19, "fp16")])
def test_refined_rows_are_certified(n, d, k, precision):
    import torch
    X = synth.gaussian_mixture(n, d, 20, seed=1, sizes="lognormal", noise_frac=0.01)
    Xd = torch.from_numpy(X).cuda()
    idx, dist, st = nbm.knn_device(Xd, k, precision=precision)
    assert int(st[_lib.STAT_RESCANNED]) == 0
    assert int(st[_lib.STAT_CERTIFIED]) == n
    rows = np.sort(np.random.default_rng(2).choice(n, 500, replace=False))
    ri, _, rd = oracle.knn_exact(X, k, rows=rows)
    np.testing.assert_array_equal(idx.cpu().numpy()[rows], ri.astype(np.int32))
    np.testing.assert_array_equal(dist.cpu().numpy()[rows], rd)
