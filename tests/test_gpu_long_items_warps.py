"""Parts of long work items with eight epilogue warps: the two column halves of a row keep a list
each, shorter than k', and are merged.  The parts keep their candidates through the merge: next to
four warps (one list a row) the lists are the same, and the rows that the certificate leaves to the
refine pass or the FP64 scan are those of near ties only."""
import numpy as np
import pytest

from msc_b200 import _lib, batch, neighbors as nbm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,kprime,precision", [
    (150_000, 30, 48, "fp16"),           # parts hold 32 of 48
    (150_000, 30, 64, "fp16"),           # ... of 64
    (150_001, 20, 48, "bf16x3"),         # no refine pass: what is left takes the FP64 scan
])
def test_eight_warps_keep_the_parts_candidates(n, d, kprime, precision, monkeypatch):
    import torch
    rng = np.random.default_rng(n + kprime)
    centres = rng.normal(0, 6, (60, d))
    X = centres[rng.integers(0, 60, n)] + rng.normal(0, 1, (n, d))
    out = rng.choice(n, 1_500, replace=False)
    X[out] = rng.normal(0, 7, (out.size, d))             # a dozen tiles that visit most keys
    X = torch.from_numpy(X.astype(np.float32)).cuda()
    got = {}
    for epi, stages in ((4, 4), (8, 2)):
        monkeypatch.setenv("MSC_B200_TILE_CONFIG", hex(batch.tile_code(256, stages, 16, epi)))
        i, dist, st = nbm.knn_device(X, 15, precision=precision, kprime=kprime)
        got[epi] = i, dist, int(st[_lib.STAT_REFINED]) + int(st[_lib.STAT_RESCANNED])
    assert torch.equal(got[8][0], got[4][0])
    assert torch.equal(got[8][1], got[4][1])
    # 1,500 outlier rows fail if their parts' lists are lost
    assert got[8][2] <= got[4][2] + 100
