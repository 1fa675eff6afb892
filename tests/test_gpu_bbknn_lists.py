"""Candidate lists of the batch-balanced search, long enough that its certificate holds for every
cell of ordinary data (a cell it leaves open takes an FP64 scan of the batch): plain and ordered
sizes, one-term and three-term operands."""
import numpy as np
import pytest

from msc_b200 import _lib, bbknn as bbm, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,batches,kwb,precision,clusters,seed", [
    (24_000, 50, 2, 7, "fp16", 8, 2),
    (70_000, 30, 3, 8, "fp16", 20, 1),
    (4_000, 50, 6, 3, "bf16", 20, 1),
    (70_000, 30, 3, 8, "bf16x3", 4, 2),
])
def test_every_cell_is_certified(n, d, batches, kwb, precision, clusters, seed):
    import torch
    X = synth.gaussian_mixture(n, d, clusters, seed=seed, sizes="lognormal", noise_frac=0.01)
    _, codes, counts = bbm.batch_codes(np.random.default_rng(seed).integers(0, batches, n))
    res = bbm.bbknn_device(torch.from_numpy(X).cuda(), torch.from_numpy(codes).cuda(), counts, kwb,
                           precision=precision)
    st = res["stats"].cpu().numpy()
    assert int(st[_lib.STAT_RESCANNED]) == 0
    assert int(st[_lib.STAT_CERTIFIED]) == n * batches
