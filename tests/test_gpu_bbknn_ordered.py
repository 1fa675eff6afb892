"""The ordered batch-balanced scan (locality order, near pass, pruned key tiles, all batches in one
launch) gives the lists of the batch-by-batch scan and of the oracle: uneven and empty-ish batches,
noise cells, coincident cells, more batches than a launch holds, both candidate precisions."""
import os

import numpy as np
import pytest

from oracle import bbknn as obb
from msc_b200 import bbknn as bbm, synth, _lib

pytestmark = pytest.mark.gpu


def lists(X, batch, kwb, precision, least):
    import torch
    os.environ["MSC_B200_BB_ORDER"] = str(least)
    try:
        _, codes, counts = bbm.batch_codes(batch)
        res = bbm.bbknn_device(torch.from_numpy(X).cuda(), torch.from_numpy(codes).cuda(), counts,
                               kwb, precision=precision)
        torch.cuda.synchronize()
    finally:
        del os.environ["MSC_B200_BB_ORDER"]
    st = res["stats"].cpu().numpy()
    assert int(st[_lib.STAT_TIMEOUT]) == 0 and int(st[_lib.STAT_NONFINITE]) == 0
    return res["knn_idx"].cpu().numpy(), res["knn_dist"].cpu().numpy(), st


def case(name):
    rng = np.random.default_rng(7)
    if name == "noise":
        X = synth.gaussian_mixture(20_001, 50, 12, seed=1, sizes="lognormal", noise_frac=0.01)
        return X, rng.integers(0, 5, X.shape[0]), 3
    if name == "uneven":
        X = synth.gaussian_mixture(9_000, 30, 9, seed=2, sizes="lognormal", noise_frac=0.02)
        return X, rng.choice(4, X.shape[0], p=[0.9, 0.0975, 0.002, 0.0005]), 6
    if name == "many_batches":
        X = synth.gaussian_mixture(3_000, 12, 5, seed=3)
        return X, rng.integers(0, 33, X.shape[0]), 3
    if name == "by_batch":                       # a batch of its own region, far from the others
        X = synth.gaussian_mixture(4_500, 64, 6, seed=4)
        b = np.repeat([0, 1, 2], 1_500)
        X[b == 2] += 30.0
        return X, b, 4
    X = rng.standard_normal((3_000, 20)).astype(np.float32)
    X[2_000:2_300] = X[:300]                     # coincident cells in two batches
    X[500:600] = X[500]
    return X, np.repeat([0, 1, 2], 1_000), 5


@pytest.mark.parametrize("name,precision", [("noise", "fp16"), ("noise", "bf16x3"),
                                            ("uneven", "fp16"), ("many_batches", "fp16"),
                                            ("by_batch", "fp16"), ("coincident", "fp16")])
def test_ordered_scan_equals_plain_scan_and_oracle(name, precision):
    X, batch, kwb = case(name)
    oi, od, st = lists(X, batch, kwb, precision, 0)
    pi, pd, _ = lists(X, batch, kwb, precision, -1)
    np.testing.assert_array_equal(oi, pi, err_msg="ordered vs batch by batch: indices")
    np.testing.assert_array_equal(od, pd, err_msg="ordered vs batch by batch: distances")
    nb = np.unique(batch).size
    assert int(st[_lib.STAT_CERTIFIED]) + int(st[_lib.STAT_RESCANNED]) == X.shape[0] * nb
    if X.shape[0] <= 9_000:
        _, _, _, inter = obb.bbknn(X, batch, kwb, n_pcs=None)   # every column, as the device call
        np.testing.assert_array_equal(oi, inter["idx"].astype(np.int32))
        np.testing.assert_array_equal(od, inter["dist"])
