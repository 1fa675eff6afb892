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


@pytest.mark.parametrize("scale", SCALES)
@pytest.mark.parametrize("precision", ["fp16", "bf16x3", "bf16", "fp32"])
def test_candidate_lists(precision, scale):
    assert_lists(cells(scale), 15, precision=precision)


@pytest.mark.parametrize("scale", [1e-20, 1e-21, 1e-22])
def test_pruned_scan(scale):
    import torch
    X = synth.gaussian_mixture(60_000, 50, 40, seed=11, sizes="lognormal", noise_frac=0.01)
    X = (X.astype(np.float64) * scale).astype(np.float32)
    idx, dist, _ = nbm.knn_device(torch.from_numpy(X).cuda(), 15)
    rows = np.sort(np.random.default_rng(5).choice(X.shape[0], 1_000, replace=False))
    ri, _, rd = oracle.knn_exact(X, 15, rows=rows)
    np.testing.assert_array_equal(idx.cpu().numpy()[rows], ri.astype(np.int32))
    np.testing.assert_array_equal(dist.cpu().numpy()[rows], rd)


@pytest.mark.parametrize("scale", SCALES)
@pytest.mark.parametrize("precision", ["fp16", "bf16x3"])
@pytest.mark.parametrize("least", ["-1", "0"])               # batch by batch, in locality order
def test_batch_balanced_lists(least, precision, scale, monkeypatch):
    import torch
    from oracle import bbknn as obb
    from msc_b200 import bbknn as bbm
    monkeypatch.setenv("MSC_B200_BB_ORDER", least)
    X, batch = cells(scale), np.random.default_rng(1).integers(0, 3, 1_500)
    _, codes, counts = bbm.batch_codes(batch)
    res = bbm.bbknn_device(torch.from_numpy(X).cuda(), torch.from_numpy(codes).cuda(), counts, 3,
                           precision=precision)
    _, _, _, inter = obb.bbknn(X, batch, 3, n_pcs=None)
    np.testing.assert_array_equal(res["knn_idx"].cpu().numpy(), inter["idx"].astype(np.int32))
    np.testing.assert_array_equal(res["knn_dist"].cpu().numpy(), inter["dist"])
