"""Which path a call takes, and that the paths beside the default one give the same lists.

Samples up to 57,344 cells take the full scan.  The locality order, near pass, pruning plan, merge of
two column halves and flag-based refine pass run below that too when the full scan is switched off
(MSC_B200_DENSE=0), at sizes whose every list the oracle can check.  Lists of more than 65
neighbours and the main scan's long items are counted by the pipeline counters: a search that fell
through to the FP64 scan, or split nothing, would give the same lists."""
import ctypes

import numpy as np
import pytest

import oracle
from msc_b200 import _lib, batch, neighbors as nbm, synth

pytestmark = pytest.mark.gpu

LONG_ITEMS, FAR_KEPT, FAR_ALL, WIDE_ROWS = 15, 10, 11, 64


def counters(call):
    import torch
    lib = _lib.load()
    lib.msc_profile_enable(1)
    try:
        call()
        torch.cuda.synchronize()
        c = (ctypes.c_ulonglong * 65)()
        _lib.check(lib.msc_profile_counters(c, 65))
    finally:
        lib.msc_profile_enable(0)
    return list(c)


def knn(X, k, **kw):
    import torch
    idx, dist, st = nbm.knn_device(torch.from_numpy(X).cuda(), k, **kw)
    torch.cuda.synchronize()
    assert int(st[_lib.STAT_TIMEOUT]) == 0
    return idx.cpu().numpy(), dist.cpu().numpy(), st.cpu().numpy()


@pytest.mark.parametrize("n,d,c,noise,k,metric", [
    (50_000, 30, 25, 0.03, 30, "euclidean"), (40_000, 50, 20, 0.00, 15, "cosine")])
def test_pruned_below_the_full_scans_line(n, d, c, noise, k, metric, monkeypatch):
    X = synth.gaussian_mixture(n, d, c, seed=11, sizes="lognormal", noise_frac=noise,
                               normalize=metric == "cosine")
    full = knn(X, k, metric=metric)
    monkeypatch.setenv("MSC_B200_DENSE", "0")
    pruned = knn(X, k, metric=metric)
    monkeypatch.setenv("MSC_B200_PRUNE", "0")
    plain = knn(X, k, metric=metric)
    monkeypatch.delenv("MSC_B200_PRUNE")
    for other in (full, plain):
        np.testing.assert_array_equal(pruned[0], other[0])
        np.testing.assert_array_equal(pruned[1], other[1])
    rows = np.sort(np.random.default_rng(5).choice(n, 1500, replace=False))
    ri, _, rd = oracle.knn_exact(X, k, metric=metric, rows=rows)
    np.testing.assert_array_equal(pruned[0][rows], ri.astype(np.int32))
    np.testing.assert_array_equal(pruned[1][rows], rd)
    cnt = counters(lambda: knn(X, k, metric=metric))
    assert 0 < cnt[FAR_ALL] and cnt[FAR_KEPT] < 0.6 * cnt[FAR_ALL]


@pytest.mark.parametrize("precision,kprime", [("bf16x3", 0), ("fp16", 32), ("bf16x3", 48)])
def test_tile_configs_under_the_plan(precision, kprime, monkeypatch):
    """Four and eight epilogue warps, single CTAs and pairs, with near-pass lists and masks."""
    X = synth.gaussian_mixture(20_000, 50, 2, seed=23)
    ri, _, rd = oracle.knn_exact(X, 15)
    monkeypatch.setenv("MSC_B200_DENSE", "0")
    tried = 0
    for code in (batch.tile_code(256, 4, 16, 4), batch.tile_code(256, 2, 16, 8),
                 batch.tile_code(128, 4, 16, 8), batch.tile_code(64, 3, 32, 8),
                 batch.tile_code(256, 5, 16, 8, 1), batch.tile_code(256, 4, 32, 4, 1)):
        monkeypatch.setenv("MSC_B200_TILE_CONFIG", hex(code))
        try:
            idx, dist, _ = knn(X, 15, precision=precision, kprime=kprime)
        except ValueError:
            continue                     # the configuration does not fit this operand width
        tried += 1
        np.testing.assert_array_equal(idx, ri.astype(np.int32), err_msg=hex(code))
        np.testing.assert_array_equal(dist, rd, err_msg=hex(code))
    assert tried >= (3 if kprime <= 32 else 1)


@pytest.mark.parametrize("precision,kprime", [("fp16", 0), ("bf16", 14), ("fp16", 14)])
def test_flagged_refine_pass(precision, kprime, monkeypatch):
    X = synth.gaussian_mixture(30_000, 50, 12, seed=31, sizes="lognormal")
    monkeypatch.setenv("MSC_B200_DENSE", "0")
    idx, dist, st = knn(X, 15, precision=precision, kprime=kprime)
    assert int(st[_lib.STAT_RESCANNED]) <= int(st[_lib.STAT_REFINED])
    assert kprime == 0 or int(st[_lib.STAT_REFINED]) > 0
    ri, _, rd = oracle.knn_exact(X, 15)
    np.testing.assert_array_equal(idx, ri.astype(np.int32))
    np.testing.assert_array_equal(dist, rd)


@pytest.mark.parametrize("n,d,k", [(512, 20, 70), (513, 20, 70), (4_000, 30, 83), (9_000, 17, 300),
                                   (20_000, 20, 100)])
def test_wide_lists_are_not_scanned(n, d, k):
    """512 cells: the sample is every key; 513: every key but one.  Rows whose list is exactly as
    long as its window (k - 1 = 128, 256, 512) are left to the scan by any near tie, so not here."""
    X = synth.gaussian_mixture(n, d, 7, seed=n + k, sizes="lognormal", noise_frac=0.01)
    got = []
    cnt = counters(lambda: got.append(knn(X, k)))
    idx, dist, st = got[0]
    assert int(st[_lib.STAT_RESCANNED]) == n
    assert n - cnt[WIDE_ROWS] <= n // 100
    ri, _, rd = oracle.knn_exact(X, k)
    np.testing.assert_array_equal(idx, ri.astype(np.int32))
    np.testing.assert_array_equal(dist, rd)


def test_long_items_are_those_of_outliers():
    rng = np.random.default_rng(9)
    n, d = 150_000, 30
    centres = rng.normal(0, 6, (60, d))
    X = centres[rng.integers(0, 60, n)] + rng.normal(0, 1, (n, d))
    out = rng.choice(n, 1_500, replace=False)
    X[out] = rng.normal(0, 7, (out.size, d))             # a dozen tiles that visit most keys
    assert counters(lambda: knn(X.astype(np.float32), 15))[LONG_ITEMS] >= 1


def test_no_item_is_long_where_all_visit_every_tile():
    """30 uniform dimensions: no tile can be pruned, so every item costs the same."""
    import torch
    X = torch.from_numpy(np.random.default_rng(1).random((31_382, 30)).astype(np.float32)).cuda()
    plan = batch.BatchedKnn(np.array([0, X.shape[0]], np.int64), 30, 13)
    cnt = counters(lambda: plan.run(X))
    plan.check()
    assert cnt[FAR_KEPT] > 0 and cnt[LONG_ITEMS] == 0
