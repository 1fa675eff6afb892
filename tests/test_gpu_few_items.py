"""Samples of fewer work items than the GPU has CTAs: their items are alike, so none is scanned in
parts, whose lists start empty.  Counted by the insertions of the main scan: a list that starts
with a row's k' nearest of one 256-key tile takes at most k' more for every e-fold of keys, in
any order that does not favour far keys first."""
import ctypes
import math

import numpy as np
import pytest

from msc_b200 import _lib, batch, synth

pytestmark = pytest.mark.gpu


def insertions(X, k):
    import torch
    lib = _lib.load()
    plan = batch.BatchedKnn(np.array([0, X.shape[0]], np.int64), X.shape[1], k)
    lib.msc_profile_enable(1)
    try:
        plan.run(torch.from_numpy(X).cuda())
        torch.cuda.synchronize()
        c = (ctypes.c_ulonglong * 64)()
        _lib.check(lib.msc_profile_counters(c, 64))
    finally:
        lib.msc_profile_enable(0)
    plan.check()
    return c[16 + 16 + 8]                                # appends of the main scan


@pytest.mark.parametrize("n,d", [(31_382, 30), (12_000, 20), (60_000, 40)])
def test_alike_items_are_not_split(n, d):
    X = np.random.default_rng(n).random((n, d)).astype(np.float32)
    kprime = 48
    assert insertions(X, 13) <= n * kprime * (1 + math.log(n / 256))


def test_clustered_sample():
    X = synth.gaussian_mixture(20_000, 30, 10, seed=3, sizes="lognormal", noise_frac=0.01)
    assert insertions(X, 15) <= 20_000 * 48 * (1 + math.log(20_000 / 256))
