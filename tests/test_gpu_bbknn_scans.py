"""FP64 scans of the ordered batch-balanced search: cells that its certificate leaves open (BF16
operands of cells far from the mean), in one group of batches, in two, and in batches of a few cells.
The batch-by-batch search scans the same cells over lists in another order; both are exact."""
import numpy as np
import pytest

from msc_b200 import _lib, bbknn as bbm, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,batches,kwb", [
    (6_001, 25, 3, 9), (7_000, 30, 70, 1), (5_000, 50, 9, 4)])
def test_scanned_cells(n, d, batches, kwb, monkeypatch):
    import torch
    rng = np.random.default_rng(n)
    X = synth.gaussian_mixture(n, d, 6, seed=n, noise_frac=0.01)
    X[: n // 2] += 60.0                                  # two halves: no centring helps both
    batch = rng.integers(0, batches, n)
    batch[:batches] = np.arange(batches)
    if batches == 9:
        batch[batch == 8] = 7                            # a batch of 12 cells among large ones
        batch[100:112] = 8
    _, codes, counts = bbm.batch_codes(batch)
    got = []
    for least in ("0", "-1"):
        monkeypatch.setenv("MSC_B200_BB_ORDER", least)
        r = bbm.bbknn_device(torch.from_numpy(X).cuda(), torch.from_numpy(codes).cuda(), counts,
                             kwb, precision="bf16")
        got.append((r["knn_idx"].cpu().numpy(), r["knn_dist"].cpu().numpy(),
                    r["stats"].cpu().numpy()))
    np.testing.assert_array_equal(got[0][0], got[1][0])
    np.testing.assert_array_equal(got[0][1], got[1][1])
    st = got[0][2]
    assert int(st[_lib.STAT_RESCANNED]) > 0
    assert int(st[_lib.STAT_CERTIFIED]) + int(st[_lib.STAT_RESCANNED]) == n * counts.size
