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


@pytest.mark.parametrize("least", ["0", "-1"])               # in locality order, batch by batch
@pytest.mark.parametrize("n,batches,kwb,lone", [
    (3_000, 2, 5, 1), (3_001, 3, 3, 7), (2_000, 1, 30, 20), (2_700, 3, 1, 300), (2_000, 1, 47, 3)])
def test_few_scanned_cells(n, batches, kwb, lone, least, monkeypatch):
    """Fewer cells to scan than blocks, each by a block whose warps split the batch: cells whose
    nearest others are closer together than the operands tell, against the oracle."""
    import torch
    from oracle import bbknn as obb
    rng = np.random.default_rng(n + lone)
    X = rng.normal(0, 5, (n, 20)).astype(np.float32)
    for c in range(lone):                                # rings of cells around a centre of their own
        ring = slice(c * 6, c * 6 + 6)
        X[ring] = rng.normal(0, 5, 20) + 1e-4 * rng.normal(size=(6, 20))
    batch = rng.integers(0, batches, n)
    monkeypatch.setenv("MSC_B200_BB_ORDER", least)
    _, codes, counts = bbm.batch_codes(batch)
    r = bbm.bbknn_device(torch.from_numpy(X).cuda(), torch.from_numpy(codes).cuda(), counts, kwb,
                         precision="fp16")
    _, _, _, inter = obb.bbknn(X, batch, kwb, n_pcs=None)
    np.testing.assert_array_equal(r["knn_idx"].cpu().numpy(), inter["idx"].astype(np.int32))
    np.testing.assert_array_equal(r["knn_dist"].cpu().numpy(), inter["dist"])


@pytest.mark.parametrize("least", ["0", "-1"])
def test_a_handful_of_scanned_cells(least, monkeypatch):
    import torch
    monkeypatch.setenv("MSC_B200_BB_ORDER", least)
    X = synth.gaussian_mixture(24_000, 50, 8, seed=2, sizes="lognormal", noise_frac=0.01)
    _, codes, counts = bbm.batch_codes(np.random.default_rng(2).integers(0, 2, X.shape[0]))
    got = {}
    for precision in ("bf16", "bf16x3"):                 # hundreds of cells scanned, and none
        r = bbm.bbknn_device(torch.from_numpy(X).cuda(), torch.from_numpy(codes).cuda(), counts, 2,
                             precision=precision)
        got[precision] = r["knn_idx"].cpu().numpy(), r["knn_dist"].cpu().numpy()
    np.testing.assert_array_equal(got["bf16"][0], got["bf16x3"][0])
    np.testing.assert_array_equal(got["bf16"][1], got["bf16x3"][1])
