"""UMAP edge preparation at the edges of its blocks (64 rows, 1,024 entries at a time): row counts
around a block, empty rows, rows longer than a chunk, entries that end exactly at one.  Bit for bit
against the oracle."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import handoff
from msc_b200 import neighbors as nbm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,lengths", [
    (1, "one"), (63, "ragged"), (64, "sixteen"), (65, "ragged"), (128, "sixteen"),
    (3000, "ragged"), (5000, "hub"), (4096, "empty_ends"), (70_001, "ragged")])
def test_umap_edges_at_block_edges(n, lengths):
    import torch
    rng = np.random.default_rng(n)
    if lengths == "one":
        cnt = np.array([1])
    elif lengths == "sixteen":                       # 64 rows of 16: chunks end at row starts
        cnt = np.full(n, 16)
    else:
        cnt = rng.integers(0, min(n, 40), n)
        if lengths == "hub":
            cnt[[0, 63, 64, n // 2]] = [n, 1024, 1025, 3000]
        if lengths == "empty_ends":
            cnt[:130] = 0
            cnt[-70:] = 0
    indptr = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int64)
    cols = np.concatenate([np.sort(rng.choice(n, c, replace=False)) for c in cnt]).astype(np.int32)
    w = np.maximum(rng.random(len(cols)).astype(np.float32) ** 4, np.float32(1e-6))
    conn = sp.csr_matrix((w, cols, indptr), shape=(n, n))
    res = {"conn_indptr": torch.from_numpy(indptr).cuda(),
           "conn_indices": torch.from_numpy(cols).cuda(),
           "conn_data": torch.from_numpy(w).cuda()}
    got = nbm.umap_edges(res, n, 200)
    ref = handoff.umap_edges(conn, 200)
    for key in ("indptr", "rows", "cols", "weights", "epochs_per_sample"):
        np.testing.assert_array_equal(got[key].cpu().numpy(), ref[key], err_msg=key)
