"""Products whose rows are of mixed lengths (slices, warp tiles and segments in one launch), against numpy.

Edges: rows at the limits of a slice (32 nonzeros), of a tile (256) and of a segment (1024, several per row), rows
without nonzeros, a last slice that is not full, matrices of one kind of row only, FP32 values; several products of
one matrix, since the counts of finished segments go back to zero.  Bound: a row of r nonzeros is within
(r + 2) 2^-53 of the sum of the magnitudes, on each side (products and sums are FP64 for FP32 values too).
"""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

LENGTHS = {
    "mixed": [0, 1, 31, 32, 33, 255, 256, 257, 1023, 1024, 1025, 4096, 5000, 2, 0, 40, 41, 42, 7] * 3,
    "long": [1500, 3000, 1024, 1025, 257],
    "tiles": [33, 100, 200, 256, 64] * 9,
    "one long of many": [3] * 1000 + [40000] + [5] * 333,
}


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_many_segments(b200, dtype):
    """More segments than two per resident warp: their sum is a launch of its own."""
    import torch

    rng = np.random.default_rng(3)
    m, n = 23, 600001
    rowptr = (np.arange(m + 1) * n).astype(np.int32)
    vals = rng.standard_normal((m, n)).astype(dtype)
    A = b200.Mat().createAIJ((rowptr, np.tile(np.arange(n, dtype=np.int32), m), vals.ravel()), size=(m, n), dtype=dtype)
    V = vals.astype(np.float64)
    for _ in range(2):
        x = rng.standard_normal(n)
        xd = torch.from_numpy(x).cuda()
        yd = torch.full((m,), np.nan, dtype=torch.float64, device="cuda")
        A.mult(xd.data_ptr(), yd.data_ptr())
        torch.cuda.synchronize()
        assert np.all(np.abs(yd.cpu().numpy() - V @ x) <= 2 * (n + 2) * 2.0 ** -53 * (np.abs(V) @ np.abs(x)))


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("name", sorted(LENGTHS))
def test_mixed_rows(b200, name, dtype):
    import torch

    rng = np.random.default_rng(len(name))
    lens = np.array(LENGTHS[name])
    m, n = len(lens), 45000
    rowptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    colind = np.concatenate([np.sort(rng.choice(n, r, replace=False)) for r in lens]).astype(np.int32)
    vals = rng.standard_normal(len(colind)).astype(dtype)
    E = sp.csr_matrix((vals.astype(np.float64), colind, rowptr), shape=(m, n))
    A = b200.Mat().createAIJ((rowptr, colind, vals), size=(m, n), dtype=dtype)
    for _ in range(3):
        for M, mult, cols, rows in ((E, A.mult, n, m), (E.T.tocsr(), A.multTranspose, m, n)):
            x = rng.standard_normal(cols)
            xd = torch.from_numpy(x).cuda()
            yd = torch.full((rows,), np.nan, dtype=torch.float64, device="cuda")
            mult(xd.data_ptr(), yd.data_ptr())
            torch.cuda.synchronize()
            bound = (np.diff(M.indptr) + 2) * 2.0 ** -53 * (abs(M) @ np.abs(x))
            assert np.all(np.abs(yd.cpu().numpy() - M @ x) <= 2 * bound)
