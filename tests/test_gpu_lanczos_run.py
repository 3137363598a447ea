"""BVMatLanczos in one launch (one cluster, or one CTA per SM) and column by column, against numpy.

Which form runs follows from the rows n and the last column m: up to 16 slices of 32 rows per CTA of a
16-CTA cluster are applied by one warp each, up to 32 by two; then one CTA per SM with up to 16 slices;
larger bases go column by column.  The sizes sit on both sides of those lines, with ragged last slices,
rows longer than the entries held in registers, FP32 values, and rows of no nonzeros.  Reference: Lanczos
with full reorthogonalisation in numpy FP64; both are backward stable and no Ritz value converges in these
runs, so they differ by rounding (1e-10, as the three-term check of test_gpu_kernels.py allows).
"""
import numpy as np
import pytest

from slepc_b200 import problems as P

pytestmark = pytest.mark.gpu


def _matrix(kind, n):
    if kind == "lap":
        csr = P.laplacian_2d(n, 1) if n < 64 else P.laplacian_2d(n // 8, 8)
        return csr
    rng = np.random.default_rng(n)  # banded, 0 to 21 entries a row (more than are held in registers), symmetric
    import scipy.sparse as sp

    offs = [0, 1, 2, 3, 5, 8, 13, 21, 34, 55, 89]
    A = sp.diags([rng.standard_normal(n - o) * (rng.random(n - o) < 0.8) for o in offs], offs, format="csr")
    A = (A + A.T).tocsr()
    A.eliminate_zeros()
    A.sort_indices()
    return A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data


def _numpy_run(csr, v, m):
    A = P.to_scipy(csr)
    V = np.zeros((len(v), m + 1))
    V[:, 0] = v / np.linalg.norm(v)
    alpha, beta = np.zeros(m), np.zeros(m)
    for j in range(m):
        w = A @ V[:, j]
        h = np.zeros(j + 1)
        for _ in range(2):
            c = V[:, : j + 1].T @ w
            w = w - V[:, : j + 1] @ c
            h += c
        alpha[j], beta[j] = h[j], np.linalg.norm(w)
        V[:, j + 1] = w / beta[j]
    return alpha, beta, V


CASES = [("lap", 40, 6, 0, False), ("lap", 504, 9, 3, False), ("lap", 8200, 12, 0, False), ("lap", 9000, 33, 8, False),
         ("lap", 16384, 10, 2, False), ("lap", 16424, 10, 2, False), ("lap", 20008, 40, 5, False),
         ("lap", 75776, 20, 0, False), ("lap", 76000, 6, 0, False), ("band", 301, 20, 0, False),
         ("band", 12001, 9, 4, False), ("band", 30011, 12, 0, False), ("band", 5003, 15, 2, True),
         ("band", 33333, 7, 0, True), ("lap", 1000, 100, 60, False)]


@pytest.mark.parametrize("kind,n,m,k,f32", CASES)
def test_run_matches_numpy(b200, kind, n, m, k, f32):
    csr = _matrix(kind, n)
    n = len(csr[0]) - 1
    vals = csr[2].astype(np.float32).astype(np.float64) if f32 else csr[2]
    csr = (csr[0], csr[1], vals)
    A = b200.Mat().createAIJ(csr, size=(n, n), dtype=np.float32) if f32 else b200.Mat().createAIJ(csr)
    v0 = P.start_vector(n, 4)
    alpha, beta, V = _numpy_run(csr, v0, m)
    bv = b200.BV().create(n, m + 1)
    bv.setColumn(0, v0)
    bv.orthonormalizeColumn(0)
    if k:
        bv.matLanczos(A, 0, k)
    a, b, mm, last, bd = bv.matLanczos(A, k, m)
    assert mm == m and not bd
    scale = max(np.abs(alpha).max(), beta.max())
    np.testing.assert_allclose(a[k:m], alpha[k:], rtol=0, atol=1e-10 * scale)
    np.testing.assert_allclose(b[k:m], beta[k:], rtol=0, atol=1e-10 * scale)
    np.testing.assert_allclose(last, beta[-1], rtol=0, atol=1e-10 * scale)
    G = bv.getColumns()
    np.testing.assert_allclose(G, V, rtol=0, atol=1e-10)
    # the same run again on the same basis gives the same bits
    a2, b2, *_ = bv.matLanczos(A, k, m)
    np.testing.assert_array_equal(a2, a)
    np.testing.assert_array_equal(b2, b)
    np.testing.assert_array_equal(bv.getColumns(), G)


@pytest.mark.parametrize("n", [64, 9000, 30000, 90000])
def test_run_stops_at_an_invariant_subspace(b200, n):
    """A diagonal operator started on a coordinate vector: w - v (v'w) is exactly zero at the first step."""
    i = np.arange(n, dtype=np.int32)
    csr = (np.arange(n + 1, dtype=np.int32), i, 1.0 + i)
    A = b200.Mat().createAIJ(csr)
    bv = b200.BV().create(n, 8)
    e = np.zeros(n)
    e[5] = 1.0
    bv.setColumn(0, e)
    for _ in range(2):  # a run after a stopped one starts afresh
        a, b, m, last, bd = bv.matLanczos(A, 0, 7)
        assert bd and m == 1 and last == 0.0
        assert a[0] == 6.0 and b[0] == 0.0
