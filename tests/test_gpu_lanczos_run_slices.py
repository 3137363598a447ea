"""Whole Lanczos runs of one CTA per SM with every number of 32-row slices to a CTA.

A CTA of 16 warps takes 1 to 16 slices.  Up to 8 several warps share a slice; from 9 on a warp owns a whole
slice and the warps past the last one have none, so every row must still be updated and scaled exactly once.
The sizes follow from the SM count: spc slices to a CTA with a ragged last slice.  References and tolerances
are those of test_gpu_lanczos_run.py; the eigenvalues of a grid Laplacian are known, and a pair with residual
norm tol |theta| has an eigenvalue within tol |theta| of theta.
"""
import numpy as np
import pytest

from slepc_b200 import problems as P
from tests.test_gpu_lanczos_run import _matrix, _numpy_run

pytestmark = pytest.mark.gpu


def _rows(spc):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return 32 * sms * (spc - 1) + 32 * (sms // 2) + 8


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("kind,m,k", [("band", 11, 0), ("lap", 44, 6)])
@pytest.mark.parametrize("spc", [8, 9, 10, 11, 12, 13, 14, 15])
def test_slices_per_cta(b200, spc, kind, m, k, f32):
    csr = _matrix(kind, _rows(spc))
    n = len(csr[0]) - 1
    csr = (csr[0], csr[1], csr[2].astype(np.float32).astype(np.float64)) if f32 else csr
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
    G = bv.getColumns()
    np.testing.assert_allclose(G, V, rtol=0, atol=1e-10)
    for _ in range(3):  # the same run on the same basis gives the same bits
        a2, b2, *_ = bv.matLanczos(A, k, m)
        np.testing.assert_array_equal(a2, a)
        np.testing.assert_array_equal(b2, b)
        np.testing.assert_array_equal(bv.getColumns(), G)


@pytest.mark.parametrize("spc", [9, 15])
def test_stops_at_an_invariant_subspace(b200, spc):
    n = _rows(spc)
    i = np.arange(n, dtype=np.int32)
    A = b200.Mat().createAIJ((np.arange(n + 1, dtype=np.int32), i, 1.0 + i))
    bv = b200.BV().create(n, 8)
    e = np.zeros(n)
    e[5] = 1.0
    bv.setColumn(0, e)
    for _ in range(2):
        a, b, m, last, bd = bv.matLanczos(A, 0, 7)
        assert bd and m == 1 and last == 0.0
        assert a[0] == 6.0 and b[0] == 0.0


def test_solve_of_a_grid_laplacian(b200):
    N, nev, tol = 200, 4, 1e-8
    A = b200.Mat().createAIJ(P.laplacian_2d(N, N))
    eps = b200.EPS().create()
    eps.setOperators(A)
    eps.setDimensions(nev, 40)
    eps.setTolerances(tol, 10000)
    eps.solve()
    assert eps.getConverged() >= nev
    s = 4 * np.sin(np.arange(1, N + 1) * np.pi / (2 * (N + 1))) ** 2
    exact = np.sort((s[:, None] + s[None, :]).ravel())[::-1]
    got = np.array([eps.getEigenvalue(i) for i in range(nev)])
    assert abs(got[0] - exact[0]) <= tol * exact[0]
    for v in got:
        assert np.abs(exact - v).min() <= tol * v
    _, x = eps.getEigenpair(0)
    i = np.arange(1, N + 1) * np.pi * N / (N + 1)
    y = np.outer(np.sin(i), np.sin(i)).ravel()
    # sine of the angle <= residual / gap to the next eigenvalue
    cos = abs(x @ y) / (np.linalg.norm(x) * np.linalg.norm(y))
    assert np.sqrt(max(0.0, 1.0 - cos * cos)) <= tol * exact[0] / (exact[0] - exact[1]) + 1e-7
