"""The batched solver's projected problem against dense eigenvalues: magnitudes at which the squares of a rotation's
entries leave the range of the reciprocal square root, every selection of eigenvalues (the sort), the smallest and
the largest projected problem, spectra with pairs of one magnitude.  Bound: a computed pair has a relative
residual of at most tol = 1e-9, which bounds the distance of its value to an eigenvalue; twice that is asked for.
"""
import numpy as np
import pytest

import slepc_b200 as S

pytestmark = pytest.mark.gpu


def _tridiagonal(n, seed, scale, zero_diagonal):
    rng = np.random.default_rng(seed)
    d = np.zeros(n) if zero_diagonal else rng.standard_normal(n) + 3.0 * np.arange(n)
    e = rng.uniform(0.5, 1.5, n - 1) * (np.linspace(4.0, 0.5, n - 1) if zero_diagonal else 1.0)
    A = np.diag(d) + np.diag(e, 1) + np.diag(e, -1)
    rows, cols = np.nonzero((np.abs(np.subtract.outer(np.arange(n), np.arange(n))) <= 1))
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    return A, rowptr.astype(np.int32), cols.astype(np.int32), A[rows, cols] * scale


@pytest.mark.parametrize("which", [S.LARGEST_MAGNITUDE, S.LARGEST_REAL, S.SMALLEST_REAL])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** 480, 2.0 ** -480])
@pytest.mark.parametrize("nev,ncv", [(1, 6), (3, 16), (6, 31)])
def test_projected_problem(b200, which, scale, nev, ncv):
    parts = [_tridiagonal(n, n, scale, z) for n, z in ((40, False), (57, True), (64, False), (90, True))]
    E = S.BatchEPS().create(np.array([len(p[0]) for p in parts], dtype=np.int32), np.concatenate([p[1] for p in parts]),
                            np.concatenate([p[2] for p in parts]), np.concatenate([p[3] for p in parts]))
    E.setDimensions(nev, ncv)
    E.setTolerances(1e-9, 5000)
    E.setWhichEigenpairs(which)
    E.solve()
    ev, info, _ = E.getAll()
    for p, (A, *_) in enumerate(parts):
        assert info[p, 2] == S.CONVERGED_TOL and info[p, 4] == 0 and info[p, 0] >= nev, (p, info[p])
        exact = np.linalg.eigvalsh(A)
        got = ev[p, :nev] / scale
        near = np.abs(np.subtract.outer(got, exact)).min(axis=1)
        assert np.all(near <= 2e-9 * np.abs(got)), p
        key = {S.LARGEST_MAGNITUDE: np.abs(got), S.LARGEST_REAL: got, S.SMALLEST_REAL: -got}[which]
        assert np.all(np.diff(key) <= 2e-9 * np.abs(key[1:])), p  # in the order asked for
