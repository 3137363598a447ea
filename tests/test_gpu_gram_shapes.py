"""BVDot at the edges of the Gram kernel's tiles, against numpy.

Edges: 16-column strips of Y (1 to 4, two blocks of 64 above that), 8-column tiles of X, the shared operand of
X = Y, rows around a stage of 32 and around the rows of one block, leading columns (l > 0), products of fewer
than 64 pairs (another kernel).  Bound: the sum of n products in any order is within (n + 2) 2^-53 of the sum
of their magnitudes.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 8, 8), (31, 9, 8), (32, 16, 17), (33, 33, 32), (129, 48, 49), (1000, 64, 64), (4097, 7, 64), (4097, 64, 7),
         (20011, 65, 15), (20011, 15, 66), (40007, 40, 24), (77, 3, 3), (38000, 24, 48)]


@pytest.mark.parametrize("l", [0, 3])
@pytest.mark.parametrize("n,kx,ky", SIZES)
def test_dot_shapes(b200, n, kx, ky, l):
    rng = np.random.default_rng([n, kx, ky])
    X, Y = rng.standard_normal((n, kx + l)), rng.standard_normal((n, ky + l))
    bx, by = b200.BV().create(n, kx + l), b200.BV().create(n, ky + l)
    bx.setColumns(X)
    by.setColumns(Y)
    bx.setActiveColumns(l, kx + l)
    by.setActiveColumns(l, ky + l)
    M = bx.dot(by)[l:, l:]
    E = Y[:, l:].T @ X[:, l:]
    bound = (n + 2) * 2.0 ** -53 * (np.abs(Y[:, l:]).T @ np.abs(X[:, l:]))
    assert np.all(np.abs(M - E) <= 2 * bound)  # both sides round
    np.testing.assert_array_equal(bx.dot(by)[l:, l:], M)


@pytest.mark.parametrize("n,k", [(31, 8), (1000, 16), (20011, 33), (4097, 64), (38000, 48)])
def test_dot_with_itself(b200, n, k):
    X = np.random.default_rng([n, k]).standard_normal((n, k))
    bx = b200.BV().create(n, k)
    bx.setColumns(X)
    M = bx.dot(bx)
    bound = (n + 2) * 2.0 ** -53 * (np.abs(X).T @ np.abs(X))
    assert np.all(np.abs(M - X.T @ X) <= 2 * bound)
