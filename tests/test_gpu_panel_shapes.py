"""BVMult and BVMultInPlace at the edges of the row-panel product's tiles, against numpy.

Edges: 8-column tiles of Q (fewer than four and more take different numbers of warps), rows around a panel of 64
and around the panels of one block, depths around a step of 16, widths where one, two or three blocks fit on an SM,
leading columns (l > 0), the previous values of Y (beta).  Bound: a sum of k products, scaled and added to beta Y,
is within (k + 4) 2^-53 of the sum of the magnitudes, on each side.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (63, 8, 8), (64, 15, 9), (65, 16, 16), (130, 17, 24), (1000, 33, 25), (4097, 48, 31), (9537, 48, 33),
         (9473, 80, 56), (20011, 100, 64), (28501, 20, 12), (28417, 12, 5), (777, 64, 97), (640, 40, 128)]


@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-1.5, 1.0), (0.5, -0.75)])
@pytest.mark.parametrize("n,k,m", SIZES)
def test_mult_shapes(b200, n, k, m, alpha, beta):
    rng = np.random.default_rng([n, k, m])
    l = 2
    X, Y, Q = (rng.standard_normal(s) for s in ((n, k + l), (n, m), (k + l, m)))
    bx, by = b200.BV().create(n, k + l), b200.BV().create(n, m)
    bx.setColumns(X)
    by.setColumns(Y)
    bx.setActiveColumns(l, k + l)
    by.mult(alpha, beta, bx, Q)
    E = alpha * (X[:, l:] @ Q[l:]) + beta * Y
    bound = (k + 4) * 2.0 ** -53 * (abs(alpha) * (np.abs(X[:, l:]) @ np.abs(Q[l:])) + abs(beta) * np.abs(Y))
    assert np.all(np.abs(by.getColumns() - E) <= 2 * bound)


@pytest.mark.parametrize("l", [0, 3])
@pytest.mark.parametrize("n,k,m", [s for s in SIZES if s[2] <= s[1]])
def test_mult_in_place_shapes(b200, n, k, m, l):
    rng = np.random.default_rng([n, k, m])
    V, Q = rng.standard_normal((n, k + l)), rng.standard_normal((k + l, k + l))
    bv = b200.BV().create(n, k + l)
    bv.setColumns(V)
    bv.setActiveColumns(l, k + l)
    bv.multInPlace(Q, l, l + m)
    E = V.copy()
    E[:, l:l + m] = V[:, l:] @ Q[l:, l:l + m]
    bound = np.zeros_like(E)
    bound[:, l:l + m] = (k + 4) * 2.0 ** -53 * (np.abs(V[:, l:]) @ np.abs(Q[l:, l:l + m]))
    assert np.all(np.abs(bv.getColumns() - E) <= 2 * bound)
