"""The one-launch column orthogonalisation at the edges of its shapes, against the oracle.

Its dispatch has edges in the basis columns j (columns held per lane: multiples of 4 up to 32; warps
that share a row: 1, 2, 4, 8 up to j = 32, 64, 128, 252) and in the rows n (chunks of 256, 128, 64 and
32 rows, one CTA, a ragged last chunk, more chunks than CTAs).  Tolerances are those of
test_orthogonalize_column_vs_oracle: the two sides differ by the order of their sums alone.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 0), (5, 4), (257, 1), (300, 5), (255, 28), (33, 32), (70, 33), (129, 64), (4097, 65), (131, 128),
         (37921, 31), (19000, 63), (9500, 127), (4769, 129), (260, 252), (40001, 12), (38000, 21)]


@pytest.mark.parametrize("normalize", [False, True])
@pytest.mark.parametrize("n,j", SIZES)
def test_column_shapes_vs_oracle(b200, oracle_mod, n, j, normalize):
    rng = np.random.default_rng([n, j])
    V = np.zeros((n, j + 1), order="F")
    if j:
        V[:, :j] = np.linalg.qr(rng.standard_normal((n, j)))[0]
    V[:, j] = (V[:, :j] @ (10 * rng.standard_normal(j)) if j else 0) + 1e-2 * rng.standard_normal(n)
    Vo = V.copy(order="F")
    Ho, no, lo = oracle_mod.bv_orthogonalize_column(Vo, j, normalize=normalize)
    bv = b200.BV().create(n, j + 1)
    bv.setColumns(V)
    if normalize:
        ng, lg = bv.orthonormalizeColumn(j)
    else:
        Hg, ng, lg = bv.orthogonalizeColumn(j)
        np.testing.assert_allclose(Hg, Ho, rtol=1e-11, atol=1e-13 * np.abs(Ho).max())
    assert lg == lo
    np.testing.assert_allclose(ng, no, rtol=1e-12)
    np.testing.assert_allclose(bv.getColumn(j), Vo[:, j], rtol=0, atol=1e-12 * np.abs(Vo[:, j]).max())
    if j:  # the basis is only read
        np.testing.assert_array_equal(bv.getColumn(j - 1), V[:, j - 1])
