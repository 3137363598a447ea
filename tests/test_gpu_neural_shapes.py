"""The one-pass kernels of the neural operator at the edges of their shapes, against the CPU oracle.

They take grids from N = 32 (a block of 256 points touches up to nine image rows) with odd N (rows that are
not 16-byte aligned, points of two rows in a warp), ragged last blocks, N past one block of mode columns, up to
64 channels (two groups of 32 outputs), 16 modes, 128 hidden channels (one to four groups), 16 outputs.  Sizes
beyond them go through the separate products.  Tolerances are those of test_gpu_learned.py.
"""
import numpy as np
import pytest

from oracle import neural_operator as NO
from slepc_b200 import learned as LN

pytestmark = pytest.mark.gpu

SHAPES = [((32, 8, 5, 1, 7, 1), 1), ((33, 3, 16, 2, 40, 16), 3), ((64, 32, 16, 2, 64, 16), 2), ((130, 17, 4, 2, 33, 5), 1),
          ((48, 33, 7, 3, 128, 9), 2), ((37, 64, 16, 2, 100, 16), 1), ((256, 5, 12, 2, 16, 3), 1),
          ((40, 65, 4, 2, 16, 4), 1), ((36, 8, 17, 2, 16, 4), 1), ((36, 8, 4, 2, 130, 4), 1), ((36, 8, 4, 2, 16, 17), 1)]


@pytest.mark.parametrize("dims,B", SHAPES)
def test_shapes_vs_oracle(b200, dims, B):
    import torch

    N, W, M, L, H, K = dims
    rng = np.random.default_rng(list(dims))
    theta = LN.init_params(*dims, seed=1)
    theta = (theta + 0.02 * rng.standard_normal(theta.size)).astype(np.float32)
    F = rng.standard_normal((B, 3, N * N)).astype(np.float32)
    T = rng.standard_normal((B, K, N * N))
    T = (T / np.linalg.norm(T, axis=2, keepdims=True)).astype(np.float32)
    op = b200.NeuralOperator().create(*dims)
    op.setParams(theta)
    Fd, Td = torch.from_numpy(F).cuda(), torch.from_numpy(T).cuda()
    Yo, _ = NO.forward(theta.astype(np.float64), F.astype(np.float64), dims)
    lo, go = NO.loss_grad(theta.astype(np.float64), F.astype(np.float64), T.astype(np.float64), dims)
    Y = op.forward(Fd).cpu().numpy()
    assert np.linalg.norm(Y - Yo) <= 1e-4 * np.linalg.norm(Yo)
    l1, g1 = op.lossGrad(Fd, Td)
    assert abs(l1 - lo) <= 1e-4 * abs(lo) and abs(op.loss(Fd, Td) - lo) <= 1e-4 * abs(lo)
    off = 0
    for name, shape in NO.sizes(*dims):
        n = int(np.prod(shape))
        a, b = g1[off:off + n], go[off:off + n]
        assert np.linalg.norm(a - b) <= 2e-3 * np.linalg.norm(b), name
        off += n
    l2, g2 = op.lossGrad(Fd, Td)
    assert l2 == l1
    np.testing.assert_array_equal(g2, g1)
