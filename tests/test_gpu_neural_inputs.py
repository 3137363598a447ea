"""A training step's inputs belong to the caller again when the call returns.

The step returns once the loss is known, with the backward pass still running on the operator's stream.  The
inputs are overwritten then from another stream: the parameters after some steps are those of an undisturbed run,
bit for bit (the kernels' sums have a fixed order).  One network for the one-pass kernels and one for the
separate products.
"""
import numpy as np
import pytest

from slepc_b200 import learned as LN

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,B", [((256, 32, 16, 4, 64, 8), 4), ((96, 65, 8, 3, 32, 4), 4)])
def test_inputs_are_free_after_a_step(b200, dims, B):
    import torch

    N, K = dims[0], dims[5]
    rng = np.random.default_rng(3)
    F0 = torch.from_numpy(rng.standard_normal((B, 3, N * N)).astype(np.float32)).cuda()
    T = rng.standard_normal((B, K, N * N))
    T0 = torch.from_numpy((T / np.linalg.norm(T, axis=2, keepdims=True)).astype(np.float32)).cuda()
    theta = LN.init_params(*dims, seed=2)
    own, other = torch.cuda.Stream(), torch.cuda.Stream()
    F, T = torch.empty_like(F0), torch.empty_like(T0)

    def run(disturb):
        op = b200.NeuralOperator().create(*dims, stream=own.cuda_stream)
        op.setParams(theta)
        losses = []
        for _ in range(4):
            other.synchronize()  # the overwrite of the step before is done, on its own stream
            F.copy_(F0)
            T.copy_(T0)
            torch.cuda.synchronize()
            losses.append(op.trainStep(F, T, 1e-3))
            if disturb:
                with torch.cuda.stream(other):
                    T.fill_(float("nan"))
                    F.fill_(float("nan"))
        out = op.getParams()
        torch.cuda.synchronize()
        op.destroy()
        return losses, out

    l0, p0 = run(False)
    l1, p1 = run(True)
    assert np.isfinite(p0).all() and l1 == l0
    np.testing.assert_array_equal(p1, p0)
