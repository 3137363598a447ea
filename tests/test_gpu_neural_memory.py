"""Device memory of the neural operator: the one-pass kernels hold no more than the separate products would.

The bound is the sum of the buffers of the separate form, from the sizes of its tensors: a batch that fits there
must fit the one-pass form too, partial sums included.
"""
import numpy as np
import pytest

from slepc_b200 import learned as LN

pytestmark = pytest.mark.gpu


def _separate_bytes(dims, B):
    N, W, M, L, H, K = dims
    P, M2, NM = N * N, M * M, N * M
    acts = 3 * P + (L + 1) * W * P + L * W * P + L * W * M2 + 2 * W * NM + W * M2 + 2 * H * P + K * P
    back = K * P + H * P + 3 * W * P + 2 * W * M2
    split = max(4 * B * max(3 * W, W * W, H * W, K * H), 1 << 22)
    return 4 * (B * (acts + back) + split)


@pytest.mark.parametrize("dims,B", [((256, 32, 16, 4, 64, 8), 4), ((128, 64, 8, 2, 128, 16), 2), ((512, 8, 16, 2, 16, 3), 1)])
def test_one_pass_form_needs_no_more_memory(b200, dims, B):
    import torch

    def step(d, b):
        op = b200.NeuralOperator().create(*d)
        op.setParams(LN.init_params(*d, seed=0))
        F = torch.zeros((b, 3, d[0] ** 2), device="cuda")
        T = torch.ones((b, d[5], d[0] ** 2), device="cuda") / d[0]
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        loss = op.trainStep(F, T, 1e-3)
        op.getParams()
        torch.cuda.synchronize()
        used = before - torch.cuda.mem_get_info()[0]
        op.destroy()
        assert np.isfinite(loss)
        return used

    step((32,) + dims[1:], 1)  # the kernels are loaded
    assert step(dims, B) <= _separate_bytes(dims, B)
