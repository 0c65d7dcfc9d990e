"""Weight gradients of the scalar-channel layers (k_wgrad_edge): runs of 32
pixels of a row, so widths around multiples of 32, one-pixel images and more
runs than warps."""
import numpy as np
import pytest
import torch

import oracle.cnn_oracle as CO
from jfem_b200.cnn import LearnedSmoother, he_init, unpack

pytestmark = pytest.mark.gpu


# every product carries at most one BF16 rounding flip of a stored activation
# or gradient (2^-8 relative, 2^-9 on average) against the rounding oracle
TOL = 2.0 ** -8


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 3, 1), (2, 5, 31), (1, 4, 32), (3, 9, 33), (1, 2, 65), (2, 300, 40)])
def test_edge_layer_weight_gradients(ctx, shape):
    rng = np.random.default_rng(31)
    w = he_init(seed=4, gain_last=1.0)
    x = rng.standard_normal(shape).astype(np.float32)
    t = rng.standard_normal(shape).astype(np.float32)
    net = LearnedSmoother(ctx, w)
    loss, g = net.loss_and_grad(torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda())
    L, gr = CO.loss_and_grads_bf16(unpack(w), x.astype(np.float64), t.astype(np.float64))
    assert abs(loss - L) / L < 1e-3
    gg = unpack(g)
    for l in (0, 5):
        err = np.linalg.norm(gg[l] - gr[l]) / np.linalg.norm(gr[l])
        assert err < TOL, (l, err)
