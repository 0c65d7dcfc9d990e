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


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 3, 29), (1, 4, 30), (1, 5, 31), (3, 8, 60), (1, 9, 61), (1, 70, 91)])
def test_conv_tiles_of_four_rows_of_thirty(ctx, shape, monkeypatch):
    """k_conv_ws tiles (4 rows x 30 output pixels) at their edges: forward and
    gradients equal the single-role kernel's bit for bit (16 x 8 tiles, the
    same accumulators), and the forward the rounding oracle."""
    rng = np.random.default_rng(32)
    w = he_init(seed=12, gain_last=1.0)
    xh = rng.standard_normal(shape).astype(np.float32)
    x = torch.from_numpy(xh).cuda()
    t = torch.from_numpy(rng.standard_normal(shape).astype(np.float32)).cuda()
    net = LearnedSmoother(ctx, w)
    monkeypatch.setenv("JFEM_CNN_PROJ", "0")
    outs = []
    for ws in ("1", "0"):
        monkeypatch.setenv("JFEM_CNN_WS", ws)
        outs.append((net.forward(x).cpu().numpy(), net.loss_and_grad(x, t)[1]))
    assert np.array_equal(outs[0][0], outs[1][0]) and np.array_equal(outs[0][1], outs[1][1])
    yr, _ = CO.forward_bf16(unpack(w), xh.astype(np.float64))
    assert np.linalg.norm(outs[0][0] - yr) < TOL * np.linalg.norm(yr)


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 7, 15), (1, 8, 16), (1, 9, 17), (3, 17, 33), (2, 200, 130)])
def test_tensor_core_weight_gradients_at_tile_edges(ctx, shape, monkeypatch):
    """k_wgrad_tc tiles (8 rows x 16 pixels, G with a halo row each side) at
    their edges and with several tiles per CTA, against the mma.sync kernel on
    the same BF16 images: FP32 sums of the same products in another order."""
    rng = np.random.default_rng(33)
    w = he_init(seed=13, gain_last=1.0)
    x = torch.from_numpy(rng.standard_normal(shape).astype(np.float32)).cuda()
    t = torch.from_numpy(rng.standard_normal(shape).astype(np.float32)).cuda()
    net = LearnedSmoother(ctx, w)
    g = []
    for tc in ("1", "0"):
        monkeypatch.setenv("JFEM_CNN_WGRAD_TC", tc)
        g.append(unpack(net.loss_and_grad(x, t)[1]))
    for l in (1, 2, 3, 4):
        # n products per entry: random-walk growth of the FP32 rounding of their sums
        bound = 2.0 ** -23 * np.sqrt(np.prod(shape) + 16.0) * 4
        assert np.linalg.norm(g[0][l] - g[1][l]) <= bound * np.linalg.norm(g[1][l]) + 1e-30, l
