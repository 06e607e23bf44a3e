"""Values that are not finite in a convolution's input reach the weight
gradients that they enter, and no others."""

import numpy as np
import pytest

from oracle import nn
from phiray_b200 import _native as N
from tests.test_gpu_nn import _np, _round64, _sync, _t

pytestmark = pytest.mark.gpu


# widths and heights that end inside a tile, at its edge, one pixel into the
# next; odd heights; all nine taps a block (cin 16) and three (cin 48, 160)
@pytest.mark.parametrize("B,H,W", [(1, 1, 1), (2, 3, 5), (1, 16, 8), (1, 17, 9), (2, 18, 12), (1, 31, 23), (1, 6, 16),
                                   (3, 9, 8), (1, 33, 7)])
@pytest.mark.parametrize("cin,cout", [(16, 32), (48, 64), (160, 160)])
def test_weight_gradients_of_inputs_that_are_not_finite(gpu, B, H, W, cin, cout):
    import torch

    rng = np.random.default_rng(H * 100 + W + cin)
    x = nn.bf16(rng.normal(size=(B, H, W, cin)))
    dy = nn.bf16(rng.normal(size=(B, H, W, cout)))
    # one channel each: the last column, the last row, the corner, anywhere
    bad = np.zeros_like(x, bool)
    bad[:, rng.integers(H), W - 1, 0] = True
    bad[:, H - 1, rng.integers(W), 3] = True
    bad[B - 1, H - 1, W - 1, 9] = True
    bad[0, rng.integers(H), rng.integers(W), 14] = True
    x[bad] = rng.choice([np.inf, -np.inf, np.nan], int(bad.sum()))
    K, Kp = 9 * cin, _round64(9 * cin)
    X, DY = _t(x, "bf16"), _t(dy, "bf16")
    dWt = torch.zeros((Kp, cout), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    N.check(N.lib().phx_nn_conv_wgrad(gpu.handle, X.data_ptr(), cin, 0, cin, DY.data_ptr(), cout, 0, cout,
                                      dWt.data_ptr(), Kp, B, H, W))
    _sync(gpu)
    got = _np(dWt)[:K].T
    # which sums a bad value enters: those with a pixel of the image at its tap
    hit = nn.conv_wgrad(bad.astype(np.float64), np.ones_like(dy)) > 0
    assert np.array_equal(~np.isfinite(got), hit)
    fine = np.where(bad, 0.0, x)
    mag = nn.conv_wgrad(np.abs(fine), np.abs(dy))
    err = np.abs(np.where(hit, 0.0, got) - np.where(hit, 0.0, nn.conv_wgrad(fine, dy)))
    assert np.all(err <= 1e-5 * mag + 1e-30)  # as test_conv_wgrad_edges
