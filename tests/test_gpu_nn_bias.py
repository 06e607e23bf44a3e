"""The bias gradients made beside the weight gradients, of every layer: each
layer's input channel 0 is held at one, so the gradient of the centre tap's
weight at that channel is the same sum, through the input's path."""

import numpy as np
import pytest

from oracle import nn
from phiray_b200.denoiser import LAYERS, Unet
from tests.test_gpu_nn import _net_inputs, _random_params, _sync, _t

pytestmark = pytest.mark.gpu


# levels of whole tiles; ragged ones down to 3 x 5 and 1 x 1; several tiles a block
@pytest.mark.parametrize("B,H,W", [(1, 16, 16), (2, 48, 80), (3, 32, 128), (7, 112, 96)])
def test_bias_gradients_equal_the_centre_tap_of_ones(gpu, B, H, W):
    import torch

    rng = np.random.default_rng(B * H + W)
    feat, irr, alb, ref = _net_inputs(rng, B, H, W)
    feat[..., 0] = 1.0
    blob = _random_params(rng)
    at = 0
    for ci, co in LAYERS:
        # output channel 0 is relu(0 x + 1); the head's is a logit
        blob[at: at + 9 * ci] = 0.0
        blob[at + 9 * ci * co] = 1.0
        at += 9 * ci * co + co
    net = Unet(gpu, params=blob)
    F, I, A, R = _t(feat, "bf16"), *(_t(a.astype(np.float32)) for a in (irr, alb, ref))
    loss = torch.zeros(1, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    net.compute_grads(F, I, A, R, B, H, W, H, W, loss)
    _sync(gpu)
    for k, ((ci, co), (gw, gb)) in enumerate(zip(LAYERS, nn.split_params(net.grads()))):
        ones = gw.reshape(co, 9, ci)[:, 4, 0]
        # the same products in the same order but for the atomics over at most
        # 148 blocks: 148 x 2^-24 of the partial sums. A tile left out of either
        # is a hundredth of the sum or more.
        assert np.linalg.norm(ones - gb) <= 1e-4 * np.linalg.norm(gb), k
        assert np.abs(ones - gb).max() <= 1e-3 * np.abs(gb).max(), k
        assert np.count_nonzero(gb) >= co // 4, k
    net.close()
