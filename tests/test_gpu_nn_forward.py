"""The network's inference forward (pooling in the convolutions' epilogues,
upsampled channels read from the level below, kernel prediction in the head's
epilogue) against the training forward, which upsamples into memory and keeps
its logits, and those against the FP64 oracle: images smaller than a tile row,
one tile wide, and with ragged runs of tiles."""

import numpy as np
import pytest

from oracle import nn
from phiray_b200 import GpuArray
from phiray_b200 import _native as N
from phiray_b200.denoiser import Unet
from tests.test_gpu_nn import _net_inputs, _np, _random_params, _sync, _t

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W,h,w", [(1, 16, 16, 9, 16), (3, 48, 80, 48, 77), (1, 16, 208, 13, 201),
                                       (2, 112, 16, 100, 3)])
def test_inference_forward_equals_training_forward(gpu, B, H, W, h, w):
    import torch

    rng = np.random.default_rng(B * H + W)
    feat, irr, alb, ref = _net_inputs(rng, B, H, W)
    blob = _random_params(rng)
    net = Unet(gpu, params=blob)
    F, I, A, R = _t(feat, "bf16"), *(_t(a.astype(np.float32)) for a in (irr, alb, ref))
    loss = torch.zeros(1, dtype=torch.float32, device="cuda")
    o1, o2 = (torch.zeros(B, H, W, 3, device="cuda") for _ in range(2))
    e1, e2 = (torch.zeros(B, H, W, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    net.compute_grads(F, I, A, R, B, H, W, h, w, loss)
    N.check(N.lib().phx_nn_kpn(gpu.handle, net.logits(), I.data_ptr(), A.data_ptr(), None, B, H, W, h, w,
                               o1.data_ptr(), e1.data_ptr(), None, None, 0.0))
    _sync(gpu)
    logits = GpuArray(gpu, B * H * W * 32 * 4, _wrap=net.logits()).read(np.float32).reshape(B, H, W, 32)
    net.forward(F.data_ptr(), I.data_ptr(), A.data_ptr(), B, H, W, h, w, o2.data_ptr(), e2.data_ptr())
    _sync(gpu)
    # the same products in the same order and rounding: only the softmax's code
    # differs (the tolerances of the fused head's own test)
    assert np.allclose(_np(o1), _np(o2), rtol=1e-6, atol=1e-7)
    assert np.allclose(_np(e1), _np(e2), rtol=1e-6, atol=1e-9)
    want, _, _ = nn.forward(nn.split_params(blob), feat, rounded=True)
    assert np.abs(logits - want).max() <= 1e-2 * np.abs(want).max()
    net.close()
