"""The weight-gradient kernel at the edges of its tiles, channel chunks and
blocks, and the whole-network Adam step, against FP64 and the same formulas
in numpy."""

import numpy as np
import pytest

from oracle import nn
from phiray_b200 import _native as N
from phiray_b200.denoiser import LAYERS, Unet
from tests.test_gpu_nn import _np, _round64, _sync, _t

pytestmark = pytest.mark.gpu


# one pixel; less than a tile; one row and column more than tiles; the
# smallest and largest channel counts, uneven chunks (144 = 80 + 64), the
# second block of output channels (160)
@pytest.mark.parametrize("cin,cout,shape", [(16, 32, (1, 1, 1)), (32, 32, (3, 17, 9)), (144, 96, (1, 15, 7)),
                                            (48, 160, (2, 16, 8)), (224, 96, (1, 33, 25)), (128, 128, (1, 4, 4)),
                                            (160, 160, (5, 8, 8)), (32, 64, (7, 48, 40))])
def test_conv_wgrad_edges(gpu, cin, cout, shape):
    import torch

    rng = np.random.default_rng(cin * 3 + cout)
    x = nn.bf16(rng.normal(size=(*shape, cin)))
    dy = nn.bf16(rng.normal(size=(*shape, cout)))
    K, Kp = 9 * cin, _round64(9 * cin)
    X, DY = _t(x, "bf16"), _t(dy, "bf16")
    dWt = torch.zeros((Kp, cout), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    N.check(N.lib().phx_nn_conv_wgrad(gpu.handle, X.data_ptr(), cin, 0, cin, DY.data_ptr(), cout, 0, cout,
                                      dWt.data_ptr(), Kp, *shape))
    _sync(gpu)
    got = _np(dWt)
    mag = nn.conv_wgrad(np.abs(x), np.abs(dy))
    # fp32 sums of exact products: as test_conv_wgrad
    assert np.all(np.abs(got[:K].T - nn.conv_wgrad(x, dy)) <= 1e-5 * mag + 1e-30)
    assert np.all(got[K:] == 0.0)


def test_network_adam_equals_the_formula_and_refreshes_both_copies(gpu):
    import torch

    g = torch.Generator(device="cuda").manual_seed(4)
    B, z = 2, 32
    feat = torch.randn(B, z, z, 16, generator=g, device="cuda").to(torch.bfloat16)
    irr, alb, ref = (torch.rand(B, z, z, 3, generator=g, device="cuda") + 0.1 for _ in range(3))
    loss = torch.zeros(1, device="cuda")
    torch.cuda.synchronize()
    net = Unet(gpu, seed=9)
    m = v = np.zeros(net.count, np.float64)
    lr, b1, b2, eps = 1e-3, 0.9, 0.999, 1e-8
    for step in (1, 2):
        net.compute_grads(feat, irr, alb, ref, B, z, z, z, z, loss)
        p0, gr = net.params().astype(np.float64), net.grads().astype(np.float64)
        net.adam(lr)
        m, v = b1 * m + (1 - b1) * gr, b2 * v + (1 - b2) * gr * gr
        want = p0 - lr * (m / (1 - b1 ** step)) / (np.sqrt(v / (1 - b2 ** step)) + eps)
        # a step is at most ~lr long and a few fp32 roundings off, the
        # weight itself half an ulp; (1 - b2) in fp32 is 1.3e-5 off
        assert np.all(np.abs(net.params() - want) <= 2e-5 * lr + 2.0 ** -23 * np.abs(want))
    # the bf16 copies of the next forward and backward are those of a network
    # given these weights
    other = Unet(gpu, params=net.params())
    net.compute_grads(feat, irr, alb, ref, B, z, z, z, z, loss)
    other.compute_grads(feat, irr, alb, ref, B, z, z, z, z, loss)
    a, b = net.grads(), other.grads()
    at = 0
    for ci, co in LAYERS:
        n = 9 * ci * co + co
        # the same sums up to the order of their atomics
        assert np.linalg.norm(a[at:at + n] - b[at:at + n]) <= 1e-5 * np.linalg.norm(b[at:at + n]) + 1e-12
        at += n
    net.close()
    other.close()
