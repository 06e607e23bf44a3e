"""The fused denoise over the whole range of depths and radiances: quotients
that would under- or overflow on the way, zeros, weights from one to nothing, against the oracle."""

import numpy as np
import pytest

import phiray_b200 as px
from tests import pxgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(65, 41), (97, 33), (130, 66)])
@pytest.mark.parametrize("strength", [None, (0.0, 0.0, 0.0, 0.0), (1e-3, 1e-4, 1e3, 40.0)])
def test_denoise_over_the_range_of_floats(gpu, orc, w, h, strength):
    n = w * h
    img = pxgen.px_image(w, h, seed=n)
    f = img.view(np.float32)
    rng = np.random.default_rng(n)
    powers = np.array([0.0, 1e-38, 1e-30, 1e-19, 1e-18, 1e-9, 1.0, 1.0, 1.0, 1e4, 1e17, 1e18, 1e19], np.float32)
    # runs of pixels share a scale, so that neighbours of every ratio meet
    scale = lambda: rng.choice(powers, size=(n + 6) // 7).repeat(7)[:n]
    f[13 * n: 14 * n] *= scale()
    f[n: 4 * n] *= scale().repeat(3)
    kw = {} if strength is None else {"strength": strength}
    want = orc.denoise(img, w, h, **kw)
    d = px.GpuArray.from_(gpu, img)
    px.denoise(gpu, d, w, h, **kw)
    got = d.read(np.uint32)
    assert np.array_equal(got[: 7 * n], want[: 7 * n])
