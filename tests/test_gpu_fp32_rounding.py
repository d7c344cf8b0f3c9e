"""Where the FP32 kernels round: the sum of a point's bonds meets the factor that all of them share in
double and is rounded once."""
import numpy as np
import pytest

import pdcuda as pd

pytestmark = pytest.mark.gpu

DX = 1e-3


# A bond-based force is the bond constant times a sum that does not depend on it. The mean of force / constant
# over 64 constants is that sum to 0.3 ulp / 8; a sum that was rounded to FP32 by itself would lie within
# that of an FP32 number, an unrounded one lies a quarter of an ulp off on average.
@pytest.mark.parametrize("pipe", [0, 5])
def test_sums_are_rounded_once(pipe):
    pos, vol = pd.uniform_box(9 * DX, 8 * DX, 7 * DX, DX)
    pos = pos + np.random.default_rng(1).uniform(-0.05 * DX, 0.05 * DX, pos.shape)
    sums = []
    for k in range(64):
        body = pd.Body(pd.BBMaterial(), pos, vol)
        pd.material(body, horizon=3.015 * DX, rho=2700.0, E=70e9 * (1.0 + 0.9 * k / 64), Gc=1e6)
        dev = pd.DeviceBody(body, precision="fp32")
        dev.set_pipeline(pipe)
        dev.set_state(displacement=1e-3 * body._pos)
        dev.force()
        sums.append(dev.field("b_int") / body.point_params[0].bc)
        dev.close()
    s = np.mean(sums, 0)
    x = s / np.spacing(np.abs(s).astype(np.float32)).astype(np.float64)
    assert np.abs(x - np.round(x)).mean() > 0.15
