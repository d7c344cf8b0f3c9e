"""The sums of the displacement gradient of FP32 correspondence: compensated unless bond-stream variant 5
asks for plain ones. 514 bonds a point: the additions of a plain sum, each within 2.5e-8 rms of a partial
sum that grows to the whole, leave 2.5e-8 sqrt(514 / 3) = 3.3e-7; the inverse of the shape tensor and the
product with it leave about 20 roundings, 1.1e-7. Bar for the compensated sums: 2e-7."""
import numpy as np
import pytest

import pdcuda as pd
from test_gpu_tiles import box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jitter", [0.0, 0.05])
@pytest.mark.parametrize("m", [5.015, 5.6])   # tiles of 1,906 and 2,081 points: both phases fit
def test_gradient_of_a_uniform_deformation(jitter, m):
    body = box(pd.CMaterial(), 17, 16, 15, m, jitter)
    G = np.array([[3.1e-3, 1.3e-3, -0.7e-3], [0.9e-3, -2.3e-3, 1.9e-3], [1.1e-3, 0.3e-3, 2.7e-3]])
    dev = pd.DeviceBody(body, precision="fp32")
    dev.set_state(displacement=body._pos @ G.T)
    for _ in range(2):   # the shape tensor in full, then the stored one
        dev.force()
        F = dev.field("defgrad").T.reshape(-1, 3, 3).transpose(0, 2, 1)   # column-major
        nn = dev.field("n_neighbors")
        H = (F - np.eye(3))[nn > 0.95 * nn.max()]
        assert len(H) > 50
        assert np.sqrt(np.mean((H - G) ** 2)) < 2e-7 * np.sqrt(np.mean(G ** 2))
    dev.close()
