"""A change of the bond layout for which there is no memory: the body keeps its layout, what was allocated for
the other is given back, and the calls after it do not find the failure."""
import numpy as np
import pytest

import pdcuda as pd

pytestmark = pytest.mark.gpu


def test_layout_without_memory():
    import torch
    dx = 1e-3
    pos, vol = pd.uniform_box(100 * dx, 100 * dx, 60 * dx, dx)
    body = pd.Body(pd.OSBMaterial(), pos, vol)
    pd.material(body, horizon=3.015 * dx, rho=2700.0, E=70e9, nu=0.25, Gc=1e6)
    dev = pd.DeviceBody(body, precision="fp32")        # 70M bonds: 1.7 GB a layout
    dev.set_state(displacement=1e-7 * np.sin(40.0 * body._pos))
    dev.force()
    forces, tiles = dev.field("b_int").copy(), dev.tile_info()
    torch.zeros(1, device="cuda")
    free = torch.cuda.mem_get_info()[0]
    fill = torch.empty(free - (600 << 20), dtype=torch.uint8, device="cuda")
    before = torch.cuda.mem_get_info()[0]
    for _ in range(3):
        with pytest.raises(Exception):
            dev.set_mapping(4)
        assert torch.cuda.mem_get_info()[0] > before - (32 << 20)
    dev.set_pipeline(2)                                 # its own order would be better, this one does
    dev.force()
    assert np.abs(dev.field("b_int") - forces).max() < 2e-5 * np.abs(forces).max()
    dev.set_pipeline(5)
    dev.set_graph(2)
    dev.force()
    assert dev.tile_info() == tiles and np.array_equal(dev.field("b_int"), forces)
    dev.run(1, 4, 0.1 * dev.stable_timestep())
    del fill
    torch.cuda.empty_cache()
    dev.set_mapping(4)
    assert dev.tile_info() == (0, 0, 0)
    dev.close()
