"""Which bodies take the point order and the tiles of pd_tiles.cu: those whose kernels read tiles. A change
of the order keeps the state and the results, bit for bit where the kernels are the same again."""
import numpy as np
import pytest

import pdcuda as pd
from test_gpu_tiles import MATERIALS, box

pytestmark = pytest.mark.gpu


def esc_box(name, prec):
    mat = {"BB": pd.BBMaterial, "OSB": pd.OSBMaterial}[name](correction=pd.EnergySurfaceCorrection())
    return pd.DeviceBody(box(mat, 17, 9, 6, 3.015), precision=prec)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("name", ["BB", "OSB"])
def test_bodies_without_tile_kernels_hold_no_tiles(name, prec):
    dev = esc_box(name, prec)
    assert dev.tile_info() == (0, 0, 0)
    dev.close()
    body = box(MATERIALS[name](), 17, 9, 6, 3.015)
    pd.point_set(body, "right", body._pos[:, 0] > 0)
    kw = dict(horizon=3.015 / 6, rho=7850.0, E=100e9, Gc=2.7)
    pd.material(body, "right", **kw, **({} if name == "BB" else {"nu": 0.25}))
    dev = pd.DeviceBody(body, precision=prec)
    assert dev.tile_info() == (0, 0, 0)
    dev.close()


@pytest.mark.parametrize("pipe", [1, 2, 3])
@pytest.mark.parametrize("name", ["BB", "OSB"])
def test_staged_variants_and_back(name, pipe):
    """The staged stream walks the points in their own order; bonds broken before and after the change."""
    body = box(MATERIALS[name](), 17, 9, 6, 3.015, jitter=0.05, fracture=True)
    dev, ref = (pd.DeviceBody(body, precision="fp32") for _ in range(2))
    tiles = dev.tile_info()
    assert tiles[0] > 0
    r = np.random.default_rng(2)
    u = [5e-7 * r.standard_normal(body._pos.shape) for _ in range(3)]
    for k, w in enumerate(u):
        for d in (dev, ref):
            d.set_state(displacement=w)
            d.force()
        if k == 0:
            dev.set_pipeline(pipe)
            assert dev.tile_info() == (0, 0, 0)
            assert np.array_equal(dev.field("bond_active"), ref.field("bond_active"))
            dev.force()
            b, c = dev.field("b_int"), ref.field("b_int")
            assert np.abs(b - c).max() < 2e-5 * np.abs(c).max()
            assert np.array_equal(dev.field("bond_active"), ref.field("bond_active"))
            dev.set_pipeline(5)
            assert dev.tile_info() == tiles
            # weighted volumes of other kernels are not kept: dev sums its own anew, and so does ref
            ref.set_state(bond_active=ref.field("bond_active"))
    for f in ("b_int", "bond_active", "n_active_bonds", "displacement"):
        assert np.array_equal(dev.field(f), ref.field(f)), f
    assert 0.0 < dev.field("bond_active").mean() < 1.0
    dev.close()
    ref.close()


def test_autotune_ends_in_the_order_of_what_it_chose():
    body = box(MATERIALS["OSB"](), 17, 9, 6, 3.015)
    dev = pd.DeviceBody(body, precision="fp32")
    tiles = dev.tile_info()
    dev.autotune()
    group, _, pipe = dev.mapping()
    assert dev.tile_info() == (tiles if group == 1 and pipe in (0, 4, 5) else (0, 0, 0))
    dev.close()
