"""The FP64 tile kernels (csrc/pd_tile64.cu): every number of warps per slice, both kernels of OSB phase
B (from tiles with one warp a slice, else from global memory), a partly filled tile, slices of one and
of several segments, a horizon whose tiles do not fit, and points in any order. Bar: the summation
order and a few roundings per bond, 1e-12 of the largest force density."""
import numpy as np
import pytest

import pdcuda as pd
from helpers import deform, oracle_body
from test_gpu_tiles import box

pytestmark = pytest.mark.gpu

MATERIALS = {"BB": pd.BBMaterial, "OSB": pd.OSBMaterial,
             "OSB-cubic": lambda: pd.OSBMaterial(kernel=pd.cubic_b_spline_kernel)}


# 8, 4, 2 and 1 warps a slice (up to 14,208, 28,416 and 56,832 points, and beyond)
@pytest.mark.parametrize("name", list(MATERIALS))
@pytest.mark.parametrize("shape,m", [((3, 3, 3), 1.8), ((17, 9, 6), 3.015), ((15, 14, 13), 5.6),
                                     ((37, 32, 12), 1.8), ((25, 24, 24), 2.015), ((41, 37, 27), 1.8),
                                     ((53, 41, 27), 1.8)])
def test_force_against_oracle(name, shape, m):
    for jitter, shuffle in ((0.0, False), (0.05, True)):
        body = box(MATERIALS[name](), *shape, m, jitter, shuffle)
        ob = oracle_body(body)
        u = deform(body._pos)
        ob.pos[:] = body._pos + u
        ob.force_density()
        dev = pd.DeviceBody(body, precision="fp64")
        dev.set_state(position=body._pos + u)
        dev.force()
        assert np.abs(dev.field("b_int").T - ob.b_int).max() < 1e-12 * np.abs(ob.b_int).max()
        assert np.array_equal(dev.field("n_active_bonds"), ob.n_active)
        dev.close()


@pytest.mark.parametrize("name", ["BB", "OSB"])
def test_failure_and_the_body_around(name):
    """Bonds that break, in a body alone (eight warps a slice) and among copies of itself (one warp):
    the same bits."""
    body = box(MATERIALS[name](), 15, 16, 15, 2.015, fracture=True)
    one = pd.Ensemble([body], precision="fp64")
    many = pd.Ensemble([body] * 33, precision="fp64")
    d = deform(body._pos, amplitude=0.002)   # stretches on both sides of the critical one
    for ens, k in ((one, 1), (many, 33)):
        ens.dev.set_state(position=np.tile(body._pos + d, (k, 1)), velocity=np.tile(d, (k, 1)))
        ens.dev.force(0.0, 1e-9)
        ens.dev.run(1, 12, 1e-9)
    u, na = one.field("displacement", 0), one.field("n_active_bonds", 0)
    assert np.abs(u).max() > 0 and (na < one.field("n_neighbors", 0)).any()
    for k in (0, 16, 32):
        assert np.array_equal(many.field("displacement", k), u)
        assert np.array_equal(many.field("n_active_bonds", k), na)
        assert np.array_equal(many.field("bond_active", k), one.field("bond_active", 0))
    one.close()
    many.close()
