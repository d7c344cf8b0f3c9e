"""The FP32 tile kernels (csrc/pd_tile32.cu, csrc/pd_tiles.cu): sides that are no multiple of a tile's,
slices of one and of several segments, every number of warps per slice, a horizon whose tiles do not
fit (the kernels without tiles then run), and points in any order. Bar: the FP32 form's 2e-5 of the
largest force density (tests/test_gpu_parity.py)."""
import numpy as np
import pytest

import pdcuda as pd
from helpers import deform, oracle_body

pytestmark = pytest.mark.gpu

MATERIALS = {"BB": pd.BBMaterial, "OSB": pd.OSBMaterial,
             "OSB-cubic": lambda: pd.OSBMaterial(kernel=pd.cubic_b_spline_kernel),
             "C": lambda: pd.CMaterial(model=pd.NeoHooke())}


def box(mat, nx, ny, nz, m, jitter=0.0, shuffle=False, fracture=False):
    dx = 1.0 / nz
    pos, vol = pd.uniform_box(nx * dx, ny * dx, nz * dx, dx)
    r = np.random.default_rng(3)
    pos = pos + r.uniform(-jitter * dx, jitter * dx, pos.shape)
    if shuffle:
        pos = pos[:, r.permutation(pos.shape[1])]
    body = pd.Body(mat, pos, vol)
    kw = dict(horizon=m * dx, rho=7850.0, E=210e9, Gc=2.7)
    if not isinstance(mat, pd.BBMaterial):
        kw["nu"] = 0.25
    pd.material(body, **kw)
    if not fracture:
        pd.no_failure(body)
    return body


# 8, 4, 2 and 1 warps a slice (14,208, 28,416 and 56,832 points are the ends of the first three), one
# partly filled tile, 12 and 250 bonds a point, 5.6 dx: more than 4095 points a tile
@pytest.mark.parametrize("name", list(MATERIALS))
@pytest.mark.parametrize("shape,m", [((3, 3, 3), 1.8), ((17, 9, 6), 3.015), ((13, 11, 10), 4.015),
                                     ((15, 14, 13), 5.6), ((37, 31, 14), 2.015), ((41, 37, 23), 1.8),
                                     ((53, 41, 27), 1.8)])
def test_force_against_oracle(name, shape, m):
    for jitter, shuffle in ((0.0, False), (0.05, True)):
        body = box(MATERIALS[name](), *shape, m, jitter, shuffle)
        ob = oracle_body(body)
        u = deform(body._pos)
        ob.pos[:] = body._pos + u
        ob.force_density()
        dev = pd.DeviceBody(body, precision="fp32")
        dev.set_state(displacement=u)
        for _ in range(2):   # the full sums of the first evaluation, then the stored ones
            dev.force()
            assert np.abs(dev.field("b_int").T - ob.b_int).max() < 2e-5 * np.abs(ob.b_int).max()
        assert np.array_equal(dev.field("n_active_bonds"), ob.n_active)
        dev.close()


@pytest.mark.parametrize("name", ["BB", "OSB", "C"])
def test_result_does_not_depend_on_the_body_around(name):
    """A body alone (eight warps a slice) and among copies of itself (one warp): the same bits, with
    bonds breaking."""
    body = box(MATERIALS[name](), 15, 16, 15, 2.015, fracture=True)
    one = pd.Ensemble([body], precision="fp32")
    many = pd.Ensemble([body] * 33, precision="fp32")
    d = deform(body._pos, amplitude=0.002)   # stretches on both sides of the critical one
    for ens, k in ((one, 1), (many, 33)):
        ens.dev.set_state(displacement=np.tile(d, (k, 1)), velocity=np.tile(d, (k, 1)))
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


def test_tile_that_leaves_no_room_for_the_segment_sums():
    """3,152 points a tile: the 72 bytes a point of CMat phase B fit a block's shared memory, but not
    together with the sums of the warps that share a slice."""
    body = box(MATERIALS["C"](), 23, 19, 21, 5.1, jitter=0.05)
    ob = oracle_body(body)
    u = deform(body._pos)
    ob.pos[:] = body._pos + u
    ob.force_density()
    dev = pd.DeviceBody(body, precision="fp32")
    dev.set_state(displacement=u)
    dev.force()
    assert np.abs(dev.field("b_int").T - ob.b_int).max() < 2e-5 * np.abs(ob.b_int).max()
    dev.close()
