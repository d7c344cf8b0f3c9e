"""FP64 force kernels off the serial order (csrc/pd_force64_fast.cu) against the oracle: slices with
fewer rows than a segment, with a ragged last segment and with several rounds of segments, every
number of warps per slice, and every lane group. Tolerance: the summation order and a few roundings
per bond, 1e-12 of the largest force density (the bar of the lane-group mappings)."""
import numpy as np
import pytest

import pdcuda as pd
from helpers import deform, oracle_body

pytestmark = pytest.mark.gpu

MATERIALS = {
    "BB": pd.BBMaterial,
    "OSB": pd.OSBMaterial,
    "OSB-cubic": lambda: pd.OSBMaterial(kernel=pd.cubic_b_spline_kernel),
    "C": pd.CMaterial,
    "C-NH-const": lambda: pd.CMaterial(model=pd.NeoHooke(), kernel=pd.const_one_kernel),
}


def box_body(mat, nx, ny, nz, m, fracture=False):
    dx = 1.0 / nz
    pos, vol = pd.uniform_box(nx * dx, ny * dx, nz * dx, dx)
    body = pd.Body(mat, pos, vol)
    kw = dict(horizon=m * dx, rho=7850.0, E=210e9, Gc=2.7)
    if not isinstance(mat, pd.BBMaterial):
        kw["nu"] = 0.25
    pd.material(body, **kw)
    if not fracture:
        pd.no_failure(body)
    return body


def force_of(body, x, prec="fp64", mapping=(1,)):
    dev = pd.DeviceBody(body, precision=prec)
    dev.set_mapping(*mapping)
    dev.set_state(position=x)
    dev.force()
    out = dev.field("b_int").T.copy(), dev.field("n_active_bonds"), dev.field("bond_active")
    dev.close()
    return out


# (nx, ny, nz, horizon / dx): 6 rows a slice, 16 and 17, 122 (a ragged eighth segment), 250 (a
# second round of eight warps); then the sizes at which 4, 2 and 1 warps walk a slice
SHAPES = [(7, 5, 5, 1.01), (9, 7, 1, 2.3), (6, 6, 6, 3.015), (9, 9, 9, 4.015), (64, 32, 31, 2.015),
          (71, 47, 41, 1.5), (91, 53, 51, 1.01)]


@pytest.mark.parametrize("name", list(MATERIALS))
@pytest.mark.parametrize("shape", SHAPES)
def test_force_against_oracle(name, shape):
    nx, ny, nz, m = shape
    if name.startswith("C") and (m < 1.5 or nz == 1):
        m, nz = 1.8, max(nz, 3)   # a shape tensor needs bonds in every direction
    body = box_body(MATERIALS[name](), nx, ny, nz, m)
    ob = oracle_body(body)
    x = body._pos + deform(body._pos)
    ob.pos[:] = x
    ob.force_density()
    b, na, _ = force_of(body, x)
    assert np.abs(b - ob.b_int).max() < 1e-12 * np.abs(ob.b_int).max()
    assert np.array_equal(na, ob.n_active)


@pytest.mark.parametrize("name", ["BB", "OSB", "C"])
@pytest.mark.parametrize("group", [1, 2, 8, 16, 32])
def test_failure_decisions_against_oracle(name, group):
    """Stretches on both sides of the critical one: the oracle's bond states, in every lane group."""
    body = box_body(MATERIALS[name](), 9, 8, 7, 3.015, fracture=True)
    ob = oracle_body(body)
    x = body._pos + deform(body._pos, amplitude=0.002)
    ob.pos[:] = x
    ob.force_density()
    b, na, states = force_of(body, x, mapping=(group,))
    assert 0 < np.count_nonzero(states == 0) < states.size
    assert np.array_equal(states, ob.bond_active[:ob.n_bonds]) and np.array_equal(na, ob.n_active)
    assert np.abs(b - ob.b_int).max() < 1e-12 * np.abs(ob.b_int).max()


@pytest.mark.parametrize("name", ["BB", "OSB", "C"])
def test_result_does_not_depend_on_the_body_around(name):
    """A body alone (eight warps a slice) and among copies of itself (one warp): the same bits."""
    body = box_body(MATERIALS[name](), 20, 24, 20, 2.015)
    dt = 1e-9
    one = pd.Ensemble([body], precision="fp64")
    many = pd.Ensemble([body] * 26, precision="fp64")
    v = 50.0 * deform(body._pos)
    for ens, k in ((one, 1), (many, 26)):
        ens.dev.set_state(velocity=np.tile(v, (k, 1)))
        ens.dev.run(1, 10, dt)
    u = one.field("displacement", 0)
    assert np.abs(u).max() > 0
    for k in (0, 13, 25):
        assert np.array_equal(many.field("displacement", k), u)
    one.close()
    many.close()
