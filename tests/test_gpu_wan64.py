"""FP64 correspondence with ZEMWan off the serial order (csrc/pd_force64_fast.cu, k_c_b64f) against the
oracle: every number of warps per slice, every lane group, slices of one and of several segments, and a
killed point beside intact ones. Bar: the summation order and a few roundings per bond, 1e-12 of the
largest force density (tests/test_gpu_force64_fast.py)."""
import numpy as np
import pytest

import pdcuda as pd
from helpers import deform, oracle_body
from test_gpu_force64_fast import box_body, force_of

pytestmark = pytest.mark.gpu

MODELS = {"linear": lambda: pd.CMaterial(zem=pd.ZEMWan()),
          "nh-cubic": lambda: pd.CMaterial(model=pd.NeoHooke(), zem=pd.ZEMWan(), kernel=pd.cubic_b_spline_kernel)}


@pytest.mark.parametrize("name", list(MODELS))
@pytest.mark.parametrize("shape,group", [((5, 4, 3, 1.8), 1), ((9, 9, 9, 4.015), 1), ((64, 32, 31, 2.015), 1),
                                         ((71, 47, 41, 1.8), 1), ((9, 8, 7, 3.015), 2), ((9, 8, 7, 3.015), 8),
                                         ((9, 8, 7, 3.015), 32)])
def test_force_against_oracle(name, shape, group):
    body = box_body(MODELS[name](), *shape)
    ob = oracle_body(body)
    x = body._pos + deform(body._pos)
    ob.pos[:] = x
    ob.force_density()
    b, na, _ = force_of(body, x, mapping=(group,))
    assert np.abs(b - ob.b_int).max() < 1e-12 * np.abs(ob.b_int).max()
    assert np.array_equal(na, ob.n_active)


def test_killed_points():
    """Stretches on both sides of the critical one: points that lose too many bonds are killed."""
    body = box_body(MODELS["linear"](), 9, 8, 7, 3.015, fracture=True)
    ob = oracle_body(body)
    x = body._pos + deform(body._pos, amplitude=0.002)
    ob.pos[:] = x
    ob.force_density()
    b, na, states = force_of(body, x)
    assert 0 < np.count_nonzero(states == 0) < states.size
    assert np.array_equal(states, ob.bond_active[:ob.n_bonds]) and np.array_equal(na, ob.n_active)
    assert np.abs(b - ob.b_int).max() < 1e-12 * np.abs(ob.b_int).max()
