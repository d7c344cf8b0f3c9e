"""A point that has lost all its bonds may be anywhere, at infinity too: the FP32 forces on the others
are those of the body with that point left in place, bit for bit, and it has none itself."""
import numpy as np
import pytest

import pdcuda as pd
from helpers import deform
from test_gpu_tiles import MATERIALS, box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pipe", [0, 5])
@pytest.mark.parametrize("away", [np.inf, -np.inf, np.nan, 1e30])
@pytest.mark.parametrize("name", ["BB", "OSB", "C"])
@pytest.mark.parametrize("shape,m,jitter", [((9, 8, 7), 3.015, 0.0), ((9, 8, 7), 3.015, 0.05),
                                            ((53, 41, 27), 1.8, 0.0)])
def test_broken_bonds_carry_nothing(name, shape, m, jitter, away, pipe):
    body = box(MATERIALS[name](), *shape, m, jitter)
    dev = pd.DeviceBody(body, precision="fp32")
    dev.set_pipeline(pipe)
    nn = dev.field("n_neighbors")
    owner = np.repeat(np.arange(dev.n), nn)
    q = dev.n // 2
    # the bond lists: a bond is one of q's if q owns it or is its neighbour (sorted lists, symmetric)
    start = np.concatenate([[0], np.cumsum(nn)])
    pos = body._pos
    near = np.flatnonzero((np.linalg.norm(pos - pos[q], axis=1) <= body.point_params[0].delta)
                          & (np.arange(dev.n) != q))
    assert len(near) == nn[q]
    active = np.ones(dev.n_bonds, np.uint8)
    active[owner == q] = 0
    for j in near:
        mine = np.flatnonzero((np.linalg.norm(pos - pos[j], axis=1) <= body.point_params[0].delta)
                              & (np.arange(dev.n) != j))
        assert len(mine) == nn[j]
        active[start[j] + np.searchsorted(mine, q)] = 0
    dev.set_state(bond_active=active)
    assert dev.info()[2] == 1
    u = deform(pos)
    forces = []
    for there in (False, True):
        w = u.copy()
        if there:
            w[q] = away
        dev.set_state(displacement=w)
        for _ in range(2):
            dev.force()
        forces.append(dev.field("b_int").T.copy())
    assert np.isfinite(forces[0]).all()
    assert (forces[0][q] == 0).all() and (forces[1][q] == 0).all()
    others = np.arange(dev.n) != q
    assert np.array_equal(forces[0][others], forces[1][others])
    dev.close()


@pytest.mark.parametrize("name", ["BB", "OSB"])
def test_bond_between_two_points_at_infinity_is_reported(name):
    """Two points far off whose only unbroken bond is the one between them: its length is undefined."""
    body = box(MATERIALS[name](), 9, 8, 7, 1.8)
    dev = pd.DeviceBody(body, precision="fp32")
    nn = dev.field("n_neighbors")
    owner = np.repeat(np.arange(dev.n), nn)
    rank = np.arange(dev.n_bonds) - np.repeat(np.cumsum(nn) - nn, nn)
    pos = body._pos
    d2 = ((pos[:, None] - pos[None]) ** 2).sum(2)
    near = (d2 <= body.point_params[0].delta ** 2) & ~np.eye(dev.n, dtype=bool)
    assert np.array_equal(near.sum(1), nn)
    nbr = np.concatenate([np.flatnonzero(near[i]) for i in range(dev.n)])
    assert len(nbr) == dev.n_bonds and (rank >= 0).all()
    p = dev.n // 2
    q = nbr[owner == p][0]
    pair = np.isin(owner, (p, q)) & np.isin(nbr, (p, q))
    active = np.where(np.isin(owner, (p, q)) | np.isin(nbr, (p, q)), pair, True).astype(np.uint8)
    dev.set_state(bond_active=active)
    assert dev.info()[2] == 1 and pair.sum() == 2
    u = deform(pos)
    dev.set_state(displacement=u)
    dev.force()
    u[[p, q]] = np.inf
    dev.set_state(displacement=u)
    with pytest.raises(pd.NaNError):
        dev.force()
    dev.close()
