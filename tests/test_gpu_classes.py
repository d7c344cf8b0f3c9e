"""Bond classes (csrc/pd_classes.cu): a lattice body's bonds as one byte each give the packed FP32
kernels the same bits as the full bond stream. The full stream is reached by adding a few loose
points far from the lattice, whose bonds are all different (more than 256 records)."""
import numpy as np
import pytest

import pdcuda as pd

pytestmark = pytest.mark.gpu

MATERIALS = {"BB": pd.BBMaterial, "OSB": pd.OSBMaterial,
             "OSB-cubic": lambda: pd.OSBMaterial(kernel=pd.cubic_b_spline_kernel),
             "C": lambda: pd.CMaterial(model=pd.NeoHooke()),
             "C-const": lambda: pd.CMaterial(kernel=pd.const_one_kernel)}


def lattice(mat, nx, ny, nz, m, permit, loose):
    dx = 1e-3
    pos, vol = pd.uniform_box(nx * dx, ny * dx, nz * dx, dx)
    n = pos.shape[1]
    if loose:
        far = np.random.default_rng(5).uniform(0.0, 3 * dx, (3, 60)) + 1.0
        pos, vol = np.concatenate([pos, far], 1), np.concatenate([vol, np.full(60, dx ** 3)])
    body = pd.Body(mat, pos, vol)
    kw = dict(horizon=m * dx, rho=2700.0, E=70e9, Gc=50.0)
    if not isinstance(mat, pd.BBMaterial):
        kw["nu"] = 0.25
    pd.material(body, **kw)
    if permit == "half":   # bonds that may not fail carry their length negative: other records
        pd.point_set(body, "kept", np.arange(n) < n // 2)
        pd.failure_permit(body, "kept", False)
    return body, n


# one to several words a lane and every remainder of a word, partly filled slices, 250 records of
# a horizon of 4.015 and both permissions at 3.015 (244), and 514 records, which have no classes
@pytest.mark.parametrize("name", list(MATERIALS))
@pytest.mark.parametrize("shape,m,permit", [((9, 7, 5), 1.8, "all"), ((11, 8, 6), 2.015, "all"),
                                            ((13, 12, 11), 3.015, "half"),
                                            ((37, 9, 10), 4.015, "all"), ((12, 11, 13), 5.015, "all")])
def test_classes_give_the_bits_of_the_full_stream(name, shape, m, permit):
    res = []
    for loose in (False, True):
        body, n = lattice(MATERIALS[name](), *shape, m, permit, loose)
        dev = pd.DeviceBody(body, precision="fp32")
        dev.set_mapping(1, 128)
        dev.set_pipeline(5)
        v = np.zeros((body.n_points, 3))
        v[:n] = 6.0 * np.sin(900.0 * body._pos[:n, [1, 2, 0]])
        dev.set_state(velocity=v)
        dt = 1e-8
        dev.force(0.0, dt)
        dev.run(1, 25, dt)
        nb = int(dev.field("n_neighbors")[:n].sum())
        res.append([dev.field(f)[..., :n] for f in ("b_int", "displacement", "velocity", "damage")]
                   + [dev.field("bond_active")[:nb]])
        dev.close()
    assert np.abs(res[0][0]).max() > 0 and (not name.startswith("BB") or (res[0][4] == 0).any())
    for a, b in zip(*res):
        assert np.array_equal(a, b)


def test_classes_follow_the_layout():
    """Lane groups drop the classes, going back finds them again: the same forces."""
    body, n = lattice(pd.OSBMaterial(), 12, 10, 9, 3.015, "all", False)
    u = 1e-6 * np.sin(900.0 * body._pos[:, [1, 2, 0]])
    dev = pd.DeviceBody(body, precision="fp32")
    res = []
    for again in range(2):
        dev.set_mapping(1, 128)
        dev.set_pipeline(5)
        dev.set_state(displacement=u)
        dev.force()
        res.append(dev.field("b_int").copy())
        dev.set_mapping(8)
        dev.force()
        assert np.abs(dev.field("b_int") - res[0]).max() < 2e-5 * np.abs(res[0]).max()
    assert np.array_equal(*res)
    dev.close()
