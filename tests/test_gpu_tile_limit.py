"""Bodies whose tiles do not fit (more than 4095 points; correspondence phase B: 72 bytes a point in a
block's shared memory): the kernels without tiles against the oracle, and a body on one side of the limit
with its partitions on the other, bit for bit. Bars of the forces: those of the tile kernels (FP32 2e-5,
FP64 1e-12 of the largest force density)."""
import numpy as np
import pytest

import pdcuda as pd
from pdcuda.halo import Partition, PartitionedBody
from helpers import deform, oracle_body
from test_gpu_tiles import MATERIALS, box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,pipe", [("fp32", 0), ("fp32", 4), ("fp32", 5), ("fp64", 0)])
@pytest.mark.parametrize("name", list(MATERIALS))
def test_force_without_tiles(name, prec, pipe):
    if name == "C" and pipe == 4:
        pytest.skip("variant 4 is for BB and OSB")
    body = box(MATERIALS[name](), 20, 20, 20, 6.5, jitter=0.02)
    ob = oracle_body(body)
    u = deform(body._pos)
    ob.pos[:] = body._pos + u
    ob.force_density()
    dev = pd.DeviceBody(body, precision=prec)
    dev.set_pipeline(pipe)
    assert dev.tile_info()[0] == 0 and dev.tile_info()[2] == 0
    dev.set_state(position=body._pos + u)
    tol = 2e-5 if prec == "fp32" else 1e-12
    for _ in range(2):   # the full sums of the first evaluation, then the stored ones
        dev.force()
        assert np.abs(dev.field("b_int").T - ob.b_int).max() < tol * np.abs(ob.b_int).max()
    assert np.array_equal(dev.field("n_active_bonds"), ob.n_active)
    dev.close()


# whole: no tiles (BB, OSB) or none in phase B (C); the halves of the body have them in all phases
@pytest.mark.parametrize("prec,pipe", [("fp32", 0), ("fp32", 4), ("fp32", 5), ("fp64", 0)])
@pytest.mark.parametrize("name,shape,m,whole", [("BB", (20, 20, 20), 6.5, 0), ("OSB", (20, 20, 20), 6.5, 0),
                                                ("OSB-cubic", (22, 20, 18), 6.2, 0), ("C", (23, 19, 21), 5.1, 1)])
def test_body_and_partitions_on_both_sides_of_the_limit(name, shape, m, whole, prec, pipe):
    if name == "C" and (pipe == 4 or prec == "fp64"):
        pytest.skip("variant 4 is for BB and OSB, FP64 correspondence has no tiles")
    body = box(MATERIALS[name](), *shape, m, fracture=True)
    phases = 1 if name == "BB" or prec == "fp64" else 3   # FP64 OSB phase B: split slices gather from memory
    dev = pd.DeviceBody(body, precision=prec)
    dev.set_pipeline(pipe)
    assert dev.tile_info()[2] == whole
    r = np.random.default_rng(8)
    u = 1e-6 * r.standard_normal(body._pos.shape)    # stretches on both sides of the critical one
    state = {"displacement": u} if prec == "fp32" else {"position": body._pos + u, "displacement": u}
    state["velocity"] = 30.0 * u
    dt = 0.5 * dev.stable_timestep()
    dev.set_state(**state)
    dev.force(0.0, dt)
    dev.run(1, 12, dt)
    parts = [Partition(body, 2, k, prec) for k in range(2)]
    for p in parts:
        p.dev.set_pipeline(pipe)
        assert p.dev.tile_info()[2] == phases
        p.dev.set_state(**{k: x[p.rows] for k, x in state.items()})
    pb = PartitionedBody(parts)
    pb.force(0.0, dt)
    pb.run(1, 12, dt)
    for f in ("displacement", "velocity", "acceleration", "damage", "bond_active"):
        assert np.array_equal(pb.field(f), dev.field(f)), f
    assert 0.3 < dev.field("bond_active").mean() < 1.0
    assert np.isfinite(dev.field("acceleration")).all() and np.abs(dev.field("b_int")).max() > 0
    pb.close()
    dev.close()
