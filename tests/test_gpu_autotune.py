"""What pd_autotune times: every kernel once, not under each of its names."""
import numpy as np
import pytest

import pdcuda as pd
from helpers import deform, oracle_body
from test_gpu_tiles import MATERIALS, box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", list(MATERIALS))
def test_autotune_times_a_kernel_once(name):
    """One lane per point: the packed kernels on tiles (correspondence: both kinds of sums) and three staged
    variants (BB, OSB); 4 and 32 lanes: one- and (BB, OSB) two-row kernels with two block sizes. Six
    evaluations each, and two more rounds of the fastest three."""
    body = box(MATERIALS[name](), 17, 9, 6, 3.015)
    dev = pd.DeviceBody(body, precision="fp32")
    u = deform(body._pos)
    dev.set_state(displacement=u)
    before = dev.launch_count()
    dev.autotune()
    corr = name == "C"
    candidates = 2 + 2 * 2 if corr else 1 + 3 + 2 * 4
    per = 1 if name == "BB" else 2
    assert dev.launch_count() - before == 6 * per * (candidates + 2 * 3)
    ob = oracle_body(body)
    ob.pos[:] = body._pos + u
    ob.force_density()
    dev.force()
    assert np.abs(dev.field("b_int").T - ob.b_int).max() < 2e-5 * np.abs(ob.b_int).max()
    dev.close()


def test_tuning_leaves_nothing_of_other_kernels_behind():
    """The kernels timed on the way store weighted volumes with their own roundings; the chosen ones sum
    theirs anew."""
    body = box(MATERIALS["OSB"](), 40, 30, 20, 3.015, jitter=0.05)
    u = deform(body._pos)
    dev, ref = (pd.DeviceBody(body, precision="fp32") for _ in range(2))
    dev.set_state(displacement=u)
    dev.autotune()
    group, block, pipe = dev.mapping()
    ref.set_mapping(group, block)
    ref.set_pipeline(pipe)
    ref.set_state(displacement=u)
    for d in (dev, ref):
        d.force()
    assert np.array_equal(dev.field("b_int"), ref.field("b_int"))
    dev.close()
    ref.close()
