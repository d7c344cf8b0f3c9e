"""Two bodies with tiles of different sizes, each stepped by a host thread of its own: handles are
independent (include/pdcuda.h), so neither's launches are refused for the other's shared memory."""
import threading

import numpy as np
import pytest

import pdcuda as pd
from test_gpu_tiles import box

pytestmark = pytest.mark.gpu

MATERIALS = {"BB": pd.BBMaterial, "OSB": pd.OSBMaterial, "C": lambda: pd.CMaterial(model=pd.NeoHooke())}


@pytest.mark.parametrize("graph", [0, 2])
@pytest.mark.parametrize("name,prec", [("BB", "fp32"), ("OSB", "fp32"), ("C", "fp32"), ("OSB", "fp64")])
def test_two_threads(name, prec, graph):
    # 1.8 spacings: a tile of 18 points; 5.1 spacings: more than the 48 KB that every kernel may use
    devs = [pd.DeviceBody(box(MATERIALS[name](), *shape, m, jitter=0.05), precision=prec)
            for shape, m in (((3, 3, 2), 1.8), ((13, 13, 13), 5.1))]
    errors, start = [], threading.Barrier(2)

    def step(dev):
        try:
            dt = 0.5 * dev.stable_timestep()
            dev.force(0.0, dt)
            start.wait()
            for k in range(400):
                if graph:
                    dev.set_graph(graph)   # captured again: as many launches per call
                dev.run(1 + 4 * k, 4, dt)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=step, args=(d,)) for d in devs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
    for d in devs:
        assert np.isfinite(d.field("displacement")).all()
        d.close()
