"""CUDA graphs of a group of bodies (pd_group_run_vv) after a change of what a captured step holds: the
group captures its steps again and they equal eager ones bit for bit."""
import numpy as np
import pytest

import pdcuda as pd
from test_gpu_ensemble import build

pytestmark = pytest.mark.gpu

FACTORIES = {"BB": pd.BBMaterial, "OSB": pd.OSBMaterial, "C": lambda: pd.CMaterial(model=pd.NeoHooke())}


def pair(name, prec):
    bodies = build(FACTORIES[name])
    return [pd.Ensemble(bodies, precision=prec, graph_steps=g, classes=2) for g in (8, 0)]


def finish(graph, eager):
    for ens in (graph, eager):
        ens.run(16, first_step=17)
    for k in range(3):
        for f in ("displacement", "velocity", "bond_active"):
            assert np.array_equal(graph.field(f, k), eager.field(f, k)), f
    graph.close()
    eager.close()


@pytest.mark.parametrize("name,prec", [("OSB", "fp32"), ("C", "fp32"), ("OSB", "fp64")])
def test_bond_states_set_between_two_runs(name, prec):
    """Stored weighted volumes and shape tensors are summed anew, and one direction of a bond switched
    off makes the bond states directed: other kernels than the captured ones."""
    graph, eager = pair(name, prec)
    for ens in (graph, eager):
        ens.run(16)
        for dev in ens.devs:
            a = dev.field("bond_active").copy()
            a[np.random.default_rng(5).choice(len(a), len(a) // 20, replace=False)] = 0
            dev.set_state(bond_active=a)
            assert dev.info()[2] == 0
    finish(graph, eager)


@pytest.mark.parametrize("name", ["C", "BB"])
def test_layout_changed_and_changed_back(name):
    """The bond arrays of a body without tiles (FP64 correspondence) and of one with tiles are
    reallocated under an equal mapping."""
    graph, eager = pair(name, "fp64")
    for ens in (graph, eager):
        ens.run(16)
    for dev in graph.devs:
        dev.set_mapping(8)
        dev.set_mapping(1)
    finish(graph, eager)
