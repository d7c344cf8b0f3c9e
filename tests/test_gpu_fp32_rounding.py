"""Where the FP32 kernels round: the sum of a point's bonds meets the factor that all of them share in
double and is rounded once, and no parameter's rounding moves all forces of a body the same way.
On jittered bodies the roundings of a bond are independent of those of the others. Reference: the FP64
kernels."""
import numpy as np
import pytest

import pdcuda as pd

pytestmark = pytest.mark.gpu

DX = 1e-3
MATERIALS = {"BB": pd.BBMaterial, "OSB": pd.OSBMaterial}


def waves(x):
    k = np.random.default_rng(9).uniform(0, 2 * np.pi, (3, 3))
    s = 2 * np.pi * x / (20 * DX)
    return 1e-6 * np.stack([sum(np.sin(s[:, a] + k[a, c]) for a in range(3)) for c in range(3)], 1)


def forces(name, m, u, pipe, seed, jitter=0.05):
    pos, vol = pd.uniform_box(30 * DX, 24 * DX, 20 * DX, DX)
    pos = pos + np.random.default_rng(seed).uniform(-jitter * DX, jitter * DX, pos.shape)
    body = pd.Body(MATERIALS[name](), pos, vol)
    kw = dict(horizon=m * DX, rho=2700.0, E=70e9, Gc=1e6)
    if name != "BB":
        kw["nu"] = 0.25
    pd.material(body, **kw)
    out = []
    for prec in ("fp64", "fp32"):
        dev = pd.DeviceBody(body, precision=prec)
        if prec == "fp32":
            dev.set_pipeline(pipe)
        dev.set_state(position=body._pos + u(body._pos))
        dev.force()
        out.append(dev.field("b_int").T.copy())
        dev.close()
    return out


# A bond-based force is the bond constant times a sum that does not depend on it. The mean of force / constant
# over 64 constants is that sum to 0.3 ulp / 8; a sum that was rounded to FP32 by itself would lie within
# that of an FP32 number, an unrounded one lies a quarter of an ulp off on average.
@pytest.mark.parametrize("pipe", [0, 5])
def test_sums_are_rounded_once(pipe):
    pos, vol = pd.uniform_box(9 * DX, 8 * DX, 7 * DX, DX)
    pos = pos + np.random.default_rng(1).uniform(-0.05 * DX, 0.05 * DX, pos.shape)
    sums = []
    for k in range(64):
        body = pd.Body(pd.BBMaterial(), pos, vol)
        pd.material(body, horizon=3.015 * DX, rho=2700.0, E=70e9 * (1.0 + 0.9 * k / 64), Gc=1e6)
        dev = pd.DeviceBody(body, precision="fp32")
        dev.set_pipeline(pipe)
        dev.set_state(displacement=1e-3 * body._pos)
        dev.force()
        sums.append(dev.field("b_int") / body.point_params[0].bc)
        dev.close()
    s = np.mean(sums, 0)
    x = s / np.spacing(np.abs(s).astype(np.float32)).astype(np.float64)
    assert np.abs(x - np.round(x)).mean() > 0.15


# (float)delta is 3.9e-8 off at this horizon. Without a common factor what is left is the mean of 72,000
# independent errors of about 1e-7 and of the approximate reciprocals, below a quarter of an ulp: 1.5e-8.
@pytest.mark.parametrize("pipe", [0, 5])
def test_horizon_moves_no_forces(pipe):
    m = 3.0076775
    assert abs(float(np.float32(m * DX)) / (m * DX) - 1.0) > 3.8e-8
    g, h = forces("OSB", m, waves, pipe, 2)
    assert abs(np.vdot(g, h) / np.vdot(g, g) - 1.0) < 1.5e-8


# On a lattice the roundings of a bond repeat in every point. Those of the reference vectors' components are
# all alike (4.7e-8 here) and leave the forces 6.6e-8 to 7.1e-8 off where the weighted volume is summed from
# them. Without them there are those of the volume times the lengths and their reciprocals: three or so of
# 1.7e-8 rms each.
@pytest.mark.parametrize("pipe", [0, 5])
@pytest.mark.parametrize("m", [2.015, 4.015])
def test_lattice_spacing_moves_no_forces(m, pipe):
    g, h = forces("OSB", m, waves, pipe, 2, jitter=0.0)
    assert abs(np.vdot(g, h) / np.vdot(g, g) - 1.0) < 4.5e-8
