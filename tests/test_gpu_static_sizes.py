"""pd_osb_force_static (csrc/pd_static.cu) with every number of lanes per point, at both ends of each
range, with lists shorter than the lanes of a point and lists of several rounds, ragged last blocks,
and bond states that differ between the two directions of a pair. Reference: the FP64 serial-order
entry points; bar: the summation order and a few roundings per bond, 1e-12 of the largest force."""
import ctypes as C

import numpy as np
import pytest

import pdcuda as pd
from helpers import deform
from test_zz_no_alloc import KERNELS, csr_bonds, regular_force

pytestmark = pytest.mark.gpu


# 32 lanes a point up to 8,192 points, 16 up to 40,960, 8 beyond
@pytest.mark.parametrize("shape,m", [((3, 1, 1), 1.01), ((7, 5, 3), 4.015), ((16, 16, 32), 2.015),
                                     ((23, 21, 17), 3.015), ((32, 32, 40), 1.8), ((43, 41, 37), 2.015)])
@pytest.mark.parametrize("kernel", ["linear", "cubic_b_spline"])
def test_lanes_per_point(shape, m, kernel):
    import torch
    dx = 0.01
    pos, vol = pd.uniform_box(*(k * dx for k in shape), dx)
    r = np.random.default_rng(5)
    pos = pos + r.uniform(-0.02 * dx, 0.02 * dx, pos.shape)   # lists whose reverse is not the mirrored place
    body = pd.Body(pd.OSBMaterial(), pos, vol)
    pd.material(body, horizon=m * dx, rho=7850.0, E=210e9, nu=0.25, Gc=1e6)
    off, nbr, L, fpb = csr_bonds(body, body.point_params[0].delta)
    x = body._pos + deform(body._pos, amplitude=1e-6)
    ba0 = (r.random(len(nbr)) > 0.1).astype(np.uint8)
    ref = regular_force(body, off, nbr, L, fpb, x, KERNELS[kernel], ba0)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    n = body.n_points
    a = [t(v) for v in (body._pos, x, body.volume, off, nbr, L, fpb, ba0)]
    b = torch.full((n, 3), float("nan"), dtype=torch.float64, device="cuda")
    na = torch.full((n,), -1, dtype=torch.int64, device="cuda")
    p = body.point_params[0].to_c()
    st = pd.lib().pd_osb_force_static(n, *(v.data_ptr() for v in a), C.byref(p), KERNELS[kernel],
                                      b.data_ptr(), na.data_ptr(),
                                      C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0, pd.lib().pd_static_last_error()
    assert np.abs(b.cpu().numpy() - ref[0]).max() <= 1e-12 * np.abs(ref[0]).max()
    assert np.array_equal(na.cpu().numpy(), ref[1])
    assert np.array_equal(a[7].cpu().numpy(), ref[2])
