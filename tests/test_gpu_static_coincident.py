"""pd_osb_force_static with two bonded points in one place: the force of their bond has no direction, so
both have none that is defined, but their dilatations are, and the points around them have the forces of
the FP64 serial-order entry points. Bar: 1e-12 of the largest force."""
import ctypes as C

import numpy as np
import pytest

import pdcuda as pd
from helpers import deform
from test_zz_no_alloc import KERNELS, csr_bonds, regular_force

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", ["linear", "cubic_b_spline"])
@pytest.mark.parametrize("cut", [False, True])
def test_two_points_in_one_place(kernel, cut):
    import torch
    dx = 0.01
    pos, vol = pd.uniform_box(9 * dx, 8 * dx, 7 * dx, dx)
    body = pd.Body(pd.OSBMaterial(), pos, vol)
    pd.material(body, horizon=3.015 * dx, rho=7850.0, E=210e9, nu=0.25, Gc=1e6)
    off, nbr, L, fpb = csr_bonds(body, body.point_params[0].delta)
    n = body.n_points
    x = body._pos + deform(body._pos, amplitude=1e-6)
    i = n // 2
    j = int(nbr[off[i]])
    x[j] = x[i]
    fpb[:] = 0                   # nothing breaks
    ba = np.ones(len(nbr), np.uint8)
    if cut:                      # the bond of the two is broken in both directions
        owner = np.repeat(np.arange(n), np.diff(off))
        ba[((owner == i) & (nbr == j)) | ((owner == j) & (nbr == i))] = 0
    others = ~np.isin(np.arange(n), (i, j))
    # the entry points report undefined forces, so the reference has the two an ulp apart
    near = x.copy()
    near[j, 0] = np.nextafter(x[i, 0], np.inf)
    ref = regular_force(body, off, nbr, L, fpb, near, KERNELS[kernel], ba.copy())
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    a = [t(v) for v in (body._pos, x, body.volume, off, nbr, L, fpb, ba)]
    b = torch.full((n, 3), 7.0, dtype=torch.float64, device="cuda")
    na = torch.full((n,), -1, dtype=torch.int64, device="cuda")
    p = body.point_params[0].to_c()
    st = pd.lib().pd_osb_force_static(n, *(v.data_ptr() for v in a), C.byref(p), KERNELS[kernel],
                                      b.data_ptr(), na.data_ptr(),
                                      C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0, pd.lib().pd_static_last_error()
    b = b.cpu().numpy()
    assert np.isnan(b[[i, j]]).all()
    assert np.abs(b[others] - ref[0][others]).max() <= 1e-12 * np.abs(ref[0][others]).max()
    assert np.array_equal(na.cpu().numpy(), ref[1])
