"""The elementary FP64 functions of the force kernels off the serial order (csrc/pd_bond64.cuh) against
64-bit significands and against CUDA's functions: random significands, powers of two and their neighbours,
perfect squares and lattice lengths, over the exponents that lengths, areas and their products take.

Bounds. With y the hardware's approximation to 2^-22 the third-order step leaves 2^-66; the residual of
1 / sqrt(x) carries the rounding of x y, half an ulp at most, halved by the step, and the last operation
rounds by half an ulp: below 1 ulp. The residual of 1 / x is exact to its own rounding: below 0.6 ulp. A
quotient's correction leaves the rounding of 1 / b times a residual below 2 ulp, far below an ulp, and
rounds by half one: below 0.6 ulp. The correction of a square root leaves less than 2^-100: as sqrt()."""
import ctypes as C

import numpy as np
import pytest

import pdcuda as pd

pytestmark = pytest.mark.gpu

RSQRT, RCP, SQRT, LENGTH, QUOTIENT, CUDA_RSQRT, CUDA_SQRT, CUDA_QUOTIENT = range(8)


def on_gpu(op, x, y=None):
    x = np.ascontiguousarray(x, np.float64)
    y = x if y is None else np.ascontiguousarray(y, np.float64)
    out = np.empty_like(x)
    assert pd.lib().pd_eval64(op, len(x), x.ctypes.data, y.ctypes.data, out.ctypes.data, 0) == 0
    return out


def arguments(n, lo, hi, seed):
    """Positive numbers between 2^lo and 2^hi."""
    r = np.random.default_rng(seed)
    e = r.integers(lo, hi, n)
    x = np.ldexp(r.uniform(1.0, 2.0, n), e)
    p = np.ldexp(1.0, np.arange(lo, hi))
    k = np.arange(1.0, 20000.0)
    a, b, c = np.meshgrid(*[np.arange(0.0, 12.0)] * 3, indexing="ij")
    lattice = (a * a + b * b + c * c).ravel()[1:]
    dx = r.uniform(1e-4, 1.0, 8)
    return np.concatenate([x, p, np.nextafter(p, 0.0), np.nextafter(p, np.inf), k * k, 1.0 / k,
                           *[lattice * d * d for d in dx], *[np.sqrt(lattice) * d for d in dx]])


def ulps(got, exact):
    """Distance from a long double in units of the double's last place."""
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("no 64-bit significands on this host")
    return np.abs((got.astype(np.longdouble) - exact) / np.spacing(np.abs(got)).astype(np.longdouble))


def test_reciprocals():
    x = arguments(1 << 20, -200, 200, 1)
    big = x.astype(np.longdouble)
    assert ulps(on_gpu(RSQRT, x), 1 / np.sqrt(big)).max() < 1.0
    assert ulps(on_gpu(RCP, x), 1 / big).max() < 0.6
    d = np.abs(on_gpu(RSQRT, x) - on_gpu(CUDA_RSQRT, x)) / np.spacing(on_gpu(CUDA_RSQRT, x))
    assert d.max() <= 2.0      # CUDA's own is within 1 ulp


def test_square_roots_are_those_of_sqrt():
    x = arguments(1 << 24, -200, 200, 2)
    ref = on_gpu(CUDA_SQRT, x)
    assert np.array_equal(ref, np.sqrt(x))
    assert np.array_equal(on_gpu(SQRT, x), ref)
    # the length of a bond, at rest and stretched
    for f in (1.0, 1.0 + 1e-15, 1.0 - 1e-6, 1.003):
        assert np.array_equal(on_gpu(LENGTH, x, np.sqrt(x) * f), ref)


def test_quotients():
    x = arguments(1 << 20, -60, 60, 3)
    r = np.random.default_rng(4)
    for y in (x * r.uniform(1.0, 6.0, len(x)), np.full(len(x), 3.015e-3), r.permutation(x)):
        exact = x.astype(np.longdouble) / y.astype(np.longdouble)
        got = on_gpu(QUOTIENT, x, y)
        assert ulps(got, exact).max() < 0.6
        assert (np.abs(got - on_gpu(CUDA_QUOTIENT, x, y)) <= np.spacing(got)).all()
