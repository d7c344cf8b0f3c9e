// pd_bond64.cuh -- the per-bond arithmetic of the FP64 kernels off the serial order, shared by those
// that gather from global memory (pd_force64_fast.cu) and from tiles (pd_tile64.cu): a body's results
// do not depend on which of them runs.
#pragma once
#include "pd_common.cuh"

namespace pd {

// Rows whose terms are summed from zero before they join the total of a point, in row order
constexpr int SEG64 = 16;

// The elementary functions below are refined from the hardware's approximations (about 22 bits), without the
// special cases of CUDA's own (which cost a branch a call): arguments are normal
// numbers. Their errors against CUDA's functions and against 64-bit significands: tests/test_gpu_math64.py.
//
// 1 / sqrt(x): one step of Chebyshev's third-order iteration (Traub, Iterative Methods for the Solution of
// Equations, 1964) for y^-2 = x. With e = 1 - x y^2 it is y + y (e / 2 + 3 e^2 / 8). Within 1 ulp.
__device__ __forceinline__ double rsqrt3(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-(x * y), y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}

// 1 / x: the same iteration for 1 / y = x. With e = 1 - x y it is y + y (e + e^2). Within 0.6 ulp.
__device__ __forceinline__ double rcp3(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// sqrt(x), with h an approximation of 1 / sqrt(x) within a few ulps: a Newton step whose residual x - l^2 is
// exact in a fused multiply-add (Markstein, Computation of elementary functions on the IBM RISC System/6000
// processor, 1990). Equal to sqrt() on all 2^24 arguments tried; a body at rest is free of force because
// the lengths of its bonds are.
__device__ __forceinline__ double sqrt_of(double x, double h) {
  const double l = x * h;
  return fma(fma(-l, l, x), 0.5 * h, l);
}

// a / b from rb = 1 / b rounded: Markstein's correction of a quotient (the same paper). Within 0.6 ulp.
__device__ __forceinline__ double quotient(double a, double b, double rb) {
  const double q = a * rb;
  return fma(fma(-q, b, a), rb, q);
}

// eps = (l - L) / L > eps_c: the division only where l - L is not clearly below eps_c L.
// thr = eps_c less a margin far above the rounding of either side, -inf for eps_c <= 0
__device__ __forceinline__ double fail_threshold(double epsc) {
  return epsc > 0 ? epsc * (1.0 - 1e-14) : (epsc <= 0 ? -INFINITY : epsc);
}
__device__ __forceinline__ bool fails64(double l2, double e, double Ls, double L, double thr,
                                        double epsc) {
  if (!(Ls > 0) || e < thr * L) return false;
  return (sqrt(l2) - L) / L > epsc;
}

// The influence functions other than the linear one (kernels.jl:10-52), rdelta = 1 / delta. The B-spline
// is evaluated in the serial kernels' form and order: near xi = 1 its terms cancel and leave their rounding,
// which another form would not share (35,520-point OSB block at a horizon of 2.015 spacings: 77 us a step
// with a division a bond, 53 so).
__device__ __forceinline__ double omega64(int kernel, double delta, double rdelta, double L) {
  if (kernel == KER_CONST_ONE) return 1.0;
  const double xi = quotient(L, delta, rdelta);
  const double x2 = xi * xi, x3 = x2 * xi;
  const double in = 2.0 / 3.0 - 4 * x2 + 4 * x3, out = 4.0 / 3.0 - 4 * xi + 4 * x2 - 4.0 / 3.0 * x3;
  return xi > 0 && xi <= 1 ? (xi <= 0.5 ? in : out) : 0.0;
}

__device__ __forceinline__ void nan_flag(const DevBody& d, int kstep, double x, double y, double z) {
  if (isnan(x) || isnan(y) || isnan(z)) {
    const long long step = d.ctrl->base + kstep;
    if (atomicExch(&d.ctrl->err, 1) == 0) d.ctrl->err_step = step;
    else atomicMin(&d.ctrl->err_step, step);
  }
}

// the bond from eta = {dx, dy, dz} and the signed length Ls: g = 1 / (l L), e = l - L. l L squared has to be a
// normal number: lengths between about 1e-76 and 1e+76
struct Bond64 {
  double L, l2, g, e;
  __device__ __forceinline__ Bond64(double dx, double dy, double dz, double Ls) {
    L = fabs(Ls);
    l2 = (dx * dx + dy * dy) + dz * dz;
    g = rsqrt3(l2 * (L * L));
    e = sqrt_of(l2, g * L) - L;
  }
};

}  // namespace pd
