// pd_force64.cu -- FP64 force-density kernels (the plain FP64 path).
//
// Compiled with -fmad=false: Julia rounds every product and sum separately, and these kernels
// keep the reference's evaluation order, so with one lane per point (G = 1, "exact order")
// the per-point results equal the serial CPU restatement bit for bit:
//   - BB: one bond sweep (failure test, then the bond force) in bond order;
//   - OSB / CMat: phase A per point (failure, damage, weighted volume and dilatation, or the
//     deformation gradient and stress), phase B gathers the force density. The reference
//     scatters b_j -= p V_i while it processes point i; phase B reproduces the order in which
//     those scattered terms reach b_i in the serial loop: first the terms of neighbours j < i
//     (ascending j), then the own bonds of i, then the terms of neighbours j > i.
// The other mappings run the kernels of pd_force64_fast.cu, and here the phase-B kernels for
// directed bond states, several parameter sets and ZEMWan (fixed butterfly order over the lanes
// of a point: deterministic, not bit-identical to the serial order).
#include "pd_common.cuh"
#include "pd_launch.h"
#include "pd_math64.cuh"

namespace pd {

__device__ __forceinline__ void flag_nan(const DevBody& d, int kstep, double x, double y, double z) {
  if (isnan(x) || isnan(y) || isnan(z)) {
    long long step = d.ctrl->base + kstep;
    if (atomicExch(&d.ctrl->err, 1) == 0) d.ctrl->err_step = step;
    else atomicMin(&d.ctrl->err_step, step);
  }
}

// new bond_active word of a row after the failure tests of its lanes; the warp owns the word
__device__ __forceinline__ void commit_row64(unsigned int* bits, long long word_idx, unsigned old,
                                             bool act, int lane) {
  const unsigned nw = __ballot_sync(0xffffffffu, act);
  if (lane == 0 && nw != old) bits[word_idx] = nw;
}

// -------------------------------------------------------------------------------------------
// BB: bond_based.jl:125-180 (calc_failure! storing the bond length, force_density_point!)
// -------------------------------------------------------------------------------------------
// ESC: the bond's surface correction factor multiplies its force (bond_based.jl:156, 175)
template <bool MULTI, bool ESC>
__global__ void PD_LB64 k_bb64(DevBody d, int kstep) {
  if (d.ctrl->err) return;
  PD_SLICE_LOOP(1) {
    PD_SLICE_SETUP
    double bx = 0.0, by = 0.0, bz = 0.0;
    int na = 0;
    const double4 xi = valid ? ld4_64(d.cur + i) : make_double4(0, 0, 0, 0);
    const DevParam& P = d.params[valid ? (d.meta[i] & META_PID_MASK) : 0];
    for (int r = 0; r < rows; r++) {
      const long long wi = (sbase >> 5) + r;
      const unsigned word = d.bits[wi];
      const int k = r;
      bool act = false;
      if (k < cnt) {
        const long long b = sbase + (long long)r * 32 + lane;
        const int j = __ldg(d.nbr + b);
        const double Ls = __ldg(d.len64 + b);
        const double L = fabs(Ls);
        const double4 xj = ld4_64(d.cur + j);
        const double dx = xj.x - xi.x, dy = xj.y - xi.y, dz = xj.z - xi.z;
        const double l = sqrt((dx * dx + dy * dy) + dz * dz);
        {
          const double eps = (l - L) / L;
          act = ((word >> lane) & 1u) && !(eps > P.epsc && Ls > 0);
          const double om = act ? (ESC ? __ldg(d.sc64 + b) : 1.0) : 0.0;
          double sc;
          if (MULTI) {
            const double bcj = d.params[d.meta[j] & META_PID_MASK].bc;
            sc = om * (P.bc + bcj) / 2 * eps * xj.w;
          } else {
            sc = om * P.bc * eps * xj.w;
          }
          bx += sc * dx / l;
          by += sc * dy / l;
          bz += sc * dz / l;
        }
      }
      na += act;
      commit_row64(d.bits, wi, word, act, lane);
    }
    if (valid) {
      d.b64[3 * i] = bx; d.b64[3 * i + 1] = by; d.b64[3 * i + 2] = bz;
      d.n_active[i] = na;
      flag_nan(d, kstep, bx, by, bz);
    }
  }
}

// -------------------------------------------------------------------------------------------
// OSB phase A: calc_failure! (ordinary_state_based.jl:107-126), calc_damage!,
// calc_weighted_volume (:176-189), calc_dilatation (:191-204), c1, c2 (:135-136)
// -------------------------------------------------------------------------------------------
// ESC: the bond factor beta in the weighted volume and the dilatation (:182, :198)
template <bool ESC>
__global__ void PD_LB64 k_osb_a64(DevBody d, int kstep) {
  if (d.ctrl->err) return;
  PD_SLICE_LOOP(1) {
    PD_SLICE_SETUP
    double wvol = 0.0;
    int na = 0;
    const DevParam& P = d.params[valid ? (d.meta[i] & META_PID_MASK) : 0];
    const double4 xi = valid ? ld4_64(d.cur + i) : make_double4(0, 0, 0, 0);
    const double4 Xi = valid ? ld4_64(d.X0 + i) : make_double4(0, 0, 0, 0);
    for (int r = 0; r < rows; r++) {
      const long long wi = (sbase >> 5) + r;
      const unsigned word = d.bits[wi];
      const int k = r;
      bool act = false;
      if (k < cnt) {
        const long long b = sbase + (long long)r * 32 + lane;
        const int j = __ldg(d.nbr + b);
        const double Ls = __ldg(d.len64 + b);
        const double L = fabs(Ls);
        const double4 xj = ld4_64(d.cur + j), Xj = ld4_64(d.X0 + j);
        const double dx = xj.x - xi.x, dy = xj.y - xi.y, dz = xj.z - xi.z;
        const double l = sqrt((dx * dx + dy * dy) + dz * dz);
        const double eps = (l - L) / L;
        act = ((word >> lane) & 1u) && !(eps > P.epsc && Ls > 0);
        const double DX = Xj.x - Xi.x, DY = Xj.y - Xi.y, DZ = Xj.z - Xi.z;
        const double om = act ? omega_of(d.kernel, P.delta, L) : 0.0;
        const double bet = ESC ? __ldg(d.sc64 + b) : 1.0;
        wvol += om * bet * ((DX * DX + DY * DY) + DZ * DZ) * xj.w;
      }
      na += act;
      commit_row64(d.bits, wi, word, act, lane);
    }
    double dil = 0.0;
    // second sweep of the reference with c1 = 3 / wvol inside every term; the bits were
    // written above by lane 0 of the warp, so the decision is recomputed from the same eps
    __syncwarp();
    const double c1d = 3.0 / wvol;
    for (int r = 0; r < rows; r++) {
      const int k = r;
      if (k >= cnt || wvol == 0.0) continue;
      const long long b = sbase + (long long)r * 32 + lane;
      const int j = __ldg(d.nbr + b);
      const double Ls = __ldg(d.len64 + b);
      const double L = fabs(Ls);
      const double4 xj = ld4_64(d.cur + j);
      const double dx = xj.x - xi.x, dy = xj.y - xi.y, dz = xj.z - xi.z;
      const double l = sqrt((dx * dx + dy * dy) + dz * dz);
      const double eps = (l - L) / L;
      const bool act = bond_bit_live(d.bits, b) && !(eps > P.epsc && Ls > 0);
      const double om = act ? omega_of(d.kernel, P.delta, L) : 0.0;
      dil += om * (ESC ? __ldg(d.sc64 + b) : 1.0) * c1d * L * (l - L) * xj.w;
    }
    if (valid) {
      double c1 = 0.0, c2 = 0.0;
      if (wvol != 0.0) {
        c1 = 15.0 * P.G / wvol;
        c2 = dil * (3.0 * P.K / wvol - c1 / 3.0);
      }
      d.coef64[i] = make_double4(c1, c2, wvol, dil);
      d.n_active[i] = na;
    }
  }
}

// p = omega beta (c2 L + c1 (l - L)) / l (ordinary_state_based.jl:144), coefficients of the
// bond owner o with the partner q (ParameterHandler form :165-166 when MULTI)
template <bool MULTI>
__device__ __forceinline__ double osb_s64(const double4& co, const DevParam& Po, const DevParam& Pq,
                                          double om, double bet, double L, double l) {
  double c1, c2;
  if (MULTI) {
    c1 = 15.0 * (Po.G + Pq.G) / (2 * co.z);
    c2 = co.w * (3.0 * (Po.K + Pq.K) / (2 * co.z) - c1 / 3.0);
  } else {
    c1 = co.x;
    c2 = co.y;
  }
  return om * bet * (c2 * L + c1 * (l - L)) / l;
}

// -------------------------------------------------------------------------------------------
// OSB phase B: force_density_point! (ordinary_state_based.jl:128-174) in gather form
// -------------------------------------------------------------------------------------------
// ESC: beta of the bond, which is also the factor of its reverse bond (equal by construction)
template <bool MULTI, bool ESC>
__global__ void PD_LB64 k_osb_b64(DevBody d, int kstep) {
  if (d.ctrl->err) return;
  PD_SLICE_LOOP(1) {
    PD_SLICE_SETUP
    double bx = 0.0, by = 0.0, bz = 0.0;
    const double4 xi = valid ? ld4_64(d.cur + i) : make_double4(0, 0, 0, 0);
    const DevParam& Pi = d.params[valid ? (d.meta[i] & META_PID_MASK) : 0];
    const double4 ci = valid ? d.coef64[i] : make_double4(0, 0, 0, 0);
    const bool own = ci.z != 0.0;
    // own term of the bond in slot b
    auto own_term = [&](long long b) {
      const int j = __ldg(d.nbr + b);
      const double L = fabs(__ldg(d.len64 + b));
      const double4 xj = ld4_64(d.cur + j);
      const double dx = xj.x - xi.x, dy = xj.y - xi.y, dz = xj.z - xi.z;
      const double l = sqrt((dx * dx + dy * dy) + dz * dz);
      const bool act = bond_bit(d.bits, b);
      const double om = act ? omega_of(d.kernel, Pi.delta, L) : 0.0;
      const DevParam& Pj = MULTI ? d.params[d.meta[j] & META_PID_MASK] : Pi;
      const double sc = osb_s64<MULTI>(ci, Pi, Pj, om, ESC ? __ldg(d.sc64 + b) : 1.0, L, l);
      bx += sc * dx * xj.w;
      by += sc * dy * xj.w;
      bz += sc * dz * xj.w;
    };
    // term that j's loop scatters into b_i through its bond j -> i
    auto nbr_term = [&](long long b) {
      const int j = __ldg(d.nbr + b);
      const double4 cj = d.coef64[j];
      if (cj.z == 0.0) return;  // j returned early (iszero(wvol))
      const double L = fabs(__ldg(d.len64 + b));
      const double4 xj = ld4_64(d.cur + j);
      const double dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
      const double l = sqrt((dx * dx + dy * dy) + dz * dz);
      const bool act = d.sym ? bond_bit(d.bits, b) : bond_bit(d.bits, rev_slot(d, b, j));
      const DevParam& Pj = d.params[d.meta[j] & META_PID_MASK];
      const double om = act ? omega_of(d.kernel, Pj.delta, L) : 0.0;
      const double sc = osb_s64<MULTI>(cj, Pj, Pi, om, ESC ? __ldg(d.sc64 + b) : 1.0, L, l);
      bx += -(sc * dx) * xj.w;
      by += -(sc * dy) * xj.w;
      bz += -(sc * dz) * xj.w;
    };
    // the serial scatter order: neighbours j < i, own bonds, neighbours j > i
    for (int r = 0; r < rows; r++) {
      const int k = r;
      const long long b = sbase + (long long)r * 32 + lane;
      if (k < cnt && __ldg(d.nbr + b) < i) nbr_term(b);
    }
    if (own)
      for (int r = 0; r < rows; r++) {
        const int k = r;
        if (k < cnt) own_term(sbase + (long long)r * 32 + lane);
      }
    for (int r = 0; r < rows; r++) {
      const int k = r;
      const long long b = sbase + (long long)r * 32 + lane;
      if (k < cnt && __ldg(d.nbr + b) > i) nbr_term(b);
    }
    if (valid) {
      d.b64[3 * i] = bx; d.b64[3 * i + 1] = by; d.b64[3 * i + 2] = bz;
      flag_nan(d, kstep, bx, by, bz);
    }
  }
}

// -------------------------------------------------------------------------------------------
// OSB phase B off the serial order where bond states differ between the two directions of a
// pair or parameter sets meet (pd_force64_fast.cu has the other case): two rows of gathers in
// flight per lane, the point's own term and its neighbour's term of a bond summed before one
// division by l.
// -------------------------------------------------------------------------------------------
// omega beta (c2 L + c1 (l - L)) of a bond owner o with partner q: osb_s64 before its division
template <bool MULTI>
__device__ __forceinline__ double osb_num64(const double4& co, const DevParam& Po, const DevParam& Pq,
                                            double om, double bet, double L, double l) {
  double c1, c2;
  if (MULTI) {
    c1 = 15.0 * (Po.G + Pq.G) / (2 * co.z);
    c2 = co.w * (3.0 * (Po.K + Pq.K) / (2 * co.z) - c1 / 3.0);
  } else {
    c1 = co.x;
    c2 = co.y;
  }
  return om * bet * (c2 * L + c1 * (l - L));
}

template <int G, bool MULTI, bool ESC>
__global__ void __launch_bounds__(256, 2) k_osb_b64g(DevBody d, int kstep) {
  if (d.ctrl->err) return;
  PD_SLICE_LOOP(G) {
    PD_SLICE_SETUP
    double bx = 0.0, by = 0.0, bz = 0.0;
    const DevParam& Pi = d.params[valid ? (d.meta[i] & META_PID_MASK) : 0];
    const double4 xi = valid ? ld4_64(d.cur + i) : make_double4(0, 0, 0, 0);
    const double4 ci = valid ? d.coef64[i] : make_double4(0, 0, 0, 0);
    const bool own = ci.z != 0.0;
    const int self = valid ? (int)i : 0;
    for (int r = 0; r < rows; r += 2) {
      const bool two = r + 1 < rows;
      const long long wi = (sbase >> 5) + r;
      const unsigned w0 = __ldg(d.bits + wi), w1 = two ? __ldg(d.bits + wi + 1) : 0u;
      const int k0 = r * G + gl, k1 = k0 + G;
      const bool h0 = k0 < cnt, h1 = two && k1 < cnt;
      const long long b0 = sbase + (long long)r * 32 + lane, b1 = b0 + 32;
      const int j0 = h0 ? __ldg(d.nbr + b0) : self, j1 = h1 ? __ldg(d.nbr + b1) : self;
      const double Ls0 = h0 ? __ldg(d.len64 + b0) : 1.0, Ls1 = h1 ? __ldg(d.len64 + b1) : 1.0;
      const double4 x0 = ld4_64(d.cur + j0), x1 = ld4_64(d.cur + j1);
      const double4 c0 = d.coef64[j0], c1 = d.coef64[j1];
#pragma unroll
      for (int u = 0; u < 2; u++) {
        if (!(u ? h1 : h0)) continue;
        const double4 xj = u ? x1 : x0;
        const double4 cj = u ? c1 : c0;
        const int j = u ? j1 : j0;
        const long long b = u ? b1 : b0;
        const double L = fabs(u ? Ls1 : Ls0);
        const double dx = xj.x - xi.x, dy = xj.y - xi.y, dz = xj.z - xi.z;
        const double l = sqrt((dx * dx + dy * dy) + dz * dz);
        const bool ai = ((u ? w1 : w0) >> lane) & 1u;
        const bool aj = d.sym ? ai : bond_bit(d.bits, rev_slot(d, b, j));
        const DevParam& Pj = d.params[d.meta[j] & META_PID_MASK];
        const double bet = ESC ? __ldg(d.sc64 + b) : 1.0;
        double num = 0.0;
        if (own && ai) num += osb_num64<MULTI>(ci, Pi, Pj, omega_of(d.kernel, Pi.delta, L), bet, L, l);
        // j returned early for a zero weighted volume (iszero(wvol))
        if (cj.z != 0.0 && aj)
          num += osb_num64<MULTI>(cj, Pj, Pi, omega_of(d.kernel, Pj.delta, L), bet, L, l);
        const double sc = num / l * xj.w;
        bx += sc * dx;
        by += sc * dy;
        bz += sc * dz;
      }
    }
    if (G > 1) { bx = group_sum<G>(bx); by = group_sum<G>(by); bz = group_sum<G>(bz); }
    if (valid && gl == 0) {
      d.b64[3 * i] = bx; d.b64[3 * i + 1] = by; d.b64[3 * i + 2] = bz;
      flag_nan(d, kstep, bx, by, bz);
    }
  }
}

// -------------------------------------------------------------------------------------------
// CMat phase A: calc_failure! (bond_system.jl:309-327), calc_damage!,
// calc_deformation_gradient! (correspondence.jl:193-214), too_much_damage! (:288-298),
// calc_first_piola_kirchhoff! (:216-224)
// -------------------------------------------------------------------------------------------
__global__ void PD_LB64 k_c_a64(DevBody d, int kstep) {
  if (d.ctrl->err) return;
  PD_SLICE_LOOP(1) {
    PD_SLICE_SETUP
    double K[9], Ft[9];
    for (int q = 0; q < 9; q++) { K[q] = 0.0; Ft[q] = 0.0; }
    int na = 0;
    const unsigned meta = valid ? d.meta[i] : 0u;
    const DevParam& P = d.params[meta & META_PID_MASK];
    const double4 xi = valid ? ld4_64(d.cur + i) : make_double4(0, 0, 0, 0);
    const double4 Xi = valid ? ld4_64(d.X0 + i) : make_double4(0, 0, 0, 0);
    for (int r = 0; r < rows; r++) {
      const long long wi = (sbase >> 5) + r;
      const unsigned word = d.bits[wi];
      const int k = r;
      bool act = false;
      if (k < cnt) {
        const long long b = sbase + (long long)r * 32 + lane;
        const int j = __ldg(d.nbr + b);
        const double Ls = __ldg(d.len64 + b);
        const double L = fabs(Ls);
        const double4 xj = ld4_64(d.cur + j), Xj = ld4_64(d.X0 + j);
        const double dx[3] = {xj.x - xi.x, xj.y - xi.y, xj.z - xi.z};
        const double l = sqrt(dot3(dx, dx));
        const double eps = (l - L) / L;
        act = ((word >> lane) & 1u) && !(eps > P.epsc && Ls > 0);
        const double DX[3] = {Xj.x - Xi.x, Xj.y - Xi.y, Xj.z - Xi.z};
        const double om = act ? omega_of(d.kernel, P.delta, L) : 0.0;
        const double temp = om * xj.w;
        for (int c = 0; c < 3; c++)
          for (int q = 0; q < 3; q++) {
            K[q + 3 * c] = K[q + 3 * c] + temp * (DX[q] * DX[c]);
            Ft[q + 3 * c] = Ft[q + 3 * c] + temp * (dx[q] * DX[c]);
          }
      }
      na += act;
      commit_row64(d.bits, wi, word, act, lane);
    }
    const bool killed = valid && c_point64(d, P, i, meta, cnt, na, K, Ft);
    if (!d.sym) {
      // directed bond states: a killed point loses all its bonds (correspondence.jl:293)
      const unsigned kill_mask = __ballot_sync(0xffffffffu, killed);
      if (kill_mask && lane == 0)
        for (int r = 0; r < rows; r++) d.bits[(sbase >> 5) + r] &= ~kill_mask;
    }
  }
}

// -------------------------------------------------------------------------------------------
// CMat phase B: c_force_density! (correspondence.jl:226-279) in gather form; the stabilisation
// term is (w beta) z for ZEMSilling (C1 null) and (w C_1) z for ZEMWan
// -------------------------------------------------------------------------------------------
__device__ __forceinline__ void c_bond_t64(const double* F, const double* PK, const double* C1,
                                           double beta, double om, const double* DX,
                                           const double* dx, double* t) {
  double FD[3], z[3], W[9], WD[3], tz[3];
  matvec3(F, DX, FD);
  for (int q = 0; q < 3; q++) z[q] = dx[q] - FD[q];
  if (C1) {
    double W1[9];
    for (int q = 0; q < 9; q++) W1[q] = om * C1[q];
    matvec3(W1, z, tz);
  } else {
    const double ob = om * beta;
    for (int q = 0; q < 3; q++) tz[q] = ob * z[q];
  }
  for (int q = 0; q < 9; q++) W[q] = om * PK[q];
  matvec3(W, DX, WD);
  for (int q = 0; q < 3; q++) t[q] = WD[q] + tz[q];
}

template <int G, bool EXACT>
__global__ void PD_LB64 k_c_b64(DevBody d, int kstep) {
  if (d.ctrl->err) return;
  PD_SLICE_LOOP(G) {
    PD_SLICE_SETUP
    double bx = 0.0, by = 0.0, bz = 0.0;
    const double4 xi = valid ? ld4_64(d.cur + i) : make_double4(0, 0, 0, 0);
    const double4 Xi = valid ? ld4_64(d.X0 + i) : make_double4(0, 0, 0, 0);
    const unsigned mi = valid ? d.meta[i] : META_KILLED;
    const DevParam& Pi = d.params[mi & META_PID_MASK];
    const bool own = !(mi & META_KILLED);
    const bool wan = d.zem == ZEM_WAN;
    double Fi[9], PKi[9], Ci[9];
    for (int q = 0; q < 9; q++) {
      Fi[q] = own ? d.F64[9 * i + q] : 0.0;
      PKi[q] = own ? d.PK64[9 * i + q] : 0.0;
      Ci[q] = own && wan ? d.C164[9 * i + q] : 0.0;
    }
    auto own_term = [&](long long b) {
      const int j = __ldg(d.nbr + b);
      const double L = fabs(__ldg(d.len64 + b));
      const double4 xj = ld4_64(d.cur + j), Xj = ld4_64(d.X0 + j);
      const double DX[3] = {Xj.x - Xi.x, Xj.y - Xi.y, Xj.z - Xi.z};
      const double dx[3] = {xj.x - xi.x, xj.y - xi.y, xj.z - xi.z};
      const bool act = bond_bit(d.bits, b);
      const double om = act ? omega_of(d.kernel, Pi.delta, L) : 0.0;
      double t[3];
      c_bond_t64(Fi, PKi, wan ? Ci : nullptr, Pi.beta, om, DX, dx, t);
      bx += t[0] * xj.w; by += t[1] * xj.w; bz += t[2] * xj.w;
    };
    auto nbr_term = [&](long long b) {
      const int j = __ldg(d.nbr + b);
      const unsigned mj = d.meta[j];
      if (mj & META_KILLED) return;  // j returned early after too_much_damage!
      const double L = fabs(__ldg(d.len64 + b));
      const bool act = d.sym ? bond_bit(d.bits, b) : bond_bit(d.bits, rev_slot(d, b, j));
      const DevParam& Pj = d.params[mj & META_PID_MASK];
      const double4 xj = ld4_64(d.cur + j), Xj = ld4_64(d.X0 + j);
      const double DX[3] = {Xi.x - Xj.x, Xi.y - Xj.y, Xi.z - Xj.z};
      const double dx[3] = {xi.x - xj.x, xi.y - xj.y, xi.z - xj.z};
      const double om = act ? omega_of(d.kernel, Pj.delta, L) : 0.0;
      double Fj[9], PKj[9], Cj[9], t[3];
      for (int q = 0; q < 9; q++) { Fj[q] = d.F64[9 * (long long)j + q]; PKj[q] = d.PK64[9 * (long long)j + q]; }
      if (wan)
        for (int q = 0; q < 9; q++) Cj[q] = d.C164[9 * (long long)j + q];
      c_bond_t64(Fj, PKj, wan ? Cj : nullptr, Pj.beta, om, DX, dx, t);
      bx += -t[0] * xj.w; by += -t[1] * xj.w; bz += -t[2] * xj.w;
    };
    if (EXACT) {
      for (int r = 0; r < rows; r++) {
        const int k = r * G + gl;
        const long long b = sbase + (long long)r * 32 + lane;
        if (k < cnt && __ldg(d.nbr + b) < i) nbr_term(b);
      }
      if (own)
        for (int r = 0; r < rows; r++) {
          const int k = r * G + gl;
          if (k < cnt) own_term(sbase + (long long)r * 32 + lane);
        }
      for (int r = 0; r < rows; r++) {
        const int k = r * G + gl;
        const long long b = sbase + (long long)r * 32 + lane;
        if (k < cnt && __ldg(d.nbr + b) > i) nbr_term(b);
      }
    } else {
      for (int r = 0; r < rows; r++) {
        const int k = r * G + gl;
        if (k >= cnt) continue;
        const long long b = sbase + (long long)r * 32 + lane;
        if (own) own_term(b);
        nbr_term(b);
      }
    }
    if (G > 1) { bx = group_sum<G>(bx); by = group_sum<G>(by); bz = group_sum<G>(bz); }
    if (valid && gl == 0) {
      d.b64[3 * i] = bx; d.b64[3 * i + 1] = by; d.b64[3 * i + 2] = bz;
      flag_nan(d, kstep, bx, by, bz);
    }
  }
}

// cauchy_stress (stress.jl:112-116) of the stored F, for the export of the CMat stress field
__global__ void k_cauchy64(DevBody d, const double* F, int from_h32, double* out) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n) return;
  const DevParam P = d.params[d.meta[i] & META_PID_MASK];
  double Fm[9], Pm[9], Ps[9], S[9];
  for (int k = 0; k < 9; k++)
    Fm[k] = from_h32 ? (double)d.H32[9 * i + k] + ((k % 4) == 0 ? 1.0 : 0.0) : F[9 * i + k];
  pk1_64(d.cmodel, P, Fm, Pm);
  const double J = det3(Fm), iJ = 1 / J;
  for (int k = 0; k < 9; k++) Ps[k] = iJ * Pm[k];
  matmulT3(Ps, Fm, S);
  const bool killed = d.meta[i] & META_KILLED;
  for (int k = 0; k < 9; k++) out[9 * i + k] = killed ? 0.0 : S[k];
}

// ------------------------------------------------------------------------------------------
// launchers
// ------------------------------------------------------------------------------------------
#define PD_DISPATCH_G(G, CALL)                  \
  switch (G) {                                  \
    case 1: { constexpr int GG = 1; CALL; } break;  \
    case 2: { constexpr int GG = 2; CALL; } break;  \
    case 4: { constexpr int GG = 4; CALL; } break;  \
    case 8: { constexpr int GG = 8; CALL; } break;  \
    case 16: { constexpr int GG = 16; CALL; } break; \
    default: { constexpr int GG = 32; CALL; } break; \
  }

static int grid_for(long long nslices, int block) {
  long long warps = nslices;
  long long blocks = (warps + block / 32 - 1) / (block / 32);
  if (blocks < 1) blocks = 1;
  if (PD_GRID_BLOCKS_PER_SM > 0 && blocks > 148LL * PD_GRID_BLOCKS_PER_SM)
    blocks = 148LL * PD_GRID_BLOCKS_PER_SM;
  return (int)blocks;
}

// the serial order (one lane per point)
static int launch_exact64(const DevBody& d, int grid, int block, int kstep, bool A, bool B, cudaStream_t s) {
  const bool esc = d.sc64 != nullptr;
  if (d.material == MAT_BB) {
    if (!A) return 0;
    if (d.multi && esc) k_bb64<true, true><<<grid, block, 0, s>>>(d, kstep);
    else if (d.multi) k_bb64<true, false><<<grid, block, 0, s>>>(d, kstep);
    else if (esc) k_bb64<false, true><<<grid, block, 0, s>>>(d, kstep);
    else k_bb64<false, false><<<grid, block, 0, s>>>(d, kstep);
    return 1;
  }
  if (d.material == MAT_OSB) {
    if (A && esc) k_osb_a64<true><<<grid, block, 0, s>>>(d, kstep);
    else if (A) k_osb_a64<false><<<grid, block, 0, s>>>(d, kstep);
    if (B) {
      if (d.multi && esc) k_osb_b64<true, true><<<grid, block, 0, s>>>(d, kstep);
      else if (d.multi) k_osb_b64<true, false><<<grid, block, 0, s>>>(d, kstep);
      else if (esc) k_osb_b64<false, true><<<grid, block, 0, s>>>(d, kstep);
      else k_osb_b64<false, false><<<grid, block, 0, s>>>(d, kstep);
    }
  } else {
    if (A) k_c_a64<<<grid, block, 0, s>>>(d, kstep);
    if (B) k_c_b64<1, true><<<grid, block, 0, s>>>(d, kstep);
  }
  return (A ? 1 : 0) + (B ? 1 : 0);
}

int launch_force64(const DevBody& d, const LaunchCfg& c, int kstep, int phase, cudaStream_t s) {
  const int grid = grid_for(d.nslices, c.block);
  const bool A = phase != 2, B = phase != 1;
  if (c.exact) return launch_exact64(d, grid, c.block, kstep, A, B, s);
  if (d.material == MAT_BB && !A) return 0;
  int launches = 0;
  if (A) {
    launch_force64_fast(d, c, kstep, 1, s);
    launches++;
  }
  if (!B || d.material == MAT_BB) return launches;
  if (fast64_supported(d)) {
    launch_force64_fast(d, c, kstep, 2, s);
  } else if (d.material == MAT_OSB) {
    const bool esc = d.sc64 != nullptr;
    if (d.multi && esc) { PD_DISPATCH_G(d.lg, (k_osb_b64g<GG, true, true><<<grid, c.block, 0, s>>>(d, kstep))); }
    else if (d.multi) { PD_DISPATCH_G(d.lg, (k_osb_b64g<GG, true, false><<<grid, c.block, 0, s>>>(d, kstep))); }
    else if (esc) { PD_DISPATCH_G(d.lg, (k_osb_b64g<GG, false, true><<<grid, c.block, 0, s>>>(d, kstep))); }
    else { PD_DISPATCH_G(d.lg, (k_osb_b64g<GG, false, false><<<grid, c.block, 0, s>>>(d, kstep))); }
  } else {
    PD_DISPATCH_G(d.lg, (k_c_b64<GG, false><<<grid, c.block, 0, s>>>(d, kstep)));
  }
  return launches + 1;
}

void launch_cauchy64(const DevBody& d, const double* F, int from_h32, double* out, cudaStream_t s) {
  int grid = (int)((d.n + 255) / 256);
  if (grid < 1) grid = 1;
  k_cauchy64<<<grid, 256, 0, s>>>(d, F, from_h32, out);
}

}  // namespace pd
