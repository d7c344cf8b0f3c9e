// pd_point32.cuh -- the per-point part of the FP32 correspondence material: 3x3 algebra, the stress
// models and the phase-B state, shared by the kernels of pd_force32.cu and pd_tile32.cu.
#pragma once
#include "pd_bond32.cuh"
#include "pd_common.cuh"

namespace pd {

// ------------------------------------------------------------------------------------------
// FP32 3x3 helpers (column-major) for the correspondence material
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ void fcross(const float* a, const float* b, float* c) {
  c[0] = a[1] * b[2] - a[2] * b[1];
  c[1] = a[2] * b[0] - a[0] * b[2];
  c[2] = a[0] * b[1] - a[1] * b[0];
}
__device__ __forceinline__ void finv3(const float* A, float* R) {
  float x0[3] = {A[0], A[1], A[2]}, y0[3], y1[3], y2[3];
  fcross(A + 3, A + 6, y0);
  const float d = x0[0] * y0[0] + x0[1] * y0[1] + x0[2] * y0[2];
  for (int k = 0; k < 3; k++) { x0[k] /= d; y0[k] /= d; }
  fcross(A + 6, x0, y1);
  fcross(x0, A + 3, y2);
  for (int c = 0; c < 3; c++) { R[3 * c] = y0[c]; R[1 + 3 * c] = y1[c]; R[2 + 3 * c] = y2[c]; }
}
__device__ __forceinline__ void fmatmul(const float* A, const float* B, float* C) {
  for (int r = 0; r < 3; r++)
    for (int c = 0; c < 3; c++)
      C[r + 3 * c] = A[r] * B[3 * c] + A[r + 3] * B[1 + 3 * c] + A[r + 6] * B[2 + 3 * c];
}

// P(F = I + H) of the reference's models, written without the cancelling F^T F - I
static __device__ void pk1_32(int cmodel, const DevParam& p, const float* H, float* P) {
  float E[9], S[9], HS[9];
  for (int r = 0; r < 3; r++)
    for (int c = 0; c < 3; c++) {
      const float hth = H[3 * r] * H[3 * c] + H[1 + 3 * r] * H[1 + 3 * c] + H[2 + 3 * r] * H[2 + 3 * c];
      E[r + 3 * c] = 0.5f * (H[r + 3 * c] + H[c + 3 * r] + hth);
    }
  const float trE = E[0] + E[4] + E[8];
  if (cmodel == CM_SVK) {
    // S = lambda tr(E) I + 2 mu E
    for (int k = 0; k < 9; k++) S[k] = 2.f * p.muf * E[k] + ((k % 4) == 0 ? p.lambdaf * trE : 0.f);
  } else {
    // J - 1 = tr H + (principal 2x2 minors of H) + det H
    const float m2 = (H[0] * H[4] - H[3] * H[1]) + (H[0] * H[8] - H[6] * H[2]) + (H[4] * H[8] - H[7] * H[5]);
    float dH;
    {
      float c[3];
      fcross(H + 3, H + 6, c);
      dH = H[0] * c[0] + H[1] * c[1] + H[2] * c[2];
    }
    const float jm1 = (H[0] + H[4] + H[8]) + m2 + dH;
    const float J = 1.f + jm1;
    float C[9], Ci[9], T[9];
    for (int k = 0; k < 9; k++) C[k] = 2.f * E[k] + ((k % 4) == 0 ? 1.f : 0.f);
    finv3(C, Ci);
    if (cmodel == CM_NEOHOOKE) {
      // S = mu (I - C^-1) + lambda ln J C^-1 = C^-1 (2 mu E + lambda ln J I)
      const float lj = p.lambdaf * log1pf(jm1);
      for (int k = 0; k < 9; k++) T[k] = 2.f * p.muf * E[k] + ((k % 4) == 0 ? lj : 0.f);
    } else {
      // NeoHookePenalty: S = C^-1 (2 G J^(-2/3) dev E + K/4 (J^2 - J^-2) I), P = 0 if J < eps
      if (!(J >= 2.220446049250313e-16f)) {
        for (int k = 0; k < 9; k++) P[k] = 0.f;
        return;
      }
      const float jp = expf(-2.f / 3.f * log1pf(jm1));
      const float iJ = 1.f / J;
      const float vol = 0.25f * p.Kf * (jm1 * (J + 1.f) * iJ) * (J + iJ);
      for (int k = 0; k < 9; k++)
        T[k] = 2.f * p.Gf * jp * (E[k] - ((k % 4) == 0 ? trE / 3.f : 0.f)) + ((k % 4) == 0 ? vol : 0.f);
    }
    fmatmul(Ci, T, S);
  }
  // P = F S = S + H S
  fmatmul(H, S, HS);
  for (int k = 0; k < 9; k++) P[k] = S[k] + HS[k];
}

// The phase-B state of a live point, from the scaled inverse shape tensor Kinv (the true
// K^-1 = Kinv / delta^5), P K^-1 (scaled the same way) and H = F - I. The bond term
// w (P K^-1 xi + S (dx - F xi)) is w (A xi + S du) with A = P K^-1 - S H, where S is the
// stabilising stiffness: ZEMSilling beta I (c_force_density!, correspondence.jl:226-251; beta
// in cst32), ZEMWan C : K^-1 (correspondence.jl:253-285, zem_stabilization.jl:32-42; the six
// entries of the symmetric S in zw32, from the nonzero entries of the Hooke tensor: a = (1 - nu)
// lambda / nu and lambda in the normal block, mu (both index orders) in the shear block).
__device__ __forceinline__ void c_state_store32(const DevBody& d, const DevParam& P, long long i,
                                                const float* PK, const float* Kinv, const float* H,
                                                float id5) {
  float A[9];
  float4* cs = d.cst32 + 3 * i;
  if (d.zem == ZEM_WAN) {
    const float a = P.zwaf, l = P.lambdaf, m = P.muf;
    const float S0 = (a * Kinv[0] + l * Kinv[4] + l * Kinv[8]) * id5;
    const float S1 = (l * Kinv[0] + a * Kinv[4] + l * Kinv[8]) * id5;
    const float S2 = (l * Kinv[0] + l * Kinv[4] + a * Kinv[8]) * id5;
    const float S01 = m * (Kinv[3] + Kinv[1]) * id5;
    const float S02 = m * (Kinv[6] + Kinv[2]) * id5;
    const float S12 = m * (Kinv[7] + Kinv[5]) * id5;
    const float Sm[9] = {S0, S01, S02, S01, S1, S12, S02, S12, S2};
    float SH[9];
    fmatmul(Sm, H, SH);
#pragma unroll
    for (int q = 0; q < 9; q++) A[q] = PK[q] * id5 - SH[q];
    d.zw32[2 * i] = make_float4(S0, S1, S2, S01);
    d.zw32[2 * i + 1] = make_float4(S02, S12, 0.f, 0.f);
  } else {
#pragma unroll
    for (int q = 0; q < 9; q++) A[q] = PK[q] * id5 - P.betaf * H[q];
  }
  cs[0] = make_float4(A[0], A[1], A[2], A[3]);
  cs[1] = make_float4(A[4], A[5], A[6], A[7]);
  cs[2] = make_float4(A[8], d.zem == ZEM_WAN ? 0.f : P.betaf, 0.f, 0.f);
}

// a killed point's phase-B state: no term of its own, none for its neighbours
__device__ __forceinline__ void c_state_clear32(const DevBody& d, long long i) {
  float4* cs = d.cst32 + 3 * i;
  cs[0] = make_float4(0.f, 0.f, 0.f, 0.f);
  cs[1] = make_float4(0.f, 0.f, 0.f, 0.f);
  cs[2] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (d.zem == ZEM_WAN) {
    d.zw32[2 * i] = make_float4(0.f, 0.f, 0.f, 0.f);
    d.zw32[2 * i + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// From the sums of a point: F - I, the kill decision (too_much_damage!, correspondence.jl:288-298)
// and the phase-B state. Returns whether the point is killed.
template <class SUMS>
__device__ __forceinline__ bool corr_point32(const DevBody& d, const DevParam& P, long long i,
                                             unsigned meta, int cnt, int na, const SUMS& S) {
  const float id = P.inv_delta;
  float k6[6];
  float2* ks = reinterpret_cast<float2*>(d.K32 + 6 * i);
  if constexpr (SUMS::FULL) {
    const float2 v01 = S.K01.value(), v23 = S.K23.value(), v45 = S.K45.value();
    k6[0] = v01.x; k6[1] = v01.y; k6[2] = v23.x; k6[3] = v23.y; k6[4] = v45.x; k6[5] = v45.y;
    ks[0] = make_float2(k6[0], k6[1]); ks[1] = make_float2(k6[2], k6[3]); ks[2] = make_float2(k6[4], k6[5]);
  } else {
    const float2 b0 = ks[0], b1 = ks[1], b2 = ks[2];
    k6[0] = b0.x; k6[1] = b0.y; k6[2] = b1.x; k6[3] = b1.y; k6[4] = b2.x; k6[5] = b2.y;
    if (S.dK[0] != 0.f || S.dK[1] != 0.f || S.dK[2] != 0.f) {  // a bond broke
#pragma unroll
      for (int q = 0; q < 6; q++) k6[q] -= S.dK[q];
      ks[0] = make_float2(k6[0], k6[1]); ks[1] = make_float2(k6[2], k6[3]); ks[2] = make_float2(k6[4], k6[5]);
    }
  }
  const float Km[9] = {k6[0], k6[3], k6[4],
                       k6[3], k6[1], k6[5],
                       k6[4], k6[5], k6[2]};
  float Kinv[9], Hm[9], H[9];
  finv3(Km, Kinv);
#pragma unroll
  for (int c = 0; c < 3; c++) {
    Hm[3 * c] = S.Hxy[c].x + S.nxy[c].x;
    Hm[3 * c + 1] = S.Hxy[c].y + S.nxy[c].y;
    Hm[3 * c + 2] = S.Hz[c] + S.nz[c];
  }
  fmatmul(Hm, Kinv, H);
  bool hasnan = false;
  for (int q = 0; q < 9; q++) { d.H32[9 * i + q] = H[q]; hasnan |= isnan(H[q]); }
  const double damage = 1.0 - (double)na / (double)cnt;
  const bool killed = (meta & META_KILLED) || (!(meta & META_HALO) && (damage > d.maxdmg || hasnan));
  if (killed) {
    if (!(meta & META_KILLED)) d.meta[i] = meta | META_KILLED;
    na = 0;
    c_state_clear32(d, i);
  } else {
    float Pm[9], PK[9];
    pk1_32(d.cmodel, P, H, Pm);
    fmatmul(Pm, Kinv, PK);
    c_state_store32(d, P, i, PK, Kinv, H, id * id * id * id * id);
  }
  d.n_active[i] = na;
  return killed;
}

}  // namespace pd
