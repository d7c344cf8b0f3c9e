// pd_math64.cuh -- FP64 3x3 algebra, the stress models and the per-point part of the
// correspondence material, in the reference's order of operations (compiled with -fmad=false),
// shared by the FP64 force kernels.
#pragma once
#include "pd_common.cuh"

namespace pd {

__device__ __forceinline__ double4 ld4_64(const double4* p) {
  const double2* q = reinterpret_cast<const double2*>(p);
  double2 a = __ldg(q), b = __ldg(q + 1);
  return make_double4(a.x, a.y, b.x, b.y);
}

__device__ __forceinline__ double dot3(const double* a, const double* b) {
  return (a[0] * b[0] + a[1] * b[1]) + a[2] * b[2];
}
__device__ __forceinline__ void cross3(const double* a, const double* b, double* c) {
  c[0] = a[1] * b[2] - a[2] * b[1];
  c[1] = a[2] * b[0] - a[0] * b[2];
  c[2] = a[0] * b[1] - a[1] * b[0];
}
// StaticArrays 3x3 det / inv (column-major), as the CPU restatement
__device__ __forceinline__ double det3(const double* A) {
  double c[3];
  cross3(A + 3, A + 6, c);
  return dot3(A, c);
}
__device__ __forceinline__ void inv3(const double* A, double* R) {
  double x0[3] = {A[0], A[1], A[2]};
  double y0[3], y1[3], y2[3];
  cross3(A + 3, A + 6, y0);
  double d = dot3(x0, y0);
  for (int k = 0; k < 3; k++) { x0[k] = x0[k] / d; y0[k] = y0[k] / d; }
  cross3(A + 6, x0, y1);
  cross3(x0, A + 3, y2);
  for (int c = 0; c < 3; c++) { R[3 * c] = y0[c]; R[1 + 3 * c] = y1[c]; R[2 + 3 * c] = y2[c]; }
}
__device__ __forceinline__ void matmul3(const double* A, const double* B, double* C) {
  for (int r = 0; r < 3; r++)
    for (int c = 0; c < 3; c++)
      C[r + 3 * c] = (A[r] * B[3 * c] + A[r + 3] * B[1 + 3 * c]) + A[r + 6] * B[2 + 3 * c];
}
__device__ __forceinline__ void matTmul3(const double* A, const double* B, double* C) {
  for (int r = 0; r < 3; r++)
    for (int c = 0; c < 3; c++)
      C[r + 3 * c] = (A[3 * r] * B[3 * c] + A[1 + 3 * r] * B[1 + 3 * c]) + A[2 + 3 * r] * B[2 + 3 * c];
}
__device__ __forceinline__ void matmulT3(const double* A, const double* B, double* C) {
  for (int r = 0; r < 3; r++)
    for (int c = 0; c < 3; c++)
      C[r + 3 * c] = (A[r] * B[c] + A[r + 3] * B[c + 3]) + A[r + 6] * B[c + 6];
}
__device__ __forceinline__ void matvec3(const double* A, const double* v, double* w) {
  for (int r = 0; r < 3; r++) w[r] = (A[r] * v[0] + A[r + 3] * v[1]) + A[r + 6] * v[2];
}

// ZEMWan stiffness (zem_stabilization.jl:32-42): C_1[i,j] = sum over k (outer), l (inner) of
// C[i,j,k,l] Kinv[k,l], all 81 products in that order, with C the Hooke tensor that
// get_hooke_matrix builds from the Voigt matrix (constitutive_models.jl:107-133): Voigt index
// of (i,j) in the order (1,1), (2,2), (3,3), (2,3), (1,3), (1,2); a = (1 - nu) lambda / nu on the
// diagonal of the normal block, lambda off it, mu on the diagonal of the shear block.
__device__ __forceinline__ int voigt_of(int i, int j) {
  if (i == j) return i;
  const int m = i + j;
  return m == 3 ? 3 : (m == 2 ? 4 : 5);
}
__device__ __forceinline__ double hooke_of(const DevParam& p, int i, int j, int k, int l) {
  const int I = voigt_of(i, j), J = voigt_of(k, l);
  if (I < 3 && J < 3) return I == J ? p.zwa : p.lambda;
  if (I >= 3 && J >= 3) return I == J ? p.mu : 0.0;
  return 0.0;
}
static __device__ void zem_wan64(const DevParam& p, const double* Kinv, double* C1) {
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) {
      double s = 0.0;
      for (int k = 0; k < 3; k++)
        for (int l = 0; l < 3; l++) s += hooke_of(p, i, j, k, l) * Kinv[k + 3 * l];
      C1[i + 3 * j] = s;
    }
}

// first_piola_kirchhoff (constitutive_models.jl:35-41, 169-176, 233-244)
static __device__ void pk1_64(int cmodel, const DevParam& p, const double* F, double* P) {
  double C[9], S[9];
  if (cmodel == CM_SVK) {
    double E[9];
    matTmul3(F, F, C);
    for (int k = 0; k < 9; k++) E[k] = 0.5 * (C[k] - ((k % 4) == 0 ? 1.0 : 0.0));
    double trE = (E[0] + E[4]) + E[8];
    double a = p.lambda * trE, m2 = 2 * p.mu;
    for (int k = 0; k < 9; k++) S[k] = (k % 4) == 0 ? m2 * E[k] + a : m2 * E[k];
  } else if (cmodel == CM_NEOHOOKE) {
    double J = det3(F), Ci[9];
    matTmul3(F, F, C);
    inv3(C, Ci);
    double lj = p.lambda * log(J);
    for (int k = 0; k < 9; k++) S[k] = p.mu * ((k % 4) == 0 ? -Ci[k] + 1.0 : -Ci[k]) + lj * Ci[k];
  } else {
    double J = det3(F);
    if (J < 2.220446049250313e-16 || isnan(J)) {
      for (int k = 0; k < 9; k++) P[k] = 0.0;
      return;
    }
    double Ci[9];
    matTmul3(F, F, C);
    inv3(C, Ci);
    double trC = (C[0] + C[4]) + C[8];
    double a = 1.0 / 3.0 * trC;
    double jp = pow(J, -2.0 / 3.0);
    double ij = 1.0 / J;
    double vol = p.K / 4 * (J * J - ij * ij);
    for (int k = 0; k < 9; k++)
      S[k] = p.G * ((k % 4) == 0 ? -(a * Ci[k]) + 1.0 : -(a * Ci[k])) * jp + vol * Ci[k];
  }
  matmul3(F, S, P);
}

// The phase-B state of a point for the kernels off the serial order: A = P K^-1 - S (F - I) and the
// stabilising stiffness S, in planes of n; zero for a killed point. ZEMSilling, S = beta I: five planes
// {A0 A1}, {A2 A3}, {A4 A5}, {A6 A7}, {A8 beta} (column-major A). ZEMWan, S = C1 = C : K^-1 (symmetric):
// {A8 Sxx}, {Syy Szz}, {Sxy Sxz}, {Syz 0} follow the first four.
__device__ __forceinline__ void c_state64(const DevBody& d, long long i, bool killed, double beta,
                                          const double* F, const double* PK, const double* C1) {
  if (d.zem == ZEM_WAN) {
    double A[16];
    for (int c = 0; c < 3; c++)
      for (int r = 0; r < 3; r++) {
        double s = 0.0;
        for (int k = 0; k < 3; k++) s += C1[r + 3 * k] * (k == c ? F[k + 3 * c] - 1.0 : F[k + 3 * c]);
        A[r + 3 * c] = PK[r + 3 * c] - s;
      }
    A[9] = C1[0];
    A[10] = C1[4];
    A[11] = C1[8];
    A[12] = 0.5 * (C1[1] + C1[3]);
    A[13] = 0.5 * (C1[2] + C1[6]);
    A[14] = 0.5 * (C1[5] + C1[7]);
    A[15] = 0.0;
    for (int k = 0; k < 8; k++)
      d.cst64[k * d.n + i] = killed ? make_double2(0.0, 0.0) : make_double2(A[2 * k], A[2 * k + 1]);
    return;
  }
  double A[10];
  for (int q = 0; q < 9; q++)
    A[q] = killed ? 0.0 : PK[q] - beta * ((q % 4) == 0 ? F[q] - 1.0 : F[q]);
  A[9] = killed ? 0.0 : beta;
  for (int k = 0; k < 5; k++) d.cst64[k * d.n + i] = make_double2(A[2 * k], A[2 * k + 1]);
}

// From the shape tensor K and the deformation sum Ft of a point: F, the kill decision
// (too_much_damage!, correspondence.jl:288-298; a halo row sees only part of its bonds, so its
// owner decides and the kill arrives with the halo exchange of the phase-A state), P K^-1 and
// the stabilising stiffness. Returns whether the point is killed.
__device__ __forceinline__ bool c_point64(const DevBody& d, const DevParam& P, long long i,
                                          unsigned meta, int cnt, int na, const double* K,
                                          const double* Ft) {
  const double damage = 1.0 - (double)na / (double)cnt;
  double Kinv[9], F[9], PKinv[9], C1[9];
  inv3(K, Kinv);
  matmul3(Ft, Kinv, F);
  bool hasnan = false;
  for (int q = 0; q < 9; q++) { d.F64[9 * i + q] = F[q]; hasnan |= isnan(F[q]); PKinv[q] = 0.0; }
  const bool killed = (meta & META_KILLED) || (!(meta & META_HALO) && (damage > d.maxdmg || hasnan));
  if (killed) {
    if (!(meta & META_KILLED)) d.meta[i] = meta | META_KILLED;
    na = 0;
  } else {
    double Pm[9];
    pk1_64(d.cmodel, P, F, Pm);
    matmul3(Pm, Kinv, PKinv);
    for (int q = 0; q < 9; q++) d.PK64[9 * i + q] = PKinv[q];
    if (d.zem == ZEM_WAN) {
      zem_wan64(P, Kinv, C1);
      for (int q = 0; q < 9; q++) d.C164[9 * i + q] = C1[q];
    }
  }
  c_state64(d, i, killed, P.beta, F, PKinv, C1);
  d.n_active[i] = na;
  return killed;
}

}  // namespace pd
