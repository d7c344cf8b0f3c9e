// pd_bond32.cuh -- the per-bond arithmetic of the packed FP32 kernels: the x and y components of
// every vector are one packed pair, z is scalar. Shared by the kernels that gather from global
// memory (pd_force32_pk.cu, pd_force32.cu) and from a tile in shared memory (pd_tile32.cu): a body's
// results do not depend on which of them runs.
#pragma once
#include "pd_common.cuh"
#include "pd_pack.cuh"

namespace pd {
namespace pack {

// Rows whose terms are summed from zero before they join the total of a point: a slice's rows may be
// shared among warps (pd_tile32.cu) without a change in the sums.
constexpr int SEG32 = 16;

// A segment's compensated sum joins the total's, in the form whose low part is below half a unit of
// the high one: rows of padding at its end (there are as many as the longest list of the slice
// asks for) leave that form as it is.
__device__ __forceinline__ void join(KSum1& t, const KSum1& s) {
  const float v = s.s + s.n;
  t.add(v);
  t.n += (s.s - v) + s.n;
}
__device__ __forceinline__ void join(KSum2& t, const KSum2& s) {
  const float2 v = add2(s.s, s.n);
  t.add(v);
  t.n = add2(t.n, add2(sub2(s.s, v), s.n));
}

// the own point's displacement, negated
struct Own32 {
  float2 nhi, nlo;
  float nhz, nlz;
  __device__ __forceinline__ Own32(const float4& hi, const float4& lo)
      : nhi(make_float2(-hi.x, -hi.y)), nlo(make_float2(-lo.x, -lo.y)), nhz(-hi.z), nlz(-lo.z) {}
};

// 1 / L of a bond
__device__ __forceinline__ float bond_rl(float w) { return __fdividef(1.f, fabsf(w)); }

// du = (h_j - h_i) + (l_j - l_i) and num = l^2 - L^2 = 2 xi . du + du . du: the two products apart,
// since the sum 2 xi + du would round xi's share of a small du
__device__ __forceinline__ void bond_du(const float4& g, const float4& hj, const float4& lj,
                                        const Own32& o, float2& dxy, float& dz, float& num) {
  dxy = add2(add2(xy(hj), o.nhi), add2(xy(lj), o.nlo));
  dz = (hj.z + o.nhz) + (lj.z + o.nlz);
  const float2 gd = mul2(xy(g), dxy), d2 = mul2(dxy, dxy);
  num = fmaf(2.f, fmaf(g.z, dz, gd.x + gd.y), fmaf(dz, dz, d2.x + d2.y));
}

// eta = xi + du, rl = 1 / |eta|, e = l - L = num / (l + L) without the cancellation of l - L
struct BondP {
  float2 exy;
  float ez;
  float rl, L, e;
};

__device__ __forceinline__ void bond_pk(const float4& g, const float4& hj, const float4& lj,
                                        const Own32& o, BondP& B) {
  float2 dxy;
  float dz, num;
  bond_du(g, hj, lj, o, dxy, dz, num);
  B.exy = add2(xy(g), dxy);
  B.ez = g.z + dz;
  const float2 e2 = mul2(B.exy, B.exy);
  const float l2 = fmaf(B.ez, B.ez, e2.x + e2.y);
  B.rl = rsqrtf(l2);
  B.L = fabsf(g.w);
  B.e = __fdividef(num, fmaf(l2, B.rl, B.L));
}

// The influence function of a point's bonds (kernels.jl:10-52). LIN: the linear one, delta / L. The
// B-spline in the products of t = 1 - xi: 2/3 - 4 xi^2 t up to xi = 1/2 and 4/3 t^3 beyond, without a
// division and without the cancellation of the expanded cubic near xi = 1 (jittered 488k-point OSB
// block: 727 us a step with the division and the expanded cubic, 594 so).
struct Influence {
  int kernel;
  float delta, rdelta;
  __device__ __forceinline__ Influence(const DevBody& d, const DevParam& P)
      : kernel(d.kernel), delta(P.deltaf), rdelta(P.inv_delta) {}
  template <bool LIN>
  __device__ __forceinline__ float at(float L, float rL) const {
    if constexpr (LIN) return delta * rL;
    const float xi = L * rdelta, t = 1.f - xi;
    const bool in = xi <= 0.5f;
    const float a = in ? xi : t, q = a * a * t;
    const float w = in ? fmaf(-4.f, q, 2.f / 3.f) : 4.f / 3.f * q;
    return kernel == KER_CONST_ONE ? 1.f : (xi > 0.f && xi <= 1.f ? w : 0.f);
  }
};

// the failure test of CriticalStretch
__device__ __forceinline__ bool stays(bool a, float eps, float epsc, float w) {
  return a && !(eps > epsc && w > 0.f);
}

// omega L V e of a bond, the dilatation's term; LIN: without the factor delta, which leaves the sum
template <bool LIN>
__device__ __forceinline__ float dil_term(const Influence& om, const BondP& B, float rL, float V) {
  if constexpr (LIN) return V * B.e;
  else return om.at<LIN>(B.L, rL) * V * B.L * B.e;
}

// What all bonds of a point share moves all of its forces the same way, and on a lattice those of all
// points: the weighted volume and c1 are therefore not left at their FP32 roundings, nor at those of xi,
// whose components on a lattice are all off alike (4.7e-8 at a spacing of 1e-3). Velocity error against 64 bits
// after 60 steps of 975-point coupons at horizons of 2.015, 3.015 and 4.015 spacings: 8.0e-7, 6.2e-7 and 1.3e-6
// with FP32 sums of omega V xi^2, 4.3e-7, 5.3e-7 and 4.7e-7 so.
//
// omega V L^2 in double, the weighted volume's term; LIN: without the factor delta
template <bool LIN>
__device__ __forceinline__ double vol_term(const Influence& om, float w, float V) {
  const float L = fabsf(w);
  if constexpr (LIN) return (double)V * (double)L;
  else return (double)(om.at<LIN>(L, 0.f) * V) * ((double)L * (double)L);
}

// a point's weighted volume from the sum of its terms; as stored, in two FP32 parts; and as stored less the
// terms of bonds that break
template <bool LIN>
__device__ __forceinline__ double vol_point(const DevParam& P, double sum) {
  return LIN ? P.delta * sum : sum;
}
__device__ __forceinline__ double vol_stored(const DevBody& d, long long i) {
  return (double)d.cm32[i].x + (double)d.mlo32[i];
}
template <bool LIN>
__device__ __forceinline__ double vol_less(const DevBody& d, const DevParam& P, long long i, float lost) {
  return vol_stored(d, i) - vol_point<LIN>(P, (double)lost);
}

// OSB: omega ((c2_i + c2_j) L + (c1_i + c1_j) e) V / l; LIN: without the factor delta
template <bool LIN>
__device__ __forceinline__ float osb_pair(const Influence& om, const BondP& B, float rL, float2 cs, float V) {
  const float f = LIN ? fmaf(cs.x, B.e * rL, cs.y)
                      : om.at<LIN>(B.L, rL) * fmaf(cs.y, B.L, cs.x * B.e);
  return f * (V * B.rl);
}

// v in FP32, up or down by a draw that the reference position decides: a value that many points share is
// rounded to either side in the proportion that keeps its mean. (To nearest, c1 of a lattice's inner points moved
// all of their forces by up to 6e-8. Any factor of a point's own on its force sum would keep two points' forces
// on each other from being opposite.) The draw: the position's bits through the mixing steps of splitmix64
__device__ __forceinline__ float round_drawn(double v, const double4& X) {
  const float lo = __double2float_rd(v), hi = __double2float_ru(v);
  unsigned long long h = 0x9E3779B97F4A7C15ull;
  const double x[3] = {X.x, X.y, X.z};
#pragma unroll
  for (int k = 0; k < 3; k++) {
    h ^= (unsigned long long)__double_as_longlong(x[k]);
    h = (h ^ (h >> 30)) * 0xBF58476D1CE4E5B9ull;
    h = (h ^ (h >> 27)) * 0x94D049BB133111EBull;
    h ^= h >> 31;
  }
  const double u = (double)(unsigned)(h >> 32) * 0x1p-32;
  return v - (double)lo > u * ((double)hi - (double)lo) ? hi : lo;
}

// OSB: {c1, c2} of a point from its weighted volume m and the sum t of the dilatation's terms, with m and
// the dilatation stored
template <bool LIN>
__device__ __forceinline__ void osb_point(const DevBody& d, const DevParam& P, long long i, double m, double t) {
  float c1 = 0.f, c2 = 0.f, th = 0.f;
  if (m != 0.0) {
    const double rm = 1.0 / m, dil = 3.0 * rm * (LIN ? P.delta * t : t);
    c1 = round_drawn(15.0 * P.G * rm, d.X0[i]);
    c2 = (float)(dil * (3.0 * P.K - 5.0 * P.G) * rm);
    th = (float)dil;
  }
  const float w = (float)m;
  d.cc32[i] = make_float2(c1, c2);
  d.cm32[i] = make_float2(w, th);
  d.mlo32[i] = (float)(m - (double)w);
}

// the force on a point: its sum times the factor f that all bonds share (in double, as above). A point
// without a bond has none, wherever it is: at infinity its own bond vectors (0 times them is added) are
// undefined
__device__ __forceinline__ void store_force(const DevBody& d, long long i, int kstep, double f,
                                            const KSum2& xy, const KSum1& zs) {
  float x = (float)(f * ((double)xy.s.x + (double)xy.n.x)), y = (float)(f * ((double)xy.s.y + (double)xy.n.y)),
        z = (float)(f * ((double)zs.s + (double)zs.n));
  if (isnan(x) || isnan(y) || isnan(z)) {
    bool bonded = false;
    const int cnt = (int)(d.off[i + 1] - d.off[i]);
    for (int k = 0; k < cnt && !bonded; k++) bonded = bond_bit_live(d.bits, bond_slot(d, i, k));
    if (bonded) {
      const long long step = d.ctrl->base + kstep;
      if (atomicExch(&d.ctrl->err, 1) == 0) d.ctrl->err_step = step;
      else atomicMin(&d.ctrl->err_step, step);
    } else {
      x = y = z = 0.f;
    }
  }
  d.b32[3 * i] = x;
  d.b32[3 * i + 1] = y;
  d.b32[3 * i + 2] = z;
}

// correspondence phase A: the constants of a point
struct CorrA {
  float epsc, thr, ks;
  Influence om;
  // ks: a bond's weight in the sums with xi and du over the horizon, omega V / delta^5; with the
  // linear influence function delta / L, V / (L delta^4). thr: l^2 - L^2 below this share of L^2 is
  // a stretch below eps_c whatever the rounding
  __device__ __forceinline__ CorrA(const DevBody& d, const DevParam& P) : epsc(P.epscf), om(d, P) {
    const float w = P.vscale * P.inv_delta * P.inv_delta;
    ks = d.kernel == KER_LINEAR ? P.deltaf * w : w;
    thr = epsc > 0.f ? (2.f * epsc + epsc * epsc) * (1.f - 1e-5f) : -INFINITY;
  }
};

// whether an active bond stays: the test on eps = (l - L) / L only for those beyond thr
__device__ __forceinline__ bool corr_stays(bool a, const CorrA& c, const float4& g, float rL,
                                           const float2 dxy, float dz, float num) {
  if (!a || !(g.w > 0.f) || num < c.thr * (g.w * g.w)) return a;
  const float2 e = add2(xy(g), dxy);
  const float ez = g.z + dz;
  const float2 e2 = mul2(e, e);
  const float l2 = fmaf(ez, ez, e2.x + e2.y);
  return !(__fdividef(num, fmaf(l2, rsqrtf(l2), g.w)) * rL > c.epsc);
}

template <bool LIN>
__device__ __forceinline__ float corr_weight(const CorrA& c, const float4& g, float rL, float V) {
  return (LIN ? rL : c.om.at<LIN>(fabsf(g.w), rL)) * V * c.ks;
}

// The sums of correspondence phase A: the displacement gradient (rows x, y of every column packed) and, in
// full, the shape tensor {xx, yy, zz, xy, xz, yz} (compensated). COMP: compensated sums of the gradient, else
// plain FP32 ones, which bond-stream variant 5 asks for (their error in the displacement after 250 steps is
// less than the rest of the form's)
template <bool FULLK, bool COMP>
struct CorrSums {
  static constexpr bool FULL = FULLK;
  float2 Hxy[3], nxy[3];  // COMP: the sums and their negated compensations
  float Hz[3], nz[3];
  KSum2 K01, K23, K45;
  float dK[6];
  __device__ __forceinline__ CorrSums() {
#pragma unroll
    for (int c = 0; c < 3; c++) { Hxy[c] = nxy[c] = both(0.f); Hz[c] = nz[c] = 0.f; }
#pragma unroll
    for (int q = 0; q < 6; q++) dK[q] = 0.f;
  }
  // column c gains f times du
  __device__ __forceinline__ void column(int c, float f, const float2 dxy, float dz) {
    if constexpr (COMP) {
      const float2 y = fma2(both(f), dxy, nxy[c]), t = add2(Hxy[c], y);
      nxy[c] = add2(sub2(Hxy[c], t), y);
      Hxy[c] = t;
      const float yz = fmaf(f, dz, nz[c]), tz = Hz[c] + yz;
      nz[c] = (Hz[c] - tz) + yz;
      Hz[c] = tz;
    } else {
      Hxy[c] = fma2(both(f), dxy, Hxy[c]);
      Hz[c] = fmaf(f, dz, Hz[c]);
    }
  }
  __device__ __forceinline__ void add(float t, const float4& g, const float2 dxy, float dz) {
    const float2 tX = mul2(both(t), xy(g));
    const float tXz = t * g.z;
    column(0, tX.x, dxy, dz);
    column(1, tX.y, dxy, dz);
    column(2, tXz, dxy, dz);
    if constexpr (FULLK) {
      K01.add(mul2(tX, xy(g)));
      K23.add(make_float2(tXz * g.z, tX.x * g.y));
      K45.add(mul2(tX, both(g.z)));
    }
  }
  // a bond breaks: its term leaves the stored shape tensor
  __device__ __forceinline__ void drop(float t, const float4& g) {
    dK[0] += t * g.x * g.x; dK[1] += t * g.y * g.y; dK[2] += t * g.z * g.z;
    dK[3] += t * g.x * g.y; dK[4] += t * g.x * g.z; dK[5] += t * g.y * g.z;
  }
};

// correspondence phase B: V omega ((A_i + A_j) xi + (beta_i + beta_j) du), A column-major in
// {a.x .. a.w, b.x .. b.w, c.x}, beta in c.y; LIN: without the factor delta
__device__ __forceinline__ void corr_pair(const float4& g, const float2 dxy, float dz, const float4& ia,
                                          const float4& ib, const float2& ic, const float4& ja,
                                          const float4& jb, const float2& jc, float2& txy, float& tz) {
  const float2 S01 = add2(make_float2(ia.x, ia.y), make_float2(ja.x, ja.y));
  const float2 S23 = add2(make_float2(ia.z, ia.w), make_float2(ja.z, ja.w));
  const float2 S45 = add2(make_float2(ib.x, ib.y), make_float2(jb.x, jb.y));
  const float2 S67 = add2(make_float2(ib.z, ib.w), make_float2(jb.z, jb.w));
  const float2 S8b = add2(ic, jc);
  txy = mul2(both(S8b.y), dxy);
  txy = fma2(S01, both(g.x), txy);
  txy = fma2(make_float2(S23.y, S45.x), both(g.y), txy);
  txy = fma2(S67, both(g.z), txy);
  tz = fmaf(S23.x, g.x, fmaf(S45.y, g.y, fmaf(S8b.x, g.z, S8b.y * dz)));
}

}  // namespace pack
}  // namespace pd
