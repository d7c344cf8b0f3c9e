// pd_force64_fast.cu -- FP64 force kernels off the serial order that gather from global memory:
// correspondence, lane groups, several parameter sets, EnergySurfaceCorrection, OSB phase B of bodies small
// enough to split their slices, and BB and OSB bodies without tiles. Others run pd_tile64.cu, with the same
// arithmetic and order of the sums: the same bits.
//
// What bounds them: per bond 12 bytes of stream (neighbour index and reference length), 32 to
// 144 bytes gathered through L1 from the neighbour's point records, and the FP64 pipe (two warp
// instructions a cycle and SM). The kernels they replace spent their time elsewhere: on the
// latency of one dependent chain per bond (an IEEE square root and two or three IEEE divisions,
// each with its slow path) and, below about 100,000 points, on a chip of which one thread per
// point fills only a part.
//
//   - One reciprocal square root per bond. g = 1 / sqrt(l^2 L^2) gives 1 / (l L) directly and
//     l = l^2 L g after one correction (the residual l^2 - l*l, exact in an fma, times 1 / 2 l;
//     pd_bond64.cuh). l^2 is formed as the reference forms it, so a body at rest is free of force exactly.
//   - The failure decision is the reference's eps = (l - L) / L > eps_c. A product decides where
//     l - L is below eps_c L by more than the rounding of either side; only the bonds beyond
//     take the division.
//   - A slice of 32 / G points is walked by W warps (G = 1: W of 1, 2, 4, 8). The rows of a slice
//     are cut into segments of SEG rows; a segment is summed from zero by one warp and the
//     segment sums are added in row order, whatever W is: results depend neither on W nor, for
//     a partition, on how many points the body has.
//   - Two rows of neighbour gathers are in flight per lane, and the stream of the next row pair
//     is loaded before the arithmetic of the current one.
//   - Correspondence in the form w (A xi + beta du) with A = P K^-1 - beta H, H = F - I, du the
//     displacement difference: the bond term of the reference, w (P K^-1 xi + beta (eta - F xi)),
//     with eta - F xi = du - H xi. A and beta are kept in five planes of double2 (structure of
//     arrays), so that the 32 lanes of a warp read consecutive 16-byte words.
//
// Time a step, lattices at a horizon of 3.015 spacings, before and after (one lane per point, without tiles, us,
// CUDA graphs): 3,200 points BB 55.6 -> 10.9, OSB 129 -> 17.5, CMat 237 -> 24; 27,347 points BB 70
// -> 23, OSB 163 -> 42, CMat 301 -> 77; 125,000 points BB 153 -> 101, OSB 401 -> 190, CMat 920 ->
// 281; 397,243 points BB 376 -> 268, OSB 1049 -> 498.
#include "pd_bond64.cuh"
#include "pd_common.cuh"
#include "pd_launch.h"
#include "pd_math64.cuh"

namespace pd {

namespace {

// Resident blocks of 256 threads per SM and rows in flight per lane, measured on lattices (us a
// launch, 397,243 points; CMat 125,000): BB 3 blocks and 2 rows 259 (4 and 1: 252, but 29 against
// 25 at 27,347 points; 2 and 2: 333; 5 and 1: 350); OSB phase A 3 and 2: 242 (4 and 1: 246, 2 and
// 2: 326), phase B 3 and 2: 252 (2 and 2: 308, 4 and 1: 298); CMat phase A 2 and 2: 150 (2 and 1:
// 189, 3 and 1: 179), phase B 2 blocks with two rows of stream, gathered one after the other: 133
// (one row of stream 158, 3 blocks 240).
constexpr int MB_BB = 3, MB_OA = 3, MB_OB = 3, MB_CA = 2, MB_CB = 2;
constexpr int RU_BB = 2, RU_OA = 2, RU_OB = 2, RU_CA = 2, RU_CB = 2;
constexpr int SEG = SEG64;

// a point record {x, y, z, V} in one 256-bit load: the 32 lanes of a warp read 32 neighbouring
// records, and two 128-bit loads would each touch every one of their sectors
__device__ __forceinline__ double4 ld_point(const double4* p) {
  double4 v;
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
      : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
  return v;
}

// An error of an earlier kernel ends the run. With several warps per slice the decision is the
// block's: another block may record its error while this one starts.
template <int W>
__device__ __forceinline__ bool stopped(const DevBody& d) {
  const int err = *(volatile const int*)&d.ctrl->err;
  return W > 1 ? __syncthreads_or(err) != 0 : err != 0;
}

// the lane's place: slice s, walked by W warps of which this is number `part`
template <int G, int W>
struct Place {
  long long s, i;
  int lane, gl, part, self, rows;
  bool valid;
  const int* nbr;
  const double* len;
  unsigned* bits;
  const double* sc;
  __device__ __forceinline__ Place(const DevBody& d, bool esc) {
    lane = threadIdx.x & 31;
    const int wb = threadIdx.x >> 5;
    const long long w = (long long)blockIdx.x * (blockDim.x >> 5) + wb;
    s = w / W;
    part = (int)(w % W);
    gl = lane % G;
    const bool live = s < d.nslices;
    const long long q = s * (32 / G) + lane / G;
    valid = live && q < d.n;
    i = valid ? point_at(d, q) : q;
    self = valid ? (int)i : 0;
    const long long sbase = live ? d.soff[s] : 0;
    rows = live ? (int)((d.soff[s + 1] - sbase) >> 5) : 0;
    nbr = d.nbr + sbase + lane;
    len = d.len64 + sbase + lane;
    bits = d.bits + (sbase >> 5);
    sc = esc ? d.sc64 + sbase + lane : nullptr;
  }
};

// the stream of rows r .. r + RU - 1 (past the last row: row r again, with no state bit set; with
// one lane per point the rows of a slice are a multiple of four)
template <int G, int RU, bool ESC, bool OWNED>
struct Rows {
  int j[RU];
  double L[RU], sc[ESC ? RU : 1];
  unsigned w[RU];
  // OWNED: the warp rewrites its state words, which are therefore loaded plainly
  template <class P>
  __device__ __forceinline__ void load(const P& p, int r) {
#pragma unroll
    for (int u = 0; u < RU; u++) {
      const bool in = (G == 1 && RU <= 2) || u == 0 || r + u < p.rows;
      const int q = in ? r + u : r;
      w[u] = OWNED ? p.bits[q] : __ldg(p.bits + q);
      if (!in) w[u] = 0u;
      j[u] = __ldcs(p.nbr + 32 * q);
      L[u] = __ldcs(p.len + 32 * q);
      if (ESC) sc[u] = __ldcs(p.sc + 32 * q);
    }
  }
};

// Adds the segment sums of a round (W segments) to the totals, in row order; after the last
// round the lanes of part 0 hold them. The barrier is the slice's own: its W warps walk the same
// rows. IN_SH: the totals live in shared memory while the segments are summed, for the kernel
// whose sums would otherwise take their registers twice.
template <int W, int NV, bool IN_SH>
struct Totals {
  double t[NV];
  int na;
  __device__ __forceinline__ double* slot(int lane) {
    __shared__ double st[IN_SH ? 8 / W : 1][IN_SH ? NV : 1][32];
    return &st[IN_SH ? (threadIdx.x >> 5) / W : 0][0][lane];
  }
  __device__ __forceinline__ Totals(int part, int lane) : na(0) {
#pragma unroll
    for (int v = 0; v < NV; v++) t[v] = 0.0;
    if constexpr (IN_SH) {
      if (part == 0) {
        double* q = slot(lane);
#pragma unroll
        for (int v = 0; v < NV; v++) q[32 * v] = 0.0;
      }
    }
  }
  __device__ __forceinline__ void add(const double (&seg)[NV], int nseg, int part, int lane, int r0,
                                      int rows) {
    if constexpr (W == 1) {
      double* q = slot(lane);
#pragma unroll
      for (int v = 0; v < NV; v++) {
        if constexpr (IN_SH) q[32 * v] += seg[v];
        else t[v] += seg[v];
      }
      na += nseg;
    } else {
      __shared__ double sh[8][NV][32];
      __shared__ int shn[8][32];
      const int wb = threadIdx.x >> 5;
#pragma unroll
      for (int v = 0; v < NV; v++) sh[wb][v][lane] = seg[v];
      shn[wb][lane] = nseg;
      const int bar = 1 + wb / W;
      asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(32 * W) : "memory");
      if (part == 0) {
        double* q = slot(lane);
#pragma unroll
        for (int w = 0; w < W; w++)
          if (r0 + w * SEG < rows) {
#pragma unroll
            for (int v = 0; v < NV; v++) {
              if constexpr (IN_SH) q[32 * v] += sh[wb + w][v][lane];
              else t[v] += sh[wb + w][v][lane];
            }
            na += shn[wb + w][lane];
          }
      }
      if (r0 + W * SEG < rows) asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(32 * W) : "memory");
    }
  }
  // the lane group's sums (part 0)
  template <int G>
  __device__ __forceinline__ void finish(int lane) {
    if constexpr (IN_SH) {
      const double* q = slot(lane);
#pragma unroll
      for (int v = 0; v < NV; v++) t[v] = q[32 * v];
    }
    if constexpr (G > 1) {
#pragma unroll
      for (int v = 0; v < NV; v++) t[v] = group_sum<G>(t[v]);
      na = group_sum<G>(na);
    }
  }
};

// the rows after r of this warp's segments, or a row past the last one
template <int W, int RU>
__device__ __forceinline__ int next_rows(int r, int ra, int rb) {
  return r + RU < rb ? r + RU : ra + W * SEG;
}

}  // namespace

// -------------------------------------------------------------------------------------------
// BB (bond_based.jl:125-180): one sweep, failure then the pairwise force
// bc eps V_j eta / l = bc V_j (l - L) g eta, g = 1 / (l L)
// -------------------------------------------------------------------------------------------
template <int G, int W, bool MULTI, bool ESC>
__global__ void __launch_bounds__(256, MB_BB) k_bb64f(DevBody d, int kstep) {
  if (stopped<W>(d)) return;
  constexpr int RU = RU_BB;
  const Place<G, W> p(d, ESC);
  const double4 xi = ld4_64(d.cur + p.self);
  const DevParam& P = d.params[p.valid ? d.meta[p.self] & META_PID_MASK : 0];
  const double epsc = P.epsc, thr = fail_threshold(epsc), bci = P.bc;
  Totals<W, 3, false> T(p.part, p.lane);
  Rows<G, RU, ESC, true> nx;
  if (p.part * SEG < p.rows) nx.load(p, p.part * SEG);
  for (int r0 = 0; r0 < p.rows; r0 += W * SEG) {
    double seg[3] = {0.0, 0.0, 0.0};
    int nseg = 0;
    const int ra = r0 + p.part * SEG, rb = min(ra + SEG, p.rows);
    for (int r = ra; r < rb; r += RU) {
      const Rows<G, RU, ESC, true> c = nx;
      bool a[RU];
      int j[RU];
#pragma unroll
      for (int u = 0; u < RU; u++) {
        a[u] = (c.w[u] >> p.lane) & 1u;
        j[u] = a[u] ? c.j[u] : p.self;
      }
      double4 x[RU];
#pragma unroll
      for (int u = 0; u < RU; u++) x[u] = ld_point(d.cur + j[u]);
      const int nr = next_rows<W, RU>(r, ra, rb);
      if (nr < p.rows) nx.load(p, nr);
      bool act[RU];
#pragma unroll
      for (int u = 0; u < RU; u++) {
        const double dx = x[u].x - xi.x, dy = x[u].y - xi.y, dz = x[u].z - xi.z;
        const Bond64 b(dx, dy, dz, c.L[u]);
        act[u] = a[u] && !fails64(b.l2, b.e, c.L[u], b.L, thr, epsc);
        double bc = bci;
        if (MULTI) bc = 0.5 * (bci + d.params[d.meta[j[u]] & META_PID_MASK].bc);
        if (ESC) bc *= c.sc[u];
        const double sc = act[u] ? (bc * x[u].w) * (b.e * b.g) : 0.0;
        seg[0] = fma(sc, dx, seg[0]);
        seg[1] = fma(sc, dy, seg[1]);
        seg[2] = fma(sc, dz, seg[2]);
      }
#pragma unroll
      for (int u = 0; u < RU; u++) {
        nseg += (int)act[u];
        const unsigned now = __ballot_sync(0xffffffffu, act[u]);
        if (p.lane == 0 && now != c.w[u]) p.bits[r + u] = now;
      }
    }
    T.add(seg, nseg, p.part, p.lane, r0, p.rows);
  }
  if (W > 1 && p.part != 0) return;
  T.template finish<G>(p.lane);
  if (p.valid && p.gl == 0) {
    d.b64[3 * p.i] = T.t[0];
    d.b64[3 * p.i + 1] = T.t[1];
    d.b64[3 * p.i + 2] = T.t[2];
    d.n_active[p.i] = T.na;
    nan_flag(d, kstep, T.t[0], T.t[1], T.t[2]);
  }
}

// -------------------------------------------------------------------------------------------
// OSB phase A (ordinary_state_based.jl:107-126, 176-204): failure, weighted volume, dilatation,
// c1 and c2 (:135-136). LIN, the linear influence function omega = delta / L: omega V L^2 =
// delta V L and omega V L e = delta V e need no reciprocal.
// -------------------------------------------------------------------------------------------
template <int G, int W, bool LIN, bool ESC>
__global__ void __launch_bounds__(256, MB_OA) k_osb_a64f(DevBody d, int kstep) {
  if (stopped<W>(d)) return;
  constexpr int RU = RU_OA;
  const Place<G, W> p(d, ESC);
  const double4 xi = ld4_64(d.cur + p.self);
  const DevParam& P = d.params[p.valid ? d.meta[p.self] & META_PID_MASK : 0];
  const double epsc = P.epsc, thr = fail_threshold(epsc), delta = P.delta, rdelta = 1.0 / delta;
  Totals<W, 2, false> T(p.part, p.lane);
  Rows<G, RU, ESC, true> nx;
  if (p.part * SEG < p.rows) nx.load(p, p.part * SEG);
  for (int r0 = 0; r0 < p.rows; r0 += W * SEG) {
    double seg[2] = {0.0, 0.0};
    int nseg = 0;
    const int ra = r0 + p.part * SEG, rb = min(ra + SEG, p.rows);
    for (int r = ra; r < rb; r += RU) {
      const Rows<G, RU, ESC, true> c = nx;
      bool a[RU];
      int j[RU];
#pragma unroll
      for (int u = 0; u < RU; u++) {
        a[u] = (c.w[u] >> p.lane) & 1u;
        j[u] = a[u] ? c.j[u] : p.self;
      }
      double4 x[RU];
#pragma unroll
      for (int u = 0; u < RU; u++) x[u] = ld_point(d.cur + j[u]);
      const int nr = next_rows<W, RU>(r, ra, rb);
      if (nr < p.rows) nx.load(p, nr);
      bool act[RU];
#pragma unroll
      for (int u = 0; u < RU; u++) {
        const double L = fabs(c.L[u]);
        const double dx = x[u].x - xi.x, dy = x[u].y - xi.y, dz = x[u].z - xi.z;
        const double l2 = (dx * dx + dy * dy) + dz * dz;
        const double e = sqrt_of(l2, rsqrt3(l2)) - L;
        act[u] = a[u] && !fails64(l2, e, c.L[u], L, thr, epsc);
        double t = ESC ? c.sc[u] * x[u].w : x[u].w;
        if (!LIN) t *= omega64(d.kernel, delta, rdelta, L) * L;
        seg[0] = fma(act[u] ? t : 0.0, L, seg[0]);
        seg[1] += act[u] ? t * e : 0.0;
      }
#pragma unroll
      for (int u = 0; u < RU; u++) {
        nseg += (int)act[u];
        const unsigned now = __ballot_sync(0xffffffffu, act[u]);
        if (p.lane == 0 && now != c.w[u]) p.bits[r + u] = now;
      }
    }
    T.add(seg, nseg, p.part, p.lane, r0, p.rows);
  }
  if (W > 1 && p.part != 0) return;
  T.template finish<G>(p.lane);
  if (p.valid && p.gl == 0) {
    const double wvol = LIN ? delta * T.t[0] : T.t[0], sdil = LIN ? delta * T.t[1] : T.t[1];
    double c1 = 0.0, c2 = 0.0, dil = 0.0;
    if (wvol != 0.0) {
      dil = 3.0 / wvol * sdil;
      c1 = 15.0 * P.G / wvol;
      c2 = dil * (3.0 * P.K / wvol - c1 / 3.0);
    }
    d.coef64[p.i] = make_double4(c1, c2, wvol, dil);
    d.n_active[p.i] = T.na;
  }
}

// -------------------------------------------------------------------------------------------
// OSB phase B (ordinary_state_based.jl:128-174) for symmetric bond states and one parameter set,
// in gather form: b_i = sum_j omega ((c2_i + c2_j) L + (c1_i + c1_j) (l - L)) V_j eta / l. A point
// without weighted volume holds c1 = c2 = 0 and adds nothing, as where the reference returns.
// -------------------------------------------------------------------------------------------
template <int G, int W, bool LIN, bool ESC>
__global__ void __launch_bounds__(256, MB_OB) k_osb_b64f(DevBody d, int kstep) {
  if (stopped<W>(d)) return;
  constexpr int RU = RU_OB;
  const Place<G, W> p(d, ESC);
  const double4 xi = ld4_64(d.cur + p.self);
  const double2 ci = *reinterpret_cast<const double2*>(d.coef64 + p.self);
  const double delta = d.params[p.valid ? d.meta[p.self] & META_PID_MASK : 0].delta, rdelta = 1.0 / delta;
  Totals<W, 3, false> T(p.part, p.lane);
  Rows<G, RU, ESC, false> nx;
  if (p.part * SEG < p.rows) nx.load(p, p.part * SEG);
  for (int r0 = 0; r0 < p.rows; r0 += W * SEG) {
    double seg[3] = {0.0, 0.0, 0.0};
    const int ra = r0 + p.part * SEG, rb = min(ra + SEG, p.rows);
    for (int r = ra; r < rb; r += RU) {
      const Rows<G, RU, ESC, false> c = nx;
      bool a[RU];
      int j[RU];
#pragma unroll
      for (int u = 0; u < RU; u++) {
        a[u] = (c.w[u] >> p.lane) & 1u;
        j[u] = a[u] ? c.j[u] : p.self;
      }
      double4 x[RU];
#pragma unroll
      for (int u = 0; u < RU; u++) x[u] = ld_point(d.cur + j[u]);
      double2 cj[RU];
#pragma unroll
      for (int u = 0; u < RU; u++) cj[u] = __ldg(reinterpret_cast<const double2*>(d.coef64 + j[u]));
      const int nr = next_rows<W, RU>(r, ra, rb);
      if (nr < p.rows) nx.load(p, nr);
#pragma unroll
      for (int u = 0; u < RU; u++) {
        const double dx = x[u].x - xi.x, dy = x[u].y - xi.y, dz = x[u].z - xi.z;
        const Bond64 b(dx, dy, dz, c.L[u]);
        const double t = fma(ci.y + cj[u].y, b.L, (ci.x + cj[u].x) * b.e);
        // omega / l = delta g (linear), omega L g otherwise
        double om = LIN ? delta : omega64(d.kernel, delta, rdelta, b.L) * b.L;
        if (ESC) om *= c.sc[u];
        const double sc = a[u] ? (om * x[u].w) * (t * b.g) : 0.0;
        seg[0] = fma(sc, dx, seg[0]);
        seg[1] = fma(sc, dy, seg[1]);
        seg[2] = fma(sc, dz, seg[2]);
      }
    }
    T.add(seg, 0, p.part, p.lane, r0, p.rows);
  }
  if (W > 1 && p.part != 0) return;
  T.template finish<G>(p.lane);
  if (p.valid && p.gl == 0) {
    d.b64[3 * p.i] = T.t[0];
    d.b64[3 * p.i + 1] = T.t[1];
    d.b64[3 * p.i + 2] = T.t[2];
    nan_flag(d, kstep, T.t[0], T.t[1], T.t[2]);
  }
}

// -------------------------------------------------------------------------------------------
// CMat phase A (correspondence.jl:193-224, 288-298; bond_system.jl:309-327): failure, the shape
// tensor (six sums) and the deformation sums (nine), then per point F, P K^-1 and the phase-B
// state. The failure decision needs no square root where l^2 is clearly below (L (1 + eps_c))^2.
// -------------------------------------------------------------------------------------------
template <int G, int W, bool LIN>
__global__ void __launch_bounds__(256, MB_CA) k_c_a64f(DevBody d, int kstep) {
  if (stopped<W>(d)) return;
  constexpr int RU = RU_CA;
  const Place<G, W> p(d, false);
  const double4 xi = ld4_64(d.cur + p.self), Xi = ld4_64(d.X0 + p.self);
  const unsigned meta = p.valid ? d.meta[p.self] : 0u;
  const DevParam& P = d.params[meta & META_PID_MASK];
  const double epsc = P.epsc, delta = P.delta, rdelta = 1.0 / delta;
  const double f1 = 1.0 + epsc;
  const double sure = epsc > -0.5 ? f1 * f1 * (1.0 - 2e-14) : 0.0;
  Totals<W, 15, true> T(p.part, p.lane);
  Rows<G, RU, false, true> nx;
  if (p.part * SEG < p.rows) nx.load(p, p.part * SEG);
  for (int r0 = 0; r0 < p.rows; r0 += W * SEG) {
    double seg[15];
#pragma unroll
    for (int v = 0; v < 15; v++) seg[v] = 0.0;
    int nseg = 0;
    const int ra = r0 + p.part * SEG, rb = min(ra + SEG, p.rows);
    for (int r = ra; r < rb; r += RU) {
      const Rows<G, RU, false, true> c = nx;
      bool a[RU];
      int j[RU];
#pragma unroll
      for (int u = 0; u < RU; u++) {
        a[u] = (c.w[u] >> p.lane) & 1u;
        j[u] = a[u] ? c.j[u] : p.self;
      }
      double4 x[RU];
#pragma unroll
      for (int u = 0; u < RU; u++) x[u] = ld_point(d.cur + j[u]);
      double4 X[RU];
#pragma unroll
      for (int u = 0; u < RU; u++) X[u] = ld_point(d.X0 + j[u]);
      const int nr = next_rows<W, RU>(r, ra, rb);
      if (nr < p.rows) nx.load(p, nr);
      bool act[RU];
#pragma unroll
      for (int u = 0; u < RU; u++) {
        const double L = fabs(c.L[u]);
        const double dx = x[u].x - xi.x, dy = x[u].y - xi.y, dz = x[u].z - xi.z;
        const double DX = X[u].x - Xi.x, DY = X[u].y - Xi.y, DZ = X[u].z - Xi.z;
        const double l2 = (dx * dx + dy * dy) + dz * dz;
        act[u] = a[u];
        if (a[u] && c.L[u] > 0 && !(l2 < sure * (L * L))) act[u] = !((sqrt(l2) - L) / L > epsc);
        const double om = LIN ? delta * rcp3(L) : omega64(d.kernel, delta, rdelta, L);
        const double t = act[u] ? om * x[u].w : 0.0;
        const double tx = t * DX, ty = t * DY, tz = t * DZ;
        seg[0] = fma(tx, DX, seg[0]); seg[1] = fma(ty, DY, seg[1]); seg[2] = fma(tz, DZ, seg[2]);
        seg[3] = fma(tx, DY, seg[3]); seg[4] = fma(tx, DZ, seg[4]); seg[5] = fma(ty, DZ, seg[5]);
        // column c of the deformation sum: eta times t DX_c
        seg[6] = fma(tx, dx, seg[6]);   seg[7] = fma(tx, dy, seg[7]);   seg[8] = fma(tx, dz, seg[8]);
        seg[9] = fma(ty, dx, seg[9]);   seg[10] = fma(ty, dy, seg[10]); seg[11] = fma(ty, dz, seg[11]);
        seg[12] = fma(tz, dx, seg[12]); seg[13] = fma(tz, dy, seg[13]); seg[14] = fma(tz, dz, seg[14]);
      }
#pragma unroll
      for (int u = 0; u < RU; u++) {
        nseg += (int)act[u];
        const unsigned now = __ballot_sync(0xffffffffu, act[u]);
        if (p.lane == 0 && now != c.w[u]) p.bits[r + u] = now;
      }
    }
    T.add(seg, nseg, p.part, p.lane, r0, p.rows);
  }
  if (W > 1 && p.part != 0) return;
  T.template finish<G>(p.lane);
  bool killed = false;
  if (p.valid && p.gl == 0) {
    const int cnt = (int)(d.off[p.i + 1] - d.off[p.i]);
    const double K[9] = {T.t[0], T.t[3], T.t[4], T.t[3], T.t[1], T.t[5], T.t[4], T.t[5], T.t[2]};
    killed = c_point64(d, P, p.i, meta, cnt, T.na, K, T.t + 6);
  }
  if (!d.sym) {
    // directed bond states: a killed point loses all its bonds (correspondence.jl:293)
    if (G > 1) killed = group_bcast<G>(killed);
    const unsigned kill_mask = __ballot_sync(0xffffffffu, p.valid && killed);
    if (kill_mask && p.lane == 0)
      for (int r = 0; r < p.rows; r++) p.bits[r] &= ~kill_mask;
  }
}

// -------------------------------------------------------------------------------------------
// CMat phase B (correspondence.jl:226-251) for symmetric bond states and one parameter set: b_i =
// sum_j omega V_j ((A_i + A_j) xi + (S_i + S_j) du), S = beta I for ZEMSilling. A killed point holds
// A = 0 and S = 0. ZEMWan's 15 values a point take 128 bytes of gathers a bond beside the 64 of the
// positions (one block an SM, no spills): 73,062 points 588 -> 289 us a step against the kernel that reads
// F, P K^-1 and C1 of both points, 2,233 points 294 -> 46.
// -------------------------------------------------------------------------------------------
template <int G, int W, bool LIN, bool WAN>
__global__ void __launch_bounds__(256, WAN ? 1 : MB_CB) k_c_b64f(DevBody d, int kstep) {
  if (stopped<W>(d)) return;
  constexpr int RU = RU_CB;
  const Place<G, W> p(d, false);
  const double4 xi = ld4_64(d.cur + p.self), Xi = ld4_64(d.X0 + p.self);
  const double delta = d.params[p.valid ? d.meta[p.self] & META_PID_MASK : 0].delta, rdelta = 1.0 / delta;
  const long long n = d.n;
  constexpr int NP = WAN ? 8 : 5;
  double2 Ai[NP];
#pragma unroll
  for (int k = 0; k < NP; k++) Ai[k] = d.cst64[k * n + p.self];
  Totals<W, 3, false> T(p.part, p.lane);
  Rows<G, RU, false, false> nx;
  if (p.part * SEG < p.rows) nx.load(p, p.part * SEG);
  for (int r0 = 0; r0 < p.rows; r0 += W * SEG) {
    double seg[3] = {0.0, 0.0, 0.0};
    const int ra = r0 + p.part * SEG, rb = min(ra + SEG, p.rows);
    for (int r = ra; r < rb; r += RU) {
      const Rows<G, RU, false, false> c = nx;
      const int nr = next_rows<W, RU>(r, ra, rb);
#pragma unroll
      for (int u = 0; u < RU; u++) {
        const bool a = (c.w[u] >> p.lane) & 1u;
        const int j = a ? c.j[u] : p.self;
        const double4 x = ld_point(d.cur + j), X = ld_point(d.X0 + j);
        double2 Aj[NP];
#pragma unroll
        for (int k = 0; k < NP; k++) Aj[k] = __ldg(d.cst64 + k * n + j);
        if (u == 0 && nr < p.rows) nx.load(p, nr);
        const double L = fabs(c.L[u]);
        const double DX = X.x - Xi.x, DY = X.y - Xi.y, DZ = X.z - Xi.z;
        const double ux = (x.x - xi.x) - DX, uy = (x.y - xi.y) - DY, uz = (x.z - xi.z) - DZ;
        const double om = LIN ? delta * rcp3(L) : omega64(d.kernel, delta, rdelta, L);
        const double f = a ? om * x.w : 0.0;
        // S du
        double s0, s1, s2;
        if constexpr (WAN) {
          const double xx = Ai[4].y + Aj[4].y, yy = Ai[5].x + Aj[5].x, zz = Ai[5].y + Aj[5].y;
          const double xy = Ai[6].x + Aj[6].x, xz = Ai[6].y + Aj[6].y, yz = Ai[7].x + Aj[7].x;
          s0 = fma(xx, ux, fma(xy, uy, xz * uz));
          s1 = fma(xy, ux, fma(yy, uy, yz * uz));
          s2 = fma(xz, ux, fma(yz, uy, zz * uz));
        } else {
          const double b = Ai[4].y + Aj[4].y;
          s0 = b * ux;
          s1 = b * uy;
          s2 = b * uz;
        }
        const double t0 = fma(Ai[0].x + Aj[0].x, DX, fma(Ai[1].y + Aj[1].y, DY, fma(Ai[3].x + Aj[3].x, DZ, s0)));
        const double t1 = fma(Ai[0].y + Aj[0].y, DX, fma(Ai[2].x + Aj[2].x, DY, fma(Ai[3].y + Aj[3].y, DZ, s1)));
        const double t2 = fma(Ai[1].x + Aj[1].x, DX, fma(Ai[2].y + Aj[2].y, DY, fma(Ai[4].x + Aj[4].x, DZ, s2)));
        seg[0] = fma(f, t0, seg[0]);
        seg[1] = fma(f, t1, seg[1]);
        seg[2] = fma(f, t2, seg[2]);
      }
    }
    T.add(seg, 0, p.part, p.lane, r0, p.rows);
  }
  if (W > 1 && p.part != 0) return;
  T.template finish<G>(p.lane);
  if (p.valid && p.gl == 0) {
    d.b64[3 * p.i] = T.t[0];
    d.b64[3 * p.i + 1] = T.t[1];
    d.b64[3 * p.i + 2] = T.t[2];
    nan_flag(d, kstep, T.t[0], T.t[1], T.t[2]);
  }
}

// the phase-B state of halo rows whose F and P K^-1 arrived
__global__ void k_c_state_rows(DevBody d, const int* rows, long long n) {
  const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const long long i = rows[r];
  if (i < 0 || i >= d.n) return;
  const unsigned meta = d.meta[i];
  c_state64(d, i, meta & META_KILLED, d.params[meta & META_PID_MASK].beta, d.F64 + 9 * i, d.PK64 + 9 * i,
            d.C164 ? d.C164 + 9 * i : nullptr);
}

void launch_c_state_rows(const DevBody& d, const int* rows, long long n, cudaStream_t s) {
  if (n <= 0 || d.cst64 == nullptr) return;
  k_c_state_rows<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(d, rows, n);
}

// ------------------------------------------------------------------------------------------
// launchers
// ------------------------------------------------------------------------------------------
// Warps per slice (one lane per point): the largest of 8, 4, 2, 1 that keeps the launch within
// four times the 24 warps per SM that the kernels' registers allow. Fewer leave SMs idle in the
// last wave, more only add partial sums. Measured (us a step): 64,000 points OSB 119 at 4 waves,
// 121 at 1, 118 at 8; 125,000 points BB 102, 115 at 1 and 2, 101 at 8 and 103 at 16; CMat 281 at
// 4 (two warps), 314 at 1, 324 at 8, 370 at 16.
constexpr long long SPLIT_WARPS = 4LL * 148 * 24;
static int warps_per_slice(const DevBody& d) {
  if (d.lg != 1) return 1;
  int W = 8;
  while (W > 1 && d.nslices * W > SPLIT_WARPS) W /= 2;
  return W;
}

struct Shape {
  int grid, block;
};
static Shape shape_for(const DevBody& d, const LaunchCfg& c, int W) {
  const int block = W > 1 ? 256 : c.block;
  const long long warps = d.nslices * W;
  long long blocks = (warps + block / 32 - 1) / (block / 32);
  if (blocks < 1) blocks = 1;
  return {(int)blocks, block};
}

#define PD_DISPATCH_GW(d, W, CALL)                                   \
  if ((d).lg == 1) {                                                 \
    constexpr int GG = 1;                                            \
    switch (W) {                                                     \
      case 8: { constexpr int WW = 8; CALL; } break;                 \
      case 4: { constexpr int WW = 4; CALL; } break;                 \
      case 2: { constexpr int WW = 2; CALL; } break;                 \
      default: { constexpr int WW = 1; CALL; } break;                \
    }                                                                \
  } else {                                                           \
    constexpr int WW = 1;                                            \
    switch ((d).lg) {                                                \
      case 2: { constexpr int GG = 2; CALL; } break;                 \
      case 4: { constexpr int GG = 4; CALL; } break;                 \
      case 8: { constexpr int GG = 8; CALL; } break;                 \
      case 16: { constexpr int GG = 16; CALL; } break;               \
      default: { constexpr int GG = 32; CALL; } break;               \
    }                                                                \
  }

// phase B (every BB evaluation and phase A run here)
bool fast64_supported(const DevBody& d) {
  if (!d.sym || d.multi) return false;  // reverse bonds, bond-averaged parameters
  return true;
}

template <bool ESC>
static void launch_bb64f(const DevBody& d, const Shape& q, int W, int kstep, cudaStream_t s) {
  if (d.multi) { PD_DISPATCH_GW(d, W, (k_bb64f<GG, WW, true, ESC><<<q.grid, q.block, 0, s>>>(d, kstep))) }
  else { PD_DISPATCH_GW(d, W, (k_bb64f<GG, WW, false, ESC><<<q.grid, q.block, 0, s>>>(d, kstep))) }
}

template <bool LIN, bool ESC>
static void launch_osb64f(const DevBody& d, const Shape& q, int W, int kstep, int phase, cudaStream_t s) {
  if (phase == 1) { PD_DISPATCH_GW(d, W, (k_osb_a64f<GG, WW, LIN, ESC><<<q.grid, q.block, 0, s>>>(d, kstep))) }
  else { PD_DISPATCH_GW(d, W, (k_osb_b64f<GG, WW, LIN, ESC><<<q.grid, q.block, 0, s>>>(d, kstep))) }
}

template <bool LIN>
static void launch_c64f(const DevBody& d, const Shape& q, int W, int kstep, int phase, cudaStream_t s) {
  if (phase == 1) { PD_DISPATCH_GW(d, W, (k_c_a64f<GG, WW, LIN><<<q.grid, q.block, 0, s>>>(d, kstep))) }
  else if (d.zem == ZEM_WAN) { PD_DISPATCH_GW(d, W, (k_c_b64f<GG, WW, LIN, true><<<q.grid, q.block, 0, s>>>(d, kstep))) }
  else { PD_DISPATCH_GW(d, W, (k_c_b64f<GG, WW, LIN, false><<<q.grid, q.block, 0, s>>>(d, kstep))) }
}

void launch_force64_fast(const DevBody& d, const LaunchCfg& c, int kstep, int phase, cudaStream_t s) {
  if (tile64_supported(d, phase)) {
    launch_tile64(d, kstep, phase, s);
    return;
  }
  const int W = warps_per_slice(d);
  const Shape q = shape_for(d, c, W);
  const bool lin = d.kernel == KER_LINEAR, esc = d.sc64 != nullptr;
  if (d.material == MAT_BB) {
    if (esc) launch_bb64f<true>(d, q, W, kstep, s);
    else launch_bb64f<false>(d, q, W, kstep, s);
  } else if (d.material == MAT_OSB) {
    if (lin && esc) launch_osb64f<true, true>(d, q, W, kstep, phase, s);
    else if (lin) launch_osb64f<true, false>(d, q, W, kstep, phase, s);
    else if (esc) launch_osb64f<false, true>(d, q, W, kstep, phase, s);
    else launch_osb64f<false, false>(d, q, W, kstep, phase, s);
  } else {
    if (lin) launch_c64f<true>(d, q, W, kstep, phase, s);
    else launch_c64f<false>(d, q, W, kstep, phase, s);
  }
}

}  // namespace pd
