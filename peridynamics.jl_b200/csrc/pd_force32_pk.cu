// pd_force32_pk.cu -- FP32-compensated BB and OSB force kernels with fewer instructions per bond and
// the bond stream of the next row pair in flight (one lane per point, the sliced layout of G = 1, bodies
// whose tiles do not fit).
//
// The two-row kernels (pd_force32.cu) issue about 93 (phase A) and 116 (phase B) warp
// instructions per bond row. These compute the same quantities with 75 / 68:
//   - the x and y components of every per-bond 3-vector (displacement difference, deformed
//     bond vector, the force and its compensated sum) are one packed pair (f32x2: one
//     instruction for both components), z is scalar;
//   - bond states select the contribution instead of branching around it: inactive bonds and
//     padding slots gather their own point (always in bounds) and add zero;
//   - the bond stream is addressed from the slice base with 32-bit row offsets;
//   - phase B is written for symmetric bond states with one parameter set, where the two
//     directions of a bond share its influence value: s_ij + s_ji = w ((c2_i + c2_j) L +
//     (c1_i + c1_j) e), one packed add for both coefficient sums.
// With fewer instructions alone the kernels ran slower (issue utilisation fell from 71 % to
// 40 %, long-scoreboard stalls per issue rose from 4.7 to 14.7 on the 1M-point block): the
// phases are bound by the latency of the bond stream and the neighbour gathers that depend on
// it, not by issue. The freed registers therefore hold the next row pair's stream records,
// loaded after the current pair's gathers and before its arithmetic, so the DRAM latency of
// the stream overlaps the gathers and arithmetic of the pair before it. The stream loads are
// streaming (evict-first) loads, so that the bond records, read once, leave L2 to the
// neighbours' point records.
// The arithmetic is the FP32 form of pd_force32.cu (deformed bond vector from the stored
// reference offset, cancellation-free extension, Kahan sums); roundings differ from the
// two-row kernels only in the order of a few operations.
// Where a body has tiles, pd_tile32.cu runs the same arithmetic on them instead.
#include "pd_bond32.cuh"
#include "pd_common.cuh"
#include "pd_launch.h"
#include "pd_pack.cuh"

namespace pd {

namespace {

using namespace pack;

}  // namespace

// occupancy bounds: phase A at 4 resident blocks of 256 threads (59 registers), phase B at 3
// (72 registers; at 4 it spills). Measured on the 8M-point OSB block, blocks of 128:
// 4.24 / 4.47 ms against 4.40 / 4.70 ms for the two-row kernels; phase B at 4 blocks (with
// spills) 4.78 ms, at 2 blocks 6.18 ms.
#ifndef PD_MINB_QA
#define PD_MINB_QA 4
#endif
#ifndef PD_MINB_QB
#define PD_MINB_QB 3
#endif

// Phase B with the bond stream of the next row pair loaded while the current pair is
// gathered and computed (one pair of rows ahead): the DRAM latency of the stream overlaps the
// gathers and arithmetic of the pair before it. MB resident blocks per SM.
template <bool LIN>
__global__ void __launch_bounds__(256, PD_MINB_QB) k_osb_b32q(DevBody d, int kstep) {
  if (d.ctrl->err) return;
  const int lane = threadIdx.x & 31;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long s = warp0; s < d.nslices; s += nwarps) {
    const long long place = s * 32 + lane;
    const bool valid = place < d.n;
    const long long i = valid ? point_at(d, place) : place;
    const int self = valid ? (int)i : 0;
    const long long sbase = d.soff[s];
    const int rows = (int)((d.soff[s + 1] - sbase) >> 5);
    const DevParam& P = d.params[d.meta[self] & META_PID_MASK];
    const Influence om(d, P);
    const float4 hi = d.uhi[self], lo = d.ulo[self];
    const float2 ci = d.cc32[self];
    const Own32 own(hi, lo);
    const int* pn = d.nbr + sbase + lane;
    const float4* pg = d.geo + sbase + lane;
    const unsigned* pw = d.bits + (sbase >> 5);
    KSum2 bxy, txy;  // the sums of the segment and of the point
    KSum1 bz, tz;
    // stream records of the pair (r, r + 1): neighbour (self when inactive), geometry, state
    int nj0 = self, nj1 = self;
    float4 ng0 = make_float4(0.f, 0.f, 0.f, 1.f), ng1 = ng0;
    unsigned nw0 = 0u, nw1 = 0u;
    auto load_pair = [&](int r) {
      const bool two = r + 1 < rows;
      nw0 = ld_stream(pw + r);
      nw1 = two ? ld_stream(pw + r + 1) : 0u;
      nj0 = ld_stream(pn + 32 * r);
      ng0 = ld_stream(pg + 32 * r);
      if (two) { nj1 = ld_stream(pn + 32 * r + 32); ng1 = ld_stream(pg + 32 * r + 32); }
      else { nj1 = self; ng1 = make_float4(0.f, 0.f, 0.f, 1.f); }
    };
    if (rows > 0) load_pair(0);
    for (int r = 0; r < rows; r += 2) {
      const bool a0 = (nw0 >> lane) & 1u, a1 = (nw1 >> lane) & 1u;
      const int j0 = a0 ? nj0 : self, j1 = a1 ? nj1 : self;
      const float4 g0 = ng0, g1 = ng1;
      // gathers of this pair, then the stream of the next pair, then the arithmetic
      const float4 hj0 = __ldg(d.uhi + j0), lj0 = __ldg(d.ulo + j0);
      const float4 hj1 = __ldg(d.uhi + j1), lj1 = __ldg(d.ulo + j1);
      const float2 cj0 = __ldg(d.cc32 + j0), cj1 = __ldg(d.cc32 + j1);
      if (r + 2 < rows) load_pair(r + 2);
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const float4& g = u ? g1 : g0;
        const float4& hj = u ? hj1 : hj0;
        BondP B;
        bond_pk(g, hj, u ? lj1 : lj0, own, B);
        const float rL = bond_rl(g.w);
        const float2 cs = add2(ci, u ? cj1 : cj0);
        float f = osb_pair<LIN>(om, B, rL, cs, hj.w);
        f = (u ? a1 : a0) ? f : 0.f;
        bxy.add(mul2(make_float2(f, f), B.exy));
        bz.add(f * B.ez);
      }
      if ((r + 2) % SEG32 == 0 || r + 2 >= rows) {
        join(txy, bxy);
        join(tz, bz);
        bxy = KSum2();
        bz = KSum1();
      }
    }
    if (valid) {
      store_force(d, i, kstep, LIN ? P.delta : 1.0, txy, tz);
    }
  }
}

// Phase A with the next row pair's stream loaded one pair ahead (as k_osb_b32q).
template <bool FULLM, bool LIN>
__global__ void __launch_bounds__(256, PD_MINB_QA) k_osb_a32q(DevBody d, int kstep) {
  if (d.ctrl->err) return;
  const int lane = threadIdx.x & 31;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long s = warp0; s < d.nslices; s += nwarps) {
    const long long place = s * 32 + lane;
    const bool valid = place < d.n;
    const long long i = valid ? point_at(d, place) : place;
    const int self = valid ? (int)i : 0;
    const long long sbase = d.soff[s];
    const int rows = (int)((d.soff[s + 1] - sbase) >> 5);
    const DevParam& P = d.params[d.meta[self] & META_PID_MASK];
    const float epsc = P.epscf;
    const Influence om(d, P);
    const float4 hi = d.uhi[self], lo = d.ulo[self];
    const Own32 own(hi, lo);
    const int* pn = d.nbr + sbase + lane;
    const float4* pg = d.geo + sbase + lane;
    unsigned* pw = d.bits + (sbase >> 5);
    double sm = 0.0, tm = 0.0;  // the sums of the segment and of the point
    KSum1 th, tth;
    float dm = 0.f, tdm = 0.f;
    int na = 0;
    int nj0 = self, nj1 = self;
    float4 ng0 = make_float4(0.f, 0.f, 0.f, 1.f), ng1 = ng0;
    unsigned nw0 = 0u, nw1 = 0u;
    // the state words are plain loads: this warp owns them and rewrites them below
    auto load_pair = [&](int r) {
      const bool two = r + 1 < rows;
      nw0 = pw[r];
      nw1 = two ? pw[r + 1] : 0u;
      nj0 = ld_stream(pn + 32 * r);
      ng0 = ld_stream(pg + 32 * r);
      if (two) { nj1 = ld_stream(pn + 32 * r + 32); ng1 = ld_stream(pg + 32 * r + 32); }
      else { nj1 = self; ng1 = make_float4(0.f, 0.f, 0.f, 1.f); }
    };
    if (rows > 0) load_pair(0);
    for (int r = 0; r < rows; r += 2) {
      const bool two = r + 1 < rows;
      const unsigned w0 = nw0, w1 = nw1;
      const bool a0 = (w0 >> lane) & 1u, a1 = (w1 >> lane) & 1u;
      const int j0 = a0 ? nj0 : self, j1 = a1 ? nj1 : self;
      const float4 g0 = ng0, g1 = ng1;
      const float4 hj0 = __ldg(d.uhi + j0), lj0 = __ldg(d.ulo + j0);
      const float4 hj1 = __ldg(d.uhi + j1), lj1 = __ldg(d.ulo + j1);
      if (r + 2 < rows) load_pair(r + 2);
      bool act0, act1;
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const float4& g = u ? g1 : g0;
        const float4& hj = u ? hj1 : hj0;
        const bool a = u ? a1 : a0;
        BondP B;
        bond_pk(g, hj, u ? lj1 : lj0, own, B);
        const float rL = bond_rl(g.w);
        const bool act = stays(a, B.e * rL, epsc, g.w);
        th.add(act ? dil_term<LIN>(om, B, rL, hj.w) : 0.f);
        if (FULLM) sm += act ? vol_term<LIN>(om, g.w, hj.w) : 0.0;
        else if (a && !act) dm += (float)vol_term<LIN>(om, g.w, hj.w);
        if (u) act1 = act; else act0 = act;
      }
      na += (int)act0 + (int)act1;
      const unsigned c0 = __ballot_sync(0xffffffffu, act0);
      const unsigned c1 = __ballot_sync(0xffffffffu, act1);
      if (lane == 0) {
        if (c0 != w0) pw[r] = c0;
        if (two && c1 != w1) pw[r + 1] = c1;
      }
      if ((r + 2) % SEG32 == 0 || r + 2 >= rows) {
        tm += sm;
        join(tth, th);
        tdm += dm;
        sm = 0.0;
        th = KSum1();
        dm = 0.f;
      }
    }
    if (valid) {
      double m;
      if (FULLM) m = vol_point<LIN>(P, tm);
      else m = tdm != 0.f ? vol_less<LIN>(d, P, i, tdm) : vol_stored(d, i);
      osb_point<LIN>(d, P, i, m, (double)tth.s + (double)tth.n);
      d.n_active[i] = na;
    }
  }
}

// BB (calc_failure! and force_density_point!, bond_based.jl:125-161) in one sweep with packed
// pairs and the next row pair's stream in flight, as the OSB phases above: f = bc eps V_j eta / l
// for the bonds that stay active, the failure test on eps = e / L.
#ifndef PD_MINB_QBB
#define PD_MINB_QBB 4
#endif
__global__ void __launch_bounds__(256, PD_MINB_QBB) k_bb32q(DevBody d, int kstep) {
  if (d.ctrl->err) return;
  const int lane = threadIdx.x & 31;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long s = warp0; s < d.nslices; s += nwarps) {
    const long long place = s * 32 + lane;
    const bool valid = place < d.n;
    const long long i = valid ? point_at(d, place) : place;
    const int self = valid ? (int)i : 0;
    const long long sbase = d.soff[s];
    const int rows = (int)((d.soff[s + 1] - sbase) >> 5);
    const DevParam& P = d.params[d.meta[self] & META_PID_MASK];
    const float epsc = P.epscf;
    const float4 hi = d.uhi[self], lo = d.ulo[self];
    const Own32 own(hi, lo);
    const int* pn = d.nbr + sbase + lane;
    const float4* pg = d.geo + sbase + lane;
    unsigned* pw = d.bits + (sbase >> 5);
    KSum2 bxy, txy;  // the sums of the segment and of the point
    KSum1 bz, tz;
    int na = 0;
    int nj0 = self, nj1 = self;
    float4 ng0 = make_float4(0.f, 0.f, 0.f, 1.f), ng1 = ng0;
    unsigned nw0 = 0u, nw1 = 0u;
    // the state words are plain loads: this warp owns them and rewrites them below
    auto load_pair = [&](int r) {
      const bool two = r + 1 < rows;
      nw0 = pw[r];
      nw1 = two ? pw[r + 1] : 0u;
      nj0 = ld_stream(pn + 32 * r);
      ng0 = ld_stream(pg + 32 * r);
      if (two) { nj1 = ld_stream(pn + 32 * r + 32); ng1 = ld_stream(pg + 32 * r + 32); }
      else { nj1 = self; ng1 = make_float4(0.f, 0.f, 0.f, 1.f); }
    };
    if (rows > 0) load_pair(0);
    for (int r = 0; r < rows; r += 2) {
      const bool two = r + 1 < rows;
      const unsigned w0 = nw0, w1 = nw1;
      const bool a0 = (w0 >> lane) & 1u, a1 = (w1 >> lane) & 1u;
      const int j0 = a0 ? nj0 : self, j1 = a1 ? nj1 : self;
      const float4 g0 = ng0, g1 = ng1;
      const float4 hj0 = __ldg(d.uhi + j0), lj0 = __ldg(d.ulo + j0);
      const float4 hj1 = __ldg(d.uhi + j1), lj1 = __ldg(d.ulo + j1);
      if (r + 2 < rows) load_pair(r + 2);
      bool act0, act1;
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const float4& g = u ? g1 : g0;
        const float4& hj = u ? hj1 : hj0;
        const bool a = u ? a1 : a0;
        BondP B;
        bond_pk(g, hj, u ? lj1 : lj0, own, B);
        const float rL = bond_rl(g.w);
        const float eps = B.e * rL;
        const bool act = stays(a, eps, epsc, g.w);
        const float sc = act ? eps * (hj.w * B.rl) : 0.f;
        bxy.add(mul2(make_float2(sc, sc), B.exy));
        bz.add(sc * B.ez);
        if (u) act1 = act; else act0 = act;
      }
      na += (int)act0 + (int)act1;
      const unsigned c0 = __ballot_sync(0xffffffffu, act0);
      const unsigned c1 = __ballot_sync(0xffffffffu, act1);
      if (lane == 0) {
        if (c0 != w0) pw[r] = c0;
        if (two && c1 != w1) pw[r + 1] = c1;
      }
      if ((r + 2) % SEG32 == 0 || r + 2 >= rows) {
        join(txy, bxy);
        join(tz, bz);
        bxy = KSum2();
        bz = KSum1();
      }
    }
    if (valid) {
      d.n_active[i] = na;
      store_force(d, i, kstep, P.bc, txy, tz);
    }
  }
}

// the packed kernels serve one lane per point, BB and OSB without surface correction and with
// one parameter set; OSB's phase B also needs symmetric bond states
bool pk_supported(const DevBody& d, int phase) {
  if (d.material == MAT_CMAT || d.lg != 1 || d.sc32 != nullptr || d.multi) return false;
  if (d.material == MAT_BB) return phase == 1;
  if (phase == 2 && !d.sym) return false;
  return true;
}

static int grid_pk(long long nslices, int block) {
  long long blocks = (nslices + block / 32 - 1) / (block / 32);
  if (blocks < 1) blocks = 1;
  if (PD_GRID_BLOCKS_PER_SM > 0 && blocks > 148LL * PD_GRID_BLOCKS_PER_SM)
    blocks = 148LL * PD_GRID_BLOCKS_PER_SM;
  return (int)blocks;
}

int launch_force32_pk(const DevBody& d, const LaunchCfg& c, int kstep, int phase, cudaStream_t s) {
  const int grid = grid_pk(d.nslices, c.block);
  const bool lin = d.kernel == KER_LINEAR;
  int launches = 0;
  if (d.material == MAT_BB) {
    if (phase == 2) return 0;
    k_bb32q<<<grid, c.block, 0, s>>>(d, kstep);
    return 1;
  }
  if (phase != 2) {
    if (c.fullk) {
      if (lin) k_osb_a32q<true, true><<<grid, c.block, 0, s>>>(d, kstep);
      else k_osb_a32q<true, false><<<grid, c.block, 0, s>>>(d, kstep);
    } else {
      if (lin) k_osb_a32q<false, true><<<grid, c.block, 0, s>>>(d, kstep);
      else k_osb_a32q<false, false><<<grid, c.block, 0, s>>>(d, kstep);
    }
    launches++;
  }
  if (phase != 1) {
    if (lin) k_osb_b32q<true><<<grid, c.block, 0, s>>>(d, kstep);
    else k_osb_b32q<false><<<grid, c.block, 0, s>>>(d, kstep);
    launches++;
  }
  return launches;
}

}  // namespace pd
