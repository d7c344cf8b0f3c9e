// pd_tile32.cu -- the packed FP32 kernels on tiles: a block of 256 threads takes the 256 points of a
// tile (pd_tiles.cu), brings the records of all their neighbours into shared memory once, and every
// bond then reads its neighbour there.
//
// What bounded the kernels that gather from global memory (pd_force32_pk.cu, 1M-point OSB block):
// first the latency of the 20-byte bond stream; with that stream cut to a byte a bond, the L1 data
// pipe. 32 consecutive 16-byte records that start anywhere cost eight wavefronts, a phase-B row 27
// in all (l1tex__data_pipe_lsu_wavefronts at 82 %), and only the three bonds of a lattice line
// shared a line in L1 (hit rate 74 %). From shared memory a row costs four wavefronts an array
// wherever it starts, and a point of the tile's surroundings is fetched once for the block: about
// six records a point in place of 122.
//
// A bond's stream is its neighbour's place in the tile (16 bits), its state bit and its reference
// vector and length: one byte where the body has bond classes (pd_classes.cu, template flag CLS; the
// records are kept in shared memory with 1 / L), 16 bytes otherwise. The arithmetic and its order
// are those of pd_force32_pk.cu: the same bits.
//
// Time of a step, lattices at a horizon of 3.015 spacings, packed kernels before and tiles (us, CUDA
// graphs): OSB 1M points 1003 -> 635, 4.24M 4381 -> 2694, jittered 1M 1056 -> 949; BB 1M 501 -> 362;
// CMat (variant 5) 320k 464 -> 317, 125k 232 -> 185. Against the one-row kernels of an untuned body: OSB 975
// points 65 -> 17, 27,347 105 -> 38, 64,000 185 -> 66; CMat 64,000 212 -> 88. OSB phase A issues 75 % of its
// slots with the L1 pipe at 63 %: arithmetic and the neighbour and class records read from shared
// memory (12 wavefronts a row) are what is left. With the full geometry stream DRAM is at 56 %, and
// copying it ahead asynchronously (4 to 8 rows in shared memory) changed no time by more than 3 %.
//
// Below the size at which tiles fill the chip, W warps of a block share a slice and W blocks a tile:
// the slice's rows are cut into segments of SEG32 rows that are summed from zero and joined in row
// order, whatever W is.
#include <cstring>

#include "pd_bond32.cuh"
#include "pd_common.cuh"
#include "pd_launch.h"
#include "pd_pack.cuh"
#include "pd_point32.cuh"

namespace pd {

namespace {

using namespace pack;

constexpr int TILE_SLICES = 8;

// dynamic shared memory: {(float)u, V} and the low part of every point of the tile, NS bytes of
// phase-B state a point, the class records and their 1 / L
__host__ __device__ __forceinline__ int tile_bytes(int cap, int ns, int ncls) {
  return cap * (32 + ns) + ncls * 20;
}

struct Pair32 {
  unsigned w[2];
  bool a[2];
  unsigned key[2];  // byte offset of the neighbour's 16-byte records
  float4 g[2];
  unsigned cls[2];
};

// A warp walks four rows at a time, with the neighbour places and classes of the four after them in
// registers. The state words: OWNED, the kernel rewrites them, so they are loaded plainly, two rows
// ahead; else four rows ahead as well (CMat phase B, 320k points: 212 -> 169 us, OSB phase B, 1M points:
// 342 -> 314; with two blocks per SM the wait for two rows' words was the largest stall. In the OWNED
// kernels the four registers cost more than the wait: OSB phase A 298 -> 350).
template <bool CLS, bool OWNED>
struct TileStream {
  const float* rl;      // CLS: 1 / L of the classes
  const float4* geo;    // CLS: their records
  const unsigned* pw;
  const uint2* pl;
  const unsigned* pc;
  const float4* pg;
  int rows;
  unsigned mask;
  uint2 nw;             // OWNED: states of the next row pair
  uint4 wi, wn;         // else: states of these four rows and of the next
  uint2 li, ln;         // neighbour places
  unsigned cw, cn;      // classes
  float4 ng0, ng1;      // without classes: geometry of the next row pair

  __device__ __forceinline__ TileStream(const DevBody& d, const float4* geo_, const float* rl_,
                                        long long sbase, int rows_, int lane)
      : rl(rl_), geo(geo_), pw(d.bits + (sbase >> 5)), pl(d.lidx + (sbase >> 2) + lane), rows(rows_),
        mask(1u << lane) {
    if constexpr (CLS) pc = d.cls + (sbase >> 2) + lane;
    else pg = d.geo + sbase + lane;
  }

  // the four rows from r on are the first that the warp walks, those from `after` the second
  __device__ __forceinline__ void start(int r, int after) {
    if (r >= rows) return;
    fetch(r);
    load<0>(r, after);
  }
  __device__ __forceinline__ void fetch(int r) {
    if constexpr (!OWNED) wn = ld_stream(reinterpret_cast<const uint4*>(pw + r));
    ln = ld_stream(pl + 8 * r);
    if constexpr (CLS) cn = ld_stream(pc + 8 * r);
  }
  // the records of rows r and r + 1; H: the second pair of its four rows; else the four rows that the
  // warp walks after them start at `after`
  template <int H>
  __device__ __forceinline__ void load(int r, int after) {
    if constexpr (OWNED) nw = *reinterpret_cast<const uint2*>(pw + r);
    if constexpr (H == 0) {
      if constexpr (!OWNED) wi = wn;
      li = ln;
      if constexpr (CLS) cw = cn;
      if (after < rows) fetch(after);
    }
    if constexpr (!CLS) {
      ng0 = ld_stream(pg + 32 * r);
      ng1 = ld_stream(pg + 32 * r + 32);
    }
  }

  template <int H>
  __device__ __forceinline__ void take(Pair32& p) const {
    const unsigned v = H ? li.y : li.x;
    p.w[0] = OWNED ? nw.x : H ? wi.z : wi.x;
    p.w[1] = OWNED ? nw.y : H ? wi.w : wi.y;
    p.a[0] = (p.w[0] & mask) != 0u;
    p.a[1] = (p.w[1] & mask) != 0u;
    p.key[0] = v & 0xffffu;
    p.key[1] = v >> 16;
    if constexpr (CLS) {
      p.cls[0] = (cw >> (16 * H)) & 255u;
      p.cls[1] = (cw >> (16 * H + 8)) & 255u;
      p.g[0] = geo[p.cls[0]];
      p.g[1] = geo[p.cls[1]];
    } else {
      p.g[0] = ng0;
      p.g[1] = ng1;
    }
  }
  __device__ __forceinline__ float rL(const Pair32& p, int u) const {
    if constexpr (CLS) return rl[p.cls[u]];
    else return bond_rl(p.g[u].w);
  }
};

// A broken bond adds zero times its vector, and a neighbour that a point has lost may be anywhere, at
// infinity too. NEAR: the tile holds every displacement within +-1e37 and its low part within +-1e30 (below
// 2^-24 of that), where zero times a bond vector is zero and an unbroken bond to such a point still has no
// defined length. A select of the point itself in the loop costs the BB kernel registers that it spills
// (17.8 -> 18.9 ms for 40 steps of 1M points); correspondence, which spills none and multiplies the
// displacement by the stabilising stiffness, takes the select.
constexpr float FAR32 = 1e37f, FAR32_LO = 1e30f;
__device__ __forceinline__ float4 near32(const float4& u, float far) {
  return make_float4(fminf(fmaxf(u.x, -far), far), fminf(fmaxf(u.y, -far), far),
                     fminf(fmaxf(u.z, -far), far), u.w);
}

// one block: its tile in shared memory, the place of every thread
template <bool CLS, int NS, int W, bool NEAR>
struct Tile {
  char* sm;
  unsigned c16;          // bytes of one array of 16-byte records
  const float4* geo;
  const float* rl;
  long long i, sbase;
  int rows, lane, part;
  unsigned own;
  bool valid;

  // false: an earlier kernel recorded an error; the block leaves together
  __device__ __forceinline__ bool begin(const DevBody& d, char* smem) {
    const int err = *(volatile const int*)&d.ctrl->err;
    sm = smem;
    c16 = 16u * (unsigned)d.tile_cap;
    const unsigned tile = blockIdx.x / W;
    const int* list = d.tile_pt + (long long)tile * d.tile_cap;
    const int n = d.tile_n[tile];
#pragma unroll 4
    for (int k = threadIdx.x; k < n; k += 32 * TILE_SLICES) {
      const int p = __ldg(list + k);
      const float4 h = __ldg(d.uhi + p), l = __ldg(d.ulo + p);
      *reinterpret_cast<float4*>(sm + 16 * k) = NEAR ? near32(h, FAR32) : h;
      *reinterpret_cast<float4*>(sm + c16 + 16 * k) = NEAR ? near32(l, FAR32_LO) : l;
      if constexpr (NS == 8)
        *reinterpret_cast<float2*>(sm + 2 * c16 + 8 * k) = __ldg(d.cc32 + p);
      if constexpr (NS == 40) {
        const float4* q = d.cst32 + 3 * (long long)p;
        const float4 c = __ldg(q + 2);
        *reinterpret_cast<float4*>(sm + 2 * c16 + 16 * k) = __ldg(q);
        *reinterpret_cast<float4*>(sm + 3 * c16 + 16 * k) = __ldg(q + 1);
        *reinterpret_cast<float2*>(sm + 4 * c16 + 8 * k) = make_float2(c.x, c.y);
      }
    }
    if constexpr (CLS) {
      float4* tg = reinterpret_cast<float4*>(sm + d.tile_cap * (32 + NS));
      float* tr = reinterpret_cast<float*>(tg + d.ncls);
      for (int k = threadIdx.x; k < d.ncls; k += blockDim.x) {
        const float4 g = __ldg(d.cls_geo + k);
        tg[k] = g;
        tr[k] = bond_rl(g.w);
      }
      geo = tg;
      rl = tr;
    }
    // warp w of the block: slice w / W of its eight / W, part w % W of that slice's rows
    const int w = threadIdx.x >> 5;
    lane = threadIdx.x & 31;
    part = w % W;
    const long long s = (long long)tile * TILE_SLICES + (blockIdx.x % W) * (TILE_SLICES / W) + w / W;
    const long long q = s * 32 + lane;
    const bool live = s < d.nslices;
    valid = q < d.n;
    i = valid ? point_at(d, q) : 0;
    sbase = live ? d.soff[s] : 0;
    rows = live ? (int)((d.soff[s + 1] - sbase) >> 5) : 0;
    own = d.lown[q];
    return __syncthreads_or(err) == 0;
  }
  __device__ __forceinline__ float4 hi(unsigned k) const { return *reinterpret_cast<const float4*>(sm + k); }
  __device__ __forceinline__ float4 lo(unsigned k) const { return *reinterpret_cast<const float4*>(sm + c16 + k); }
  __device__ __forceinline__ float2 s8(unsigned k) const {
    return *reinterpret_cast<const float2*>(sm + 2 * c16 + (k >> 1));
  }
  __device__ __forceinline__ float4 sa(unsigned k) const { return *reinterpret_cast<const float4*>(sm + 2 * c16 + k); }
  __device__ __forceinline__ float4 sb(unsigned k) const { return *reinterpret_cast<const float4*>(sm + 3 * c16 + k); }
  __device__ __forceinline__ float2 sc(unsigned k) const {
    return *reinterpret_cast<const float2*>(sm + 4 * c16 + (k >> 1));
  }
};

// The rows of this warp's segments: first the segment of its part, then W segments on. A segment's
// sums (ACC, trivially copyable, joined by join) start from zero and join the total in row order;
// after the last round part 0 holds it. The barrier is the slice's own: its W warps walk the same
// rows.
template <int W, class ACC, class ST, class F>
__device__ __forceinline__ ACC walk_rows(ST& st, int rows, int part, int lane, F&& pair) {
  ACC tot;
  // the four rows that the warp walks after those at r: on in the segment, or W segments on
  auto next = [&](int r) {
    if constexpr (W == 1) return r + 4;
    else return (r + 4) % SEG32 != 0 && r + 4 < rows ? r + 4 : r / SEG32 * SEG32 + W * SEG32;
  };
  st.start(part * SEG32, next(part * SEG32));
  for (int r0 = 0; r0 < rows; r0 += W * SEG32) {
    ACC seg;
    const int ra = r0 + part * SEG32, rb = min(ra + SEG32, rows);
    for (int r = ra; r < rb; r += 4) {
      Pair32 p;
      st.template take<0>(p);
      st.template load<1>(r + 2, 0);
      pair(p, r, seg);
      st.template take<1>(p);
      const int nx = next(r);
      if (nx < rows) st.template load<0>(nx, next(nx));
      pair(p, r + 2, seg);
    }
    if constexpr (W == 1) {
      tot.join(seg);
    } else {
      constexpr int NW = sizeof(ACC) / 4;
      __shared__ unsigned sh[TILE_SLICES][NW][32];
      const int w = threadIdx.x >> 5, bar = 1 + w / W;
      unsigned v[NW];
      memcpy(v, &seg, sizeof(ACC));
#pragma unroll
      for (int k = 0; k < NW; k++) sh[w][k][lane] = v[k];
      asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(32 * W) : "memory");
      if (part == 0) {
#pragma unroll
        for (int q = 0; q < W; q++)
          if (r0 + q * SEG32 < rows) {
#pragma unroll
            for (int k = 0; k < NW; k++) v[k] = sh[w + q][k][lane];
            memcpy(&seg, v, sizeof(ACC));
            tot.join(seg);
          }
      }
      if (r0 + W * SEG32 < rows) asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(32 * W) : "memory");
    }
  }
  return tot;
}

// Whether the tile has the point at the end of its range: two such points are not at rest. (OSB has seen
// that in phase A.)
__device__ __forceinline__ bool far_off(const Own32& o) {
  return !(fmaxf(fmaxf(fabsf(o.nhi.x), fabsf(o.nhi.y)), fabsf(o.nhz)) < FAR32);
}

// a force sum and a count
struct ForceSum {
  KSum2 xy;
  KSum1 z;
  int lost = 0;
  __device__ __forceinline__ void add(float f, const float2 v, float vz) {
    xy.add(mul2(both(f), v));
    z.add(f * vz);
  }
  __device__ __forceinline__ void join(const ForceSum& o) {
    pack::join(xy, o.xy);
    pack::join(z, o.z);
    lost += o.lost;
  }
};

// the sums of OSB phase A: dilatation; in full also the weighted volume (in double), else what the stored
// one loses; the active bonds in full, else those that break
template <bool FULLM>
struct DilSum {
  KSum1 th;
  float dm = 0.f;
  int na = 0;
  __device__ __forceinline__ void join(const DilSum& o) {
    pack::join(th, o.th);
    dm += o.dm;
    na += o.na;
  }
};
template <>
struct DilSum<true> {
  double m = 0.0;
  KSum1 th;
  int na = 0;
  __device__ __forceinline__ void join(const DilSum& o) {
    m += o.m;
    pack::join(th, o.th);
    na += o.na;
  }
};

// Resident blocks of 256 threads per SM, measured on 1M-point blocks with the first form of these kernels
// (us a launch): BB 4 blocks (64 registers) 295 / 3 361 / 5 426; OSB phase A 4 blocks 287 / 3 360 / 5 406, full geometry stream 438 /
// 476 / 701; OSB phase B 3 blocks (80 registers) 336 / 4 377; CMat phase A 3 blocks 403 / 2 507, with
// compensated sums 2 blocks 525, phase B 2 blocks (tiles of 72 bytes a point fill the SM) 537 / 3 579.
constexpr int MT_BB = 4, MT_A = 4, MT_B = 3, MT_CA = 3, MT_CAK = 2, MT_CB = 2;

}  // namespace

extern __shared__ __align__(16) char tile_smem[];

// BB (bond_based.jl:125-161)
template <bool CLS, int W>
__global__ void __launch_bounds__(256, MT_BB) k_bb32s(DevBody d, int kstep) {
  Tile<CLS, 0, W, true> t;
  if (!t.begin(d, tile_smem)) return;
  const DevParam& P = d.params[t.valid ? d.meta[t.i] & META_PID_MASK : 0];
  const float epsc = P.epscf;
  const Own32 own(t.hi(t.own), t.lo(t.own));
  TileStream<CLS, true> st(d, t.geo, t.rl, t.sbase, t.rows, t.lane);
  ForceSum S = walk_rows<W, ForceSum>(st, t.rows, t.part, t.lane, [&](const Pair32& p, int r, ForceSum& s) {
    bool act[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const float4 hj = t.hi(p.key[u]);
      BondP B;
      bond_pk(p.g[u], hj, t.lo(p.key[u]), own, B);
      const float eps = B.e * st.rL(p, u);
      act[u] = stays(p.a[u], eps, epsc, p.g[u].w);
      s.add(act[u] ? eps * (hj.w * B.rl) : 0.f, B.exy, B.ez);
    }
    const unsigned c0 = __ballot_sync(0xffffffffu, act[0]), c1 = __ballot_sync(0xffffffffu, act[1]);
    if (c0 != p.w[0] || c1 != p.w[1]) {  // bonds of this warp break
      s.lost += (int)(p.a[0] && !act[0]) + (int)(p.a[1] && !act[1]);
      if (t.lane == 0) *reinterpret_cast<uint2*>(d.bits + (t.sbase >> 5) + r) = make_uint2(c0, c1);
    }
  });
  if (t.valid && t.part == 0) {
    if (far_off(own)) S.z.s = NAN;
    if (S.lost) d.n_active[t.i] -= S.lost;
    store_force(d, t.i, kstep, P.bc, S.xy, S.z);
  }
}

// OSB phase A (ordinary_state_based.jl:107-126, 176-204): failure, the stored weighted volume less
// the bonds that break (FULLM: summed in full), dilatation, c1 and c2
template <bool CLS, int W, bool FULLM, bool LIN>
__global__ void __launch_bounds__(256, MT_A) k_osb_a32s(DevBody d, int kstep) {
  Tile<CLS, 0, W, false> t;
  if (!t.begin(d, tile_smem)) return;
  const DevParam& P = d.params[t.valid ? d.meta[t.i] & META_PID_MASK : 0];
  const float epsc = P.epscf;
  const Influence om(d, P);
  const Own32 own(t.hi(t.own), t.lo(t.own));
  TileStream<CLS, true> st(d, t.geo, t.rl, t.sbase, t.rows, t.lane);
  using Sum = DilSum<FULLM>;
  const Sum S = walk_rows<W, Sum>(st, t.rows, t.part, t.lane, [&](const Pair32& p, int r, Sum& s) {
    bool act[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const float4 hj = t.hi(p.key[u]);
      BondP B;
      bond_pk(p.g[u], hj, t.lo(p.key[u]), own, B);
      const float rL = st.rL(p, u);
      act[u] = stays(p.a[u], B.e * rL, epsc, p.g[u].w);
      s.th.add(act[u] ? dil_term<LIN>(om, B, rL, hj.w) : 0.f);
      if constexpr (FULLM) {
        s.m += act[u] ? vol_term<LIN>(om, p.g[u].w, hj.w) : 0.0;
        s.na += (int)act[u];
      }
    }
    const unsigned c0 = __ballot_sync(0xffffffffu, act[0]), c1 = __ballot_sync(0xffffffffu, act[1]);
    if (c0 != p.w[0] || c1 != p.w[1]) {  // bonds of this warp break
      if constexpr (!FULLM) {
#pragma unroll
        for (int u = 0; u < 2; u++)
          if (p.a[u] && !act[u]) {
            s.dm += (float)vol_term<LIN>(om, p.g[u].w, t.hi(p.key[u]).w);
            s.na++;
          }
      }
      if (t.lane == 0) *reinterpret_cast<uint2*>(d.bits + (t.sbase >> 5) + r) = make_uint2(c0, c1);
    }
  });
  if (t.valid && t.part == 0) {
    double m;
    if constexpr (FULLM) m = vol_point<LIN>(P, S.m);
    else m = S.dm != 0.f ? vol_less<LIN>(d, P, t.i, S.dm) : vol_stored(d, t.i);
    osb_point<LIN>(d, P, t.i, m, (double)S.th.s + (double)S.th.n);
    if (FULLM) d.n_active[t.i] = S.na;
    else if (S.na) d.n_active[t.i] -= S.na;
  }
}

// OSB phase B (ordinary_state_based.jl:128-174) for symmetric bond states
template <bool CLS, int W, bool LIN>
__global__ void __launch_bounds__(256, MT_B) k_osb_b32s(DevBody d, int kstep) {
  Tile<CLS, 8, W, true> t;
  if (!t.begin(d, tile_smem)) return;
  const DevParam& P = d.params[t.valid ? d.meta[t.i] & META_PID_MASK : 0];
  const Influence om(d, P);
  const Own32 own(t.hi(t.own), t.lo(t.own));
  const float2 ci = t.s8(t.own);
  TileStream<CLS, false> st(d, t.geo, t.rl, t.sbase, t.rows, t.lane);
  const ForceSum S = walk_rows<W, ForceSum>(st, t.rows, t.part, t.lane, [&](const Pair32& p, int r, ForceSum& s) {
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const float4 hj = t.hi(p.key[u]);
      BondP B;
      bond_pk(p.g[u], hj, t.lo(p.key[u]), own, B);
      const float f = osb_pair<LIN>(om, B, st.rL(p, u), add2(ci, t.s8(p.key[u])), hj.w);
      s.add(p.a[u] ? f : 0.f, B.exy, B.ez);
    }
  });
  if (t.valid && t.part == 0)
    store_force(d, t.i, kstep, LIN ? P.delta : 1.0, S.xy, S.z);
}

// the sums of correspondence phase A and its count; not cut into segments (their sums would take
// their registers twice), so always one warp a slice
template <bool FULLK, bool COMP>
struct CorrAcc : CorrSums<FULLK, COMP> {
  int na = 0;  // FULLK: the active bonds; else the bonds that break in this evaluation
};

// CMat phase A (correspondence.jl:193-224, 288-298; bond_system.jl:309-327)
template <bool CLS, bool FULLK, bool LIN, bool COMP>
__global__ void __launch_bounds__(256, COMP ? MT_CAK : MT_CA) k_c_a32s(DevBody d, int kstep) {
  Tile<CLS, 0, 1, false> t;
  if (!t.begin(d, tile_smem)) return;
  const unsigned meta = t.valid ? d.meta[t.i] : 0u;
  const DevParam& P = d.params[meta & META_PID_MASK];
  const CorrA cp(d, P);
  const Own32 own(t.hi(t.own), t.lo(t.own));
  CorrAcc<FULLK, COMP> S;
  TileStream<CLS, true> st(d, t.geo, t.rl, t.sbase, t.rows, t.lane);
  auto pair = [&](const Pair32& p, int r) {
    bool act[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const unsigned k = p.a[u] ? p.key[u] : t.own;
      const float4 hj = t.hi(k);
      float2 dxy;
      float dz, num;
      bond_du(p.g[u], hj, t.lo(k), own, dxy, dz, num);
      const float rL = st.rL(p, u);
      act[u] = corr_stays(p.a[u], cp, p.g[u], rL, dxy, dz, num);
      const float w = corr_weight<LIN>(cp, p.g[u], rL, hj.w);
      S.add(act[u] ? w : 0.f, p.g[u], dxy, dz);
      if (FULLK) S.na += (int)act[u];
    }
    const unsigned c0 = __ballot_sync(0xffffffffu, act[0]), c1 = __ballot_sync(0xffffffffu, act[1]);
    if (c0 != p.w[0] || c1 != p.w[1]) {  // bonds of this warp break
      if (!FULLK) {
#pragma unroll
        for (int u = 0; u < 2; u++)
          if (p.a[u] && !act[u]) {
            S.drop(corr_weight<LIN>(cp, p.g[u], st.rL(p, u), t.hi(p.key[u]).w), p.g[u]);
            S.na++;
          }
      }
      if (t.lane == 0) *reinterpret_cast<uint2*>(d.bits + (t.sbase >> 5) + r) = make_uint2(c0, c1);
    }
  };
  st.start(0, 4);
  for (int r = 0; r < t.rows; r += 4) {
    Pair32 p;
    st.template take<0>(p);
    st.template load<1>(r + 2, 0);
    pair(p, r);
    st.template take<1>(p);
    if (r + 4 < t.rows) st.template load<0>(r + 4, r + 8);
    pair(p, r + 2);
  }
  bool killed = false;
  if (t.valid) {
    const int cnt = (int)(d.off[t.i + 1] - d.off[t.i]);
    const int na = FULLK ? S.na : d.n_active[t.i] - S.na;
    killed = corr_point32(d, P, t.i, meta, cnt, na, S);
  }
  if (!d.sym) {
    // directed bond states: a killed point loses all its bonds (correspondence.jl:293)
    const unsigned kill_mask = __ballot_sync(0xffffffffu, killed);
    if (kill_mask && t.lane == 0)
      for (int r = 0; r < t.rows; r++) d.bits[(t.sbase >> 5) + r] &= ~kill_mask;
  }
}

// CMat phase B (correspondence.jl:226-251) for ZEMSilling and symmetric bond states
template <bool CLS, int W, bool LIN>
__global__ void __launch_bounds__(256, MT_CB) k_c_b32s(DevBody d, int kstep) {
  Tile<CLS, 40, W, false> t;
  if (!t.begin(d, tile_smem)) return;
  const DevParam& P = d.params[t.valid ? d.meta[t.i] & META_PID_MASK : 0];
  const Influence om(d, P);
  const Own32 own(t.hi(t.own), t.lo(t.own));
  const float4 ia = t.sa(t.own), ib = t.sb(t.own);
  const float2 ic = t.sc(t.own);
  TileStream<CLS, false> st(d, t.geo, t.rl, t.sbase, t.rows, t.lane);
  const ForceSum S = walk_rows<W, ForceSum>(st, t.rows, t.part, t.lane, [&](const Pair32& p, int r, ForceSum& s) {
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const unsigned k = p.a[u] ? p.key[u] : t.own;
      const float4 hj = t.hi(k);
      float2 dxy, txy;
      float dz, num, tz;
      bond_du(p.g[u], hj, t.lo(k), own, dxy, dz, num);
      corr_pair(p.g[u], dxy, dz, ia, ib, ic, t.sa(k), t.sb(k), t.sc(k), txy, tz);
      const float f = (LIN ? st.rL(p, u) : om.at<LIN>(fabsf(p.g[u].w), 0.f)) * hj.w;
      s.add(p.a[u] ? f : 0.f, txy, tz);
    }
  });
  if (t.valid && t.part == 0)
    store_force(d, t.i, kstep, LIN ? P.delta : 1.0, S.xy, S.z);
}

static int state_bytes(const DevBody& d, int phase) {
  return phase == 1 ? 0 : d.material == MAT_OSB ? 8 : 40;
}

// a tile, its classes and the segment sums of the warps that share a slice fit the 227 KB of a block
bool tile32_supported(const DevBody& d, int phase) {
  return d.tile_pt != nullptr && tile_bytes(d.tile_cap, state_bytes(d, phase), d.ncls) <= TILE_SMEM;
}

// Warps per slice: the largest of 8, 4, 2, 1 that keeps the launch within the 24 warps per SM that
// the tiles leave room for. More warps leave each less of the tile it waits for, fewer leave SMs
// idle. Measured (OSB, us a step): 27,347 points 4 warps 37, 2 warps 44, 8 warps 46; 64,000 points 1
// warp 69, 2 warps 78, 4 warps 74.
constexpr long long SPLIT32 = 148 * 24;
static int tile_split(const DevBody& d) {
  int W = 8;
  while (W > 1 && d.nslices * W > SPLIT32) W /= 2;
  return W;
}

#define PD_TILE_LAUNCH(W, K)                                                               \
  do {                                                                                     \
    if (allow_tile_smem(K)) K<<<grid * (W), 32 * TILE_SLICES, smem, s>>>(d, kstep);        \
  } while (0)
#define PD_TILE_W(CALL)                                            \
  switch (W) {                                                     \
    case 8: { constexpr int WW = 8; CALL; } break;                 \
    case 4: { constexpr int WW = 4; CALL; } break;                 \
    case 2: { constexpr int WW = 2; CALL; } break;                 \
    default: { constexpr int WW = 1; CALL; } break;                \
  }

// correspondence phase A: plain sums of the displacement gradient are bond-stream variant 5's
template <bool CLS, bool COMP>
static void launch_c_a(const DevBody& d, const LaunchCfg& c, int kstep, int grid, int smem, cudaStream_t s) {
  const bool lin = d.kernel == KER_LINEAR;
  if (c.fullk) {
    if (lin) PD_TILE_LAUNCH(1, (k_c_a32s<CLS, true, true, COMP>));
    else PD_TILE_LAUNCH(1, (k_c_a32s<CLS, true, false, COMP>));
  } else {
    if (lin) PD_TILE_LAUNCH(1, (k_c_a32s<CLS, false, true, COMP>));
    else PD_TILE_LAUNCH(1, (k_c_a32s<CLS, false, false, COMP>));
  }
}

template <bool CLS>
static void launch_tile(const DevBody& d, const LaunchCfg& c, int kstep, int phase, cudaStream_t s) {
  const long long nt = (d.nslices + TILE_SLICES - 1) / TILE_SLICES;
  const int grid = (int)(nt < 1 ? 1 : nt), smem = tile_bytes(d.tile_cap, state_bytes(d, phase), d.ncls);
  const bool lin = d.kernel == KER_LINEAR;
  const int W = tile_split(d);
  if (d.material == MAT_BB) {
    PD_TILE_W(PD_TILE_LAUNCH(WW, (k_bb32s<CLS, WW>)))
  } else if (d.material == MAT_OSB) {
    if (phase == 2) {
      if (lin) { PD_TILE_W(PD_TILE_LAUNCH(WW, (k_osb_b32s<CLS, WW, true>))) }
      else { PD_TILE_W(PD_TILE_LAUNCH(WW, (k_osb_b32s<CLS, WW, false>))) }
    } else if (c.fullk) {
      if (lin) { PD_TILE_W(PD_TILE_LAUNCH(WW, (k_osb_a32s<CLS, WW, true, true>))) }
      else { PD_TILE_W(PD_TILE_LAUNCH(WW, (k_osb_a32s<CLS, WW, true, false>))) }
    } else {
      if (lin) { PD_TILE_W(PD_TILE_LAUNCH(WW, (k_osb_a32s<CLS, WW, false, true>))) }
      else { PD_TILE_W(PD_TILE_LAUNCH(WW, (k_osb_a32s<CLS, WW, false, false>))) }
    }
  } else if (phase == 2) {
    if (lin) { PD_TILE_W(PD_TILE_LAUNCH(WW, (k_c_b32s<CLS, WW, true>))) }
    else { PD_TILE_W(PD_TILE_LAUNCH(WW, (k_c_b32s<CLS, WW, false>))) }
  } else if (c.pipe == 5) {
    launch_c_a<CLS, false>(d, c, kstep, grid, smem, s);
  } else {
    launch_c_a<CLS, true>(d, c, kstep, grid, smem, s);
  }
}

void launch_tile32(const DevBody& d, const LaunchCfg& c, int kstep, int phase, cudaStream_t s) {
  if (d.ncls > 0) launch_tile<true>(d, c, kstep, phase, s);
  else launch_tile<false>(d, c, kstep, phase, s);
}

}  // namespace pd
