// pd_tile64.cu -- the FP64 BB and OSB force kernels on tiles (pd_tiles.cu), for the mappings off the
// serial order with one lane per point: the neighbours' records come from shared memory.
//
// What bounded the kernels that gather from global memory (pd_force64_fast.cu): on the 397,243-point
// block 250 us a launch whatever the occupancy (16 to 40 warps an SM) or the rows in flight, with the
// FP64 pipe at 32 %, DRAM at 26 % and half of every stall a wait for L1: the gathers, one in five of
// them to L2, queue with the bond stream. Here a tile's records are fetched once (about six a point in
// place of 122) and the stream is 8 bytes of length and 2 of the neighbour's place in the tile.
// W warps of a block share a slice and W blocks a tile, as in pd_tile32.cu; the arithmetic and the
// order of the sums are those of pd_force64_fast.cu: the same bits.
#include "pd_bond64.cuh"
#include "pd_common.cuh"
#include "pd_launch.h"

namespace pd {

namespace {

constexpr int TILE_SLICES = 8;

extern __shared__ __align__(16) char tile_smem64[];

// NS: bytes of phase-B state a point (OSB: {c1, c2})
template <int NS, int W>
struct Tile64 {
  const char* sm;
  unsigned c16;  // bytes of one array of 16-byte records
  long long i;
  int rows, lane, part;
  unsigned own, mask;
  bool valid;
  unsigned* bits;
  const unsigned* lidx;
  const double* len;

  __device__ __forceinline__ explicit Tile64(const DevBody& d) {
    const int w = threadIdx.x >> 5;
    lane = threadIdx.x & 31;
    mask = 1u << lane;
    part = w % W;
    const long long sl = (long long)(blockIdx.x / W) * TILE_SLICES + (blockIdx.x % W) * (TILE_SLICES / W) + w / W;
    const long long q = sl * 32 + lane;
    const bool live = sl < d.nslices;
    valid = q < d.n;
    const long long sbase = live ? d.soff[sl] : 0;
    rows = live ? (int)((d.soff[sl + 1] - sbase) >> 5) : 0;
    i = valid ? point_at(d, q) : 0;
    own = d.lown[q];
    bits = d.bits + (sbase >> 5);
    lidx = reinterpret_cast<const unsigned*>(d.lidx + (sbase >> 2) + lane);
    len = d.len64 + sbase + lane;
  }

  // The tile into shared memory, with the first rows of the stream on their way. False: an earlier
  // kernel recorded an error; the block leaves together
  __device__ __forceinline__ bool stage(const DevBody& d) {
    const int err = *(volatile const int*)&d.ctrl->err;
    char* s = tile_smem64;
    sm = s;
    c16 = 16u * (unsigned)d.tile_cap;
    const unsigned tile = blockIdx.x / W;
    const int* list = d.tile_pt + (long long)tile * d.tile_cap;
    const int n = d.tile_n[tile];
#pragma unroll 4
    for (int k = threadIdx.x; k < n; k += 32 * TILE_SLICES) {
      const int p = __ldg(list + k);
      const double2* q = reinterpret_cast<const double2*>(d.cur + p);
      *reinterpret_cast<double2*>(s + 16 * k) = __ldg(q);
      *reinterpret_cast<double2*>(s + c16 + 16 * k) = __ldg(q + 1);
      if constexpr (NS == 16)
        *reinterpret_cast<double2*>(s + 2 * c16 + 16 * k) = __ldg(reinterpret_cast<const double2*>(d.coef64 + p));
    }
    return __syncthreads_or(err) == 0;
  }
  __device__ __forceinline__ double2 xy(unsigned k) const { return *reinterpret_cast<const double2*>(sm + k); }
  __device__ __forceinline__ double2 zv(unsigned k) const { return *reinterpret_cast<const double2*>(sm + c16 + k); }
  __device__ __forceinline__ double2 st(unsigned k) const { return *reinterpret_cast<const double2*>(sm + 2 * c16 + k); }
};

// the stream of rows r (even) and r + 1
struct Pair64 {
  uint2 w;
  unsigned k;
  double L[2];
  // OWNED: the kernel rewrites its state words, which are therefore loaded plainly
  template <bool OWNED, class T>
  __device__ __forceinline__ void load(const T& t, int r) {
    const uint2* q = reinterpret_cast<const uint2*>(t.bits + r);
    w = OWNED ? *q : __ldg(q);
    // four rows hold two words a lane
    k = __ldcs(t.lidx + 16 * (r & ~3) + ((r >> 1) & 1));
    L[0] = __ldcs(t.len + 32 * r);
    L[1] = __ldcs(t.len + 32 * r + 32);
  }
};

// The rows of this warp's segments, as in pd_tile32.cu, the first two in nx: pair(rows, r, sums) adds to the sums of a
// segment, which start from zero and are added to the total in row order; part 0 ends up with it.
template <int W, bool OWNED, int NV, class T, class F>
__device__ __forceinline__ void walk64(const T& t, Pair64 nx, double (&tot)[NV], int& count, F&& pair) {
#pragma unroll
  for (int v = 0; v < NV; v++) tot[v] = 0.0;
  count = 0;
  for (int r0 = 0; r0 < t.rows; r0 += W * SEG64) {
    double seg[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) seg[v] = 0.0;
    int nseg = 0;
    const int ra = r0 + t.part * SEG64, rb = min(ra + SEG64, t.rows);
    for (int r = ra; r < rb; r += 2) {
      const Pair64 c = nx;
      const int nr = r + 2 < rb ? r + 2 : ra + W * SEG64;
      if (nr < t.rows) nx.template load<OWNED>(t, nr);
      pair(c, r, seg, nseg);
    }
    if constexpr (W == 1) {
#pragma unroll
      for (int v = 0; v < NV; v++) tot[v] += seg[v];
      count += nseg;
    } else {
      __shared__ double sh[TILE_SLICES][NV][32];
      __shared__ int shn[TILE_SLICES][32];
      const int w = threadIdx.x >> 5, bar = 1 + w / W;
#pragma unroll
      for (int v = 0; v < NV; v++) sh[w][v][t.lane] = seg[v];
      shn[w][t.lane] = nseg;
      asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(32 * W) : "memory");
      if (t.part == 0) {
#pragma unroll
        for (int q = 0; q < W; q++)
          if (r0 + q * SEG64 < t.rows) {
#pragma unroll
            for (int v = 0; v < NV; v++) tot[v] += sh[w + q][v][t.lane];
            count += shn[w + q][t.lane];
          }
      }
      if (r0 + W * SEG64 < t.rows) asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(32 * W) : "memory");
    }
  }
}

// The same for a kernel that changes no state, one warp a slice: four rows at a time, the four after
// them in registers (nx: the first). OSB phase B, 397,243 points: 230 -> 209 us.
struct Four64 {
  uint4 w;
  uint2 k;
  double L[4];
  template <class T>
  __device__ __forceinline__ void load(const T& t, int r) {
    w = __ldg(reinterpret_cast<const uint4*>(t.bits + r));
    k = __ldcs(reinterpret_cast<const uint2*>(t.lidx) + 8 * r);
#pragma unroll
    for (int u = 0; u < 4; u++) L[u] = __ldcs(t.len + 32 * (r + u));
  }
};

template <int NV, class T, class F>
__device__ __forceinline__ void walk64_four(const T& t, Four64 nx, double (&tot)[NV], F&& pair) {
#pragma unroll
  for (int v = 0; v < NV; v++) tot[v] = 0.0;
  for (int r0 = 0; r0 < t.rows; r0 += SEG64) {
    double seg[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) seg[v] = 0.0;
    const int rb = min(r0 + SEG64, t.rows);
    for (int r = r0; r < rb; r += 4) {
      const Four64 c = nx;
      if (r + 4 < t.rows) nx.load(t, r + 4);
      pair(Pair64{make_uint2(c.w.x, c.w.y), c.k.x, {c.L[0], c.L[1]}}, seg);
      pair(Pair64{make_uint2(c.w.z, c.w.w), c.k.y, {c.L[2], c.L[3]}}, seg);
    }
#pragma unroll
    for (int v = 0; v < NV; v++) tot[v] += seg[v];
  }
}

// the new state words of a row pair where bonds of the warp break
template <class T>
__device__ __forceinline__ void commit(const T& t, const Pair64& c, int r, const bool (&act)[2]) {
  const unsigned c0 = __ballot_sync(0xffffffffu, act[0]), c1 = __ballot_sync(0xffffffffu, act[1]);
  if ((c0 != c.w.x || c1 != c.w.y) && t.lane == 0)
    *reinterpret_cast<uint2*>(t.bits + r) = make_uint2(c0, c1);
}

__device__ __forceinline__ void store64(const DevBody& d, long long i, int kstep, const double (&b)[3]) {
  d.b64[3 * i] = b[0];
  d.b64[3 * i + 1] = b[1];
  d.b64[3 * i + 2] = b[2];
  nan_flag(d, kstep, b[0], b[1], b[2]);
}

// Bodies small enough for eight warps a slice have at most two blocks an SM: those instances take 128
// registers and no spills (BB, 3,200 points: 11.3 -> 10.7 us a step, with the first rows on their way
// while the tile is staged). Resident blocks of 256 threads per SM else, us a launch on the
// 397,243-point block: BB 3 blocks (80 registers) 192 / 2 233; OSB phase A 3 blocks 176 / 2 242; OSB phase
// B (48 bytes a point) 2 blocks 230 / 3 249.
constexpr int MT64_BB = 3, MT64_A = 3, MT64_B = 2;

}  // namespace

// BB (bond_based.jl:125-161)
template <int W>
__global__ void __launch_bounds__(256, W == 8 ? 2 : MT64_BB) k_bb64s(DevBody d, int kstep) {
  Tile64<0, W> t(d);
  Pair64 nx;
  if (t.part * SEG64 < t.rows) nx.load<true>(t, t.part * SEG64);
  if (!t.stage(d)) return;
  const DevParam& P = d.params[t.valid ? d.meta[t.i] & META_PID_MASK : 0];
  const double epsc = P.epsc, thr = fail_threshold(epsc), bc = P.bc;
  const double2 xi = t.xy(t.own);
  const double zi = t.zv(t.own).x;
  double b[3];
  int na;
  walk64<W, true>(t, nx, b, na, [&](const Pair64& c, int r, double (&s)[3], int& n) {
    bool act[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const unsigned k = u ? c.k >> 16 : c.k & 0xffffu;
      const bool a = (u ? c.w.y : c.w.x) & t.mask;
      const double2 x = t.xy(k), z = t.zv(k);
      const double dx = x.x - xi.x, dy = x.y - xi.y, dz = z.x - zi;
      const Bond64 q(dx, dy, dz, c.L[u]);
      act[u] = a && !fails64(q.l2, q.e, c.L[u], q.L, thr, epsc);
      const double sc = act[u] ? (bc * z.y) * (q.e * q.g) : 0.0;
      s[0] = fma(sc, dx, s[0]);
      s[1] = fma(sc, dy, s[1]);
      s[2] = fma(sc, dz, s[2]);
      n += (int)act[u];
    }
    commit(t, c, r, act);
  });
  if (t.valid && t.part == 0) {
    d.n_active[t.i] = na;
    store64(d, t.i, kstep, b);
  }
}

// OSB phase A (ordinary_state_based.jl:107-126, 176-204)
template <int W, bool LIN>
__global__ void __launch_bounds__(256, W == 8 ? 2 : MT64_A) k_osb_a64s(DevBody d, int kstep) {
  Tile64<0, W> t(d);
  Pair64 nx;
  if (t.part * SEG64 < t.rows) nx.load<true>(t, t.part * SEG64);
  if (!t.stage(d)) return;
  const DevParam& P = d.params[t.valid ? d.meta[t.i] & META_PID_MASK : 0];
  const double epsc = P.epsc, thr = fail_threshold(epsc), delta = P.delta, rdelta = 1.0 / delta;
  const double2 xi = t.xy(t.own);
  const double zi = t.zv(t.own).x;
  double m[2];
  int na;
  walk64<W, true>(t, nx, m, na, [&](const Pair64& c, int r, double (&s)[2], int& n) {
    bool act[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const unsigned k = u ? c.k >> 16 : c.k & 0xffffu;
      const bool a = (u ? c.w.y : c.w.x) & t.mask;
      const double2 x = t.xy(k), z = t.zv(k);
      const double dx = x.x - xi.x, dy = x.y - xi.y, dz = z.x - zi;
      const double L = fabs(c.L[u]);
      const double l2 = (dx * dx + dy * dy) + dz * dz;
      const double e = sqrt_of(l2, rsqrt3(l2)) - L;
      act[u] = a && !fails64(l2, e, c.L[u], L, thr, epsc);
      double w = z.y;
      if (!LIN) w *= omega64(d.kernel, delta, rdelta, L) * L;
      s[0] = fma(act[u] ? w : 0.0, L, s[0]);
      s[1] += act[u] ? w * e : 0.0;
      n += (int)act[u];
    }
    commit(t, c, r, act);
  });
  if (t.valid && t.part == 0) {
    const double wvol = LIN ? delta * m[0] : m[0], sdil = LIN ? delta * m[1] : m[1];
    double c1 = 0.0, c2 = 0.0, dil = 0.0;
    if (wvol != 0.0) {
      dil = 3.0 / wvol * sdil;
      c1 = 15.0 * P.G / wvol;
      c2 = dil * (3.0 * P.K / wvol - c1 / 3.0);
    }
    d.coef64[t.i] = make_double4(c1, c2, wvol, dil);
    d.n_active[t.i] = na;
  }
}

// OSB phase B (ordinary_state_based.jl:128-174) for symmetric bond states and one parameter set
template <bool LIN>
__global__ void __launch_bounds__(256, MT64_B) k_osb_b64s(DevBody d, int kstep) {
  Tile64<16, 1> t(d);
  Four64 nx;
  if (t.rows > 0) nx.load(t, 0);
  if (!t.stage(d)) return;
  const double delta = d.params[t.valid ? d.meta[t.i] & META_PID_MASK : 0].delta, rdelta = 1.0 / delta;
  const double2 xi = t.xy(t.own), ci = t.st(t.own);
  const double zi = t.zv(t.own).x;
  double b[3];
  walk64_four(t, nx, b, [&](const Pair64& c, double (&s)[3]) {
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const unsigned k = u ? c.k >> 16 : c.k & 0xffffu;
      const bool a = (u ? c.w.y : c.w.x) & t.mask;
      const double2 x = t.xy(k), z = t.zv(k), cj = t.st(k);
      const double dx = x.x - xi.x, dy = x.y - xi.y, dz = z.x - zi;
      const Bond64 q(dx, dy, dz, c.L[u]);
      const double f = fma(ci.y + cj.y, q.L, (ci.x + cj.x) * q.e);
      const double om = LIN ? delta : omega64(d.kernel, delta, rdelta, q.L) * q.L;
      const double sc = a ? (om * z.y) * (f * q.g) : 0.0;
      s[0] = fma(sc, dx, s[0]);
      s[1] = fma(sc, dy, s[1]);
      s[2] = fma(sc, dz, s[2]);
    }
  });
  if (t.valid) store64(d, t.i, kstep, b);
}

static int tile_bytes64(const DevBody& d, int phase) { return d.tile_cap * (phase == 2 ? 48 : 32); }

// the warps that share a slice: enough for SPLIT64 slices' worth
constexpr long long SPLIT64 = 148 * 24, SPLIT64_8 = 148 * 16;
static int split64(const DevBody& d) {
  int W = 8;
  while (W > 1 && d.nslices * W > (W == 8 ? SPLIT64_8 : SPLIT64)) W /= 2;
  return W;
}

bool tile64_supported(const DevBody& d, int phase) {
  if (d.tile_pt == nullptr || d.len64 == nullptr || d.material == MAT_CMAT || d.multi || d.sc64) return false;
  if (phase == 2 && (!d.sym || split64(d) > 1)) return false;
  return tile_bytes64(d, phase) <= TILE_SMEM;
}

#define PD_TILE_LAUNCH64(W, K)                                                             \
  do {                                                                                     \
    if (allow_tile_smem(K)) K<<<grid * (W), 32 * TILE_SLICES, smem, s>>>(d, kstep);        \
  } while (0)
#define PD_TILE_W64(CALL)                                          \
  switch (W) {                                                     \
    case 8: { constexpr int WW = 8; CALL; } break;                 \
    case 4: { constexpr int WW = 4; CALL; } break;                 \
    case 2: { constexpr int WW = 2; CALL; } break;                 \
    default: { constexpr int WW = 1; CALL; } break;                \
  }

void launch_tile64(const DevBody& d, int kstep, int phase, cudaStream_t s) {
  const long long nt = (d.nslices + TILE_SLICES - 1) / TILE_SLICES;
  const int grid = (int)(nt < 1 ? 1 : nt), smem = tile_bytes64(d, phase);
  const bool lin = d.kernel == KER_LINEAR;
  const int W = split64(d);
  if (d.material == MAT_BB) {
    PD_TILE_W64(PD_TILE_LAUNCH64(WW, (k_bb64s<WW>)))
  } else if (phase == 1) {
    if (lin) { PD_TILE_W64(PD_TILE_LAUNCH64(WW, (k_osb_a64s<WW, true>))) }
    else { PD_TILE_W64(PD_TILE_LAUNCH64(WW, (k_osb_a64s<WW, false>))) }
  } else if (lin) {
    PD_TILE_LAUNCH64(1, (k_osb_b64s<true>));
  } else {
    PD_TILE_LAUNCH64(1, (k_osb_b64s<false>));
  }
}

}  // namespace pd
