// pd_tiles.cu -- which points share a slice, and tiles of eight slices (one lane per point).
//
// The neighbour records that the 256 points of a block gather are fetched once into shared memory
// instead of once per bond. What a block then has to fetch is the union of its points' horizons,
// which is smallest for a compact block: a brick of 8 x 8 x 4 points at a horizon of 3.015 spacings
// has 1,400 of them, where 256 consecutive points of a lattice (one or two rows of it) have about
// 5,000. So with one lane per point the places of the slices follow the points through columns of
// 8 x 4 spacings that run the length of the body, up one and down the next: eight consecutive
// slices are 8 x 4 x 8 spacings wherever along the column they begin. (Bricks on a Morton curve do as
// well where the body's sides are multiples of the brick's; elsewhere eight slices straddle two of
// them: on 211 x 199 x 101 points 1,522 on average and 1,934 at most, against 1,361 and 1,628.) The
// long edge of the column's section runs along the axis on which consecutive points lie, so that
// eight lanes read consecutive records. Points keep their numbers everywhere else; bond lists, their
// order and the sums over them do not depend on the places.
#include <cub/cub.cuh>

#include "pd_common.cuh"
#include "pd_launch.h"

namespace pd {

__global__ void k_place_key(DevBody d, PlaceGrid g, unsigned long long* key, int* idx) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n) return;
  const double4 X = d.X0[i];
  const double c[3] = {X.x, X.y, X.z};
  unsigned q[3];
  for (int a = 0; a < 3; a++) {
    const double v = floor((c[g.axis[a]] - g.lo[g.axis[a]]) * g.inv + 0.5);
    q[a] = v > 0.0 ? (v < 65535.0 ? (unsigned)v : 65535u) : 0u;
  }
  // parameter set (the specimens of an ensemble, which may share coordinates), column, place along
  // it, place in its section
  const unsigned cx = q[0] >> 3, cz = q[2] >> 2;
  const unsigned long long along = (cx + cz) & 1u ? 65535u - q[1] : q[1];
  const unsigned long long col = (unsigned long long)cx << 14 | (cx & 1u ? 16383u - cz : cz);
  key[i] = (unsigned long long)(d.meta[i] & META_PID_MASK) << 48 | col << 21 | along << 5 |
           (q[0] & 7u) | (q[2] & 3u) << 3;
  idx[i] = (int)i;
}

__global__ void k_place_inverse(long long n, const int* pt, int* place) {
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q < n) place[pt[q]] = (int)q;
}

cudaError_t build_places(const DevBody& d, const PlaceGrid& g, int** pt, int** place, cudaStream_t s) {
  const long long n = d.n;
  *pt = nullptr;
  *place = nullptr;
  if (n == 0) return cudaSuccess;
  unsigned long long *k0 = nullptr, *k1 = nullptr;
  int* idx = nullptr;
  void* tmp = nullptr;
  size_t need = 0;
  const unsigned grid = (unsigned)((n + 255) / 256);
  cudaError_t e = cudaMalloc(pt, sizeof(int) * n);
  if (e == cudaSuccess) e = cudaMalloc(place, sizeof(int) * n);
  if (e == cudaSuccess) e = cudaMalloc(&k0, sizeof(*k0) * n);
  if (e == cudaSuccess) e = cudaMalloc(&k1, sizeof(*k1) * n);
  if (e == cudaSuccess) e = cudaMalloc(&idx, sizeof(int) * n);
  if (e == cudaSuccess) {
    k_place_key<<<grid, 256, 0, s>>>(d, g, k0, idx);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cub::DeviceRadixSort::SortPairs(nullptr, need, k0, k1, idx, *pt, (int)n, 0, 64, s);
  if (e == cudaSuccess) e = cudaMalloc(&tmp, need > 0 ? need : 1);
  if (e == cudaSuccess) e = cub::DeviceRadixSort::SortPairs(tmp, need, k0, k1, idx, *pt, (int)n, 0, 64, s);
  if (e == cudaSuccess) {
    k_place_inverse<<<grid, 256, 0, s>>>(n, *pt, *place);
    e = cudaGetLastError();
  }
  const cudaError_t es = cudaStreamSynchronize(s);
  if (e == cudaSuccess) e = es;
  cudaFree(k0);
  cudaFree(k1);
  cudaFree(idx);
  cudaFree(tmp);
  if (e != cudaSuccess) {
    cudaFree(*pt);
    cudaFree(*place);
    *pt = nullptr;
    *place = nullptr;
  }
  return e;
}

// ------------------------------------------------------------------------------------------
// tiles
// ------------------------------------------------------------------------------------------
constexpr int TILE_SLICES = 8, TILE_POINTS = 32 * TILE_SLICES;
constexpr int TILE_HASH = 8192;

// One block per tile: the points of its slices and their neighbours, each once, in a hash set in
// shared memory; then sorted. WRITE false: their number only. stat: {largest number, failed}.
template <bool WRITE>
__global__ void __launch_bounds__(256) k_tile_points(DevBody d, int cap, int* tile_pt, int* tile_n,
                                                     uint2* lidx, unsigned short* lown, int* stat) {
  extern __shared__ int sm[];
  int* set = sm;                // [TILE_HASH]
  int* list = sm + TILE_HASH;   // [TILE_MAX + 1]
  __shared__ int n;
  const long long q = (long long)blockIdx.x * TILE_POINTS + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const long long s = q >> 5;
  const bool live = s < d.nslices, valid = q < d.n;
  const long long i = valid ? point_at(d, q) : 0;
  const long long sbase = live ? d.soff[s] : 0;
  const int rows = live ? (int)((d.soff[s + 1] - sbase) >> 5) : 0;
  const int cnt = valid ? (int)(d.off[i + 1] - d.off[i]) : 0;
  for (int k = threadIdx.x; k < TILE_HASH; k += blockDim.x) set[k] = -1;
  if (threadIdx.x == 0) n = 0;
  __syncthreads();
  auto insert = [&](int p) {
    unsigned h = (unsigned)p * 2654435761u >> 19;  // 13 bits
    for (int t = 0; t < TILE_HASH; t++) {
      const int old = *(volatile int*)&set[h];
      if (old == p) return;
      if (old == -1) {
        const int was = atomicCAS(&set[h], -1, p);
        if (was == -1) {
          const int at = atomicAdd(&n, 1);
          if (at < TILE_MAX) list[at] = p;
          return;
        }
        if (was == p) return;
      }
      if (*(volatile int*)&n > TILE_MAX) return;
      h = (h + 1) % TILE_HASH;
    }
  };
  if (valid) insert((int)i);
  for (int r = 0; r < cnt; r++) {
    if (*(volatile int*)&n > TILE_MAX) break;
    insert(d.nbr[sbase + 32LL * r + lane]);
  }
  __syncthreads();
  const int total = n;
  if (total > TILE_MAX) {
    if (threadIdx.x == 0) stat[1] = 1;
    return;
  }
  if (!WRITE) {
    if (threadIdx.x == 0) atomicMax(&stat[0], total);
    return;
  }
  // bitonic sort, padded to a power of two
  int m = 1;
  while (m < total) m *= 2;
  for (int k = total + threadIdx.x; k < m; k += blockDim.x) list[k] = 0x7fffffff;
  for (int w = 2; w <= m; w *= 2)
    for (int h = w / 2; h > 0; h /= 2) {
      __syncthreads();
      for (int k = threadIdx.x; k < m / 2; k += blockDim.x) {
        const int a = 2 * h * (k / h) + k % h, b = a + h;
        const bool up = (a & w) == 0;
        const int x = list[a], y = list[b];
        if ((x > y) == up) { list[a] = y; list[b] = x; }
      }
    }
  __syncthreads();
  auto find = [&](int p) {
    int a = 0, z = total;
    while (a < z) {
      const int mid = (a + z) >> 1;
      if (list[mid] < p) a = mid + 1; else z = mid;
    }
    return (unsigned)a * 16u;  // the byte offset of a 16-byte record
  };
  int* out = tile_pt + (long long)blockIdx.x * cap;
  for (int k = threadIdx.x; k < total; k += blockDim.x) out[k] = list[k];
  if (threadIdx.x == 0) tile_n[blockIdx.x] = total;
  const unsigned own = valid ? find((int)i) : 0u;
  lown[q] = (unsigned short)own;
  for (int r = 0; r < rows; r += 4) {
    unsigned v[4];
    for (int u = 0; u < 4; u++) v[u] = r + u < cnt ? find(d.nbr[sbase + 32LL * (r + u) + lane]) : own;
    lidx[(sbase >> 2) + 8LL * r + lane] = make_uint2(v[0] | v[1] << 16, v[2] | v[3] << 16);
  }
}

cudaError_t build_tiles(const DevBody& d, long long nslots, TileArrays* out, cudaStream_t s) {
  *out = TileArrays{};
  if (d.n == 0 || d.nb == 0 || d.lg != 1) return cudaSuccess;
  const long long nt = (d.nslices + TILE_SLICES - 1) / TILE_SLICES;
  const int smem = sizeof(int) * (TILE_HASH + TILE_MAX + 1);
  int *stat = nullptr, h[2] = {0, 0};
  TileArrays t{};
  auto status = [&]() {
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, stat, sizeof(h), cudaMemcpyDeviceToHost, s);
    return e == cudaSuccess ? cudaStreamSynchronize(s) : e;
  };
  cudaError_t e = cudaMalloc(&stat, sizeof(h));
  if (e == cudaSuccess) e = cudaMemsetAsync(stat, 0, sizeof(h), s);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_tile_points<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_tile_points<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess) {
    k_tile_points<false><<<(unsigned)nt, 256, smem, s>>>(d, 0, nullptr, nullptr, nullptr, nullptr, stat);
    e = status();
  }
  if (e == cudaSuccess && h[1] == 0) {
    t.cap = (h[0] + 7) / 8 * 8;
    e = cudaMalloc(&t.pt, sizeof(int) * t.cap * nt);
    if (e == cudaSuccess) e = cudaMalloc(&t.n, sizeof(int) * nt);
    if (e == cudaSuccess) e = cudaMalloc(&t.lidx, sizeof(uint2) * (nslots / 4));
    if (e == cudaSuccess) e = cudaMalloc(&t.lown, sizeof(unsigned short) * TILE_POINTS * nt);
    if (e == cudaSuccess) {
      k_tile_points<true><<<(unsigned)nt, 256, smem, s>>>(d, t.cap, t.pt, t.n, t.lidx, t.lown, stat);
      e = status();
    }
    if (e != cudaSuccess) {
      cudaFree(t.pt);
      cudaFree(t.n);
      cudaFree(t.lidx);
      cudaFree(t.lown);
    } else {
      *out = t;
    }
  }
  cudaFree(stat);
  return e;
}

}  // namespace pd
