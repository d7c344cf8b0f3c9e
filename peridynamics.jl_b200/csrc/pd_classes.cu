// pd_classes.cu -- bond classes: the distinct {reference vector, +-length} records of a body's
// bonds in the FP32 form.
//
// On a regular lattice every bond repeats one of a hundred or so records (122 at a horizon of
// 3.015 spacings), so that one byte a bond replaces the 16 bytes of geometry that the kernels
// otherwise stream from DRAM in every phase. Found once per layout:
//   k_class_collect  every bond looks its record up in an open-addressed table of 64-bit
//                    fingerprints and claims a slot when there is none; the claimant writes the
//                    record. More than 256 records (a jittered lattice, a mesh) end the pass
//                    after the first few rows of every warp;
//   k_class_number   numbers the claimed slots in the order of their bits, so that the numbering
//                    does not depend on which bond came first;
//   k_class_write    writes the byte of every bond, comparing the whole record: two records with
//                    one fingerprint leave the body without classes.
#include "pd_common.cuh"
#include "pd_launch.h"

namespace pd {

constexpr int CLASS_SLOTS = 4096;

struct ClassScratch {
  unsigned long long fp[CLASS_SLOTS];  // 0: free
  uint4 rec[CLASS_SLOTS];
  int id[CLASS_SLOTS];
  int count, failed;
};

__device__ __forceinline__ uint4 class_record(const DevBody& d, long long b) {
  const float4 g = d.geo[b];
  return make_uint4(__float_as_uint(g.x), __float_as_uint(g.y), __float_as_uint(g.z), __float_as_uint(g.w));
}

__device__ __forceinline__ bool class_same(const uint4& a, const uint4& b) {
  return a.x == b.x && a.y == b.y && a.z == b.z && a.w == b.w;
}

// a nonzero 64-bit fingerprint: the words through the mixing steps of splitmix64 (Steele, Lea and Flood, Fast
// splittable pseudorandom number generators, 2014)
__device__ __forceinline__ unsigned long long class_print(const uint4& r) {
  const unsigned v[4] = {r.x, r.y, r.z, r.w};
  unsigned long long h = 0x9E3779B97F4A7C15ull;
  for (int k = 0; k < 4; k++) {
    h ^= v[k];
    h *= 0xBF58476D1CE4E5B9ull;
    h ^= h >> 27;
    h *= 0x94D049BB133111EBull;
    h ^= h >> 31;
  }
  return h ? h : 1ull;
}

__global__ void __launch_bounds__(256) k_class_collect(DevBody d, ClassScratch* t) {
  const int lane = threadIdx.x & 31;
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= d.n) return;
  const long long i = point_at(d, q), sbase = d.soff[q >> 5];
  const int cnt = (int)(d.off[i + 1] - d.off[i]);
  for (int r = 0; r < cnt; r++) {
    if (*(volatile const int*)&t->failed) return;
    const uint4 rec = class_record(d, sbase + 32LL * r + lane);
    const unsigned long long f = class_print(rec);
    int h = (int)(f % CLASS_SLOTS);
    bool in = false;
    for (int probe = 0; probe < CLASS_SLOTS && !in; probe++) {
      unsigned long long old = *(volatile const unsigned long long*)&t->fp[h];
      if (old == 0) {
        old = atomicCAS(&t->fp[h], 0ull, f);
        if (old == 0) {
          t->rec[h] = rec;
          if (atomicAdd(&t->count, 1) >= MAX_CLASSES) atomicExch(&t->failed, 1);
          old = f;
        }
      }
      in = old == f;
      if (!in) h = (h + 1) % CLASS_SLOTS;
    }
    if (!in) atomicExch(&t->failed, 1);
  }
}

__device__ __forceinline__ bool class_less(const uint4& a, const uint4& b) {
  if (a.x != b.x) return a.x < b.x;
  if (a.y != b.y) return a.y < b.y;
  return a.z != b.z ? a.z < b.z : a.w < b.w;
}

// one block: the rank of every claimed slot among the claimed ones
__global__ void __launch_bounds__(1024) k_class_number(ClassScratch* t, float4* geo) {
  __shared__ int used[MAX_CLASSES];
  __shared__ int n;
  if (t->failed) return;
  if (threadIdx.x == 0) n = 0;
  __syncthreads();
  for (int q = threadIdx.x; q < CLASS_SLOTS; q += blockDim.x)
    if (t->fp[q]) used[atomicAdd(&n, 1)] = q;
  __syncthreads();
  for (int a = threadIdx.x; a < n; a += blockDim.x) {
    const uint4 me = t->rec[used[a]];
    int rank = 0;
    for (int b = 0; b < n; b++) rank += class_less(t->rec[used[b]], me);
    t->id[used[a]] = rank;
    geo[rank] = make_float4(__uint_as_float(me.x), __uint_as_float(me.y), __uint_as_float(me.z),
                            __uint_as_float(me.w));
  }
}

// word r / 4 of a slice: the classes of its rows r .. r + 3 (row r lowest) of 32 lanes
__global__ void __launch_bounds__(256) k_class_write(DevBody d, ClassScratch* t, unsigned* cls) {
  const int lane = threadIdx.x & 31;
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x, s = q >> 5;
  if (s >= d.nslices || t->failed) return;
  const long long i = q < d.n ? point_at(d, q) : 0, sbase = d.soff[s];
  const int rows = (int)((d.soff[s + 1] - sbase) >> 5);
  const int cnt = q < d.n ? (int)(d.off[i + 1] - d.off[i]) : 0;
  unsigned* out = cls + (sbase >> 2) + lane;
  for (int r4 = 0; r4 < rows; r4 += 4) {
    unsigned w = 0;
    for (int u = 0; u < 4 && r4 + u < cnt; u++) {
      const uint4 rec = class_record(d, sbase + 32LL * (r4 + u) + lane);
      const unsigned long long f = class_print(rec);
      int h = (int)(f % CLASS_SLOTS);
      for (int probe = 0; probe < CLASS_SLOTS && t->fp[h] != f && t->fp[h] != 0; probe++)
        h = (h + 1) % CLASS_SLOTS;
      if (t->fp[h] != f || !class_same(t->rec[h], rec)) { t->failed = 2; return; }
      w |= (unsigned)t->id[h] << (8 * u);
    }
    out[8 * r4] = w;
  }
}

cudaError_t build_classes(const DevBody& d, long long nslots, unsigned** cls, float4** geo, int* ncls,
                          cudaStream_t s) {
  *cls = nullptr;
  *geo = nullptr;
  *ncls = 0;
  if (d.n == 0 || d.nb == 0 || d.lg != 1 || d.geo == nullptr) return cudaSuccess;
  ClassScratch* t = nullptr;
  const unsigned grid = (unsigned)((d.nslices + 7) / 8);
  int found[2] = {0, 1};
  auto status = [&]() {
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(found, &t->count, sizeof(found), cudaMemcpyDeviceToHost, s);
    return e == cudaSuccess ? cudaStreamSynchronize(s) : e;
  };
  cudaError_t e = cudaMalloc(&t, sizeof(ClassScratch));
  if (e == cudaSuccess) e = cudaMemsetAsync(t, 0, sizeof(ClassScratch), s);
  if (e == cudaSuccess) {
    k_class_collect<<<grid, 256, 0, s>>>(d, t);
    e = status();
  }
  if (e == cudaSuccess && found[1] == 0) {
    e = cudaMalloc(cls, (size_t)nslots);
    if (e == cudaSuccess) e = cudaMalloc(geo, sizeof(float4) * MAX_CLASSES);
    if (e == cudaSuccess) {
      k_class_number<<<1, 1024, 0, s>>>(t, *geo);
      k_class_write<<<grid, 256, 0, s>>>(d, t, *cls);
      e = status();
    }
    if (e == cudaSuccess && found[1] == 0) *ncls = found[0];
  }
  cudaFree(t);
  if (*ncls == 0) {
    cudaFree(*cls);
    cudaFree(*geo);
    *cls = nullptr;
    *geo = nullptr;
  }
  return e;
}

}  // namespace pd
