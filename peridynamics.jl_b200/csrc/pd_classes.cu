// pd_classes.cu -- bond classes: the distinct (j - i, reference vector, +-length) records of a
// body's bonds.
//
// On a regular lattice every bond repeats one of a hundred or so records (122 at a horizon of
// 3.015 spacings), so that one byte a bond replaces the 20 bytes of neighbour index and geometry
// that the packed FP32 kernels otherwise stream from DRAM in every phase. Found once per body:
//   k_class_collect  every bond looks its record up in an open-addressed table of 64-bit
//                    fingerprints and claims a slot when there is none; the claimant writes the
//                    record. More than 256 records (a jittered lattice, a mesh) end the pass
//                    after the first few rows of every warp;
//   k_class_number   numbers the claimed slots in ascending (j - i, record) order, so that the
//                    numbering does not depend on which bond came first;
//   k_class_write    writes the byte of every bond, comparing the whole record: two records with
//                    one fingerprint leave the body without classes.
#include "pd_common.cuh"
#include "pd_launch.h"
#include "pd_stream32.cuh"

namespace pd {

constexpr int CLASS_SLOTS = 4096;

struct ClassRec {
  unsigned v[5];  // j - i and the bits of the geometry record
};

struct ClassScratch {
  unsigned long long fp[CLASS_SLOTS];  // 0: free
  ClassRec rec[CLASS_SLOTS];
  int id[CLASS_SLOTS];
  int count, failed;
};

__device__ __forceinline__ ClassRec class_record(const DevBody& d, long long b, long long i) {
  const float4 g = d.geo[b];
  return ClassRec{{(unsigned)(d.nbr[b] - (int)i), __float_as_uint(g.x), __float_as_uint(g.y),
                   __float_as_uint(g.z), __float_as_uint(g.w)}};
}

// a nonzero 64-bit fingerprint (splitmix64 finaliser over the words)
__device__ __forceinline__ unsigned long long class_print(const ClassRec& r) {
  unsigned long long h = 0x9E3779B97F4A7C15ull;
  for (int k = 0; k < 5; k++) {
    h ^= r.v[k];
    h *= 0xBF58476D1CE4E5B9ull;
    h ^= h >> 27;
    h *= 0x94D049BB133111EBull;
    h ^= h >> 31;
  }
  return h ? h : 1ull;
}

__device__ __forceinline__ unsigned long long class_fp(const ClassScratch* t, int q) {
  return *(volatile const unsigned long long*)&t->fp[q];
}

__global__ void __launch_bounds__(256) k_class_collect(DevBody d, ClassScratch* t) {
  const int lane = threadIdx.x & 31;
  const long long s = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (s >= d.nslices) return;
  const long long i = s * 32 + lane;
  const long long sbase = d.soff[s];
  const int cnt = i < d.n ? (int)(d.off[i + 1] - d.off[i]) : 0;
  for (int r = 0; r < cnt; r++) {
    if (*(volatile const int*)&t->failed) return;
    const ClassRec rec = class_record(d, sbase + 32LL * r + lane, i);
    const unsigned long long f = class_print(rec);
    int q = (int)(f % CLASS_SLOTS);
    bool in = false;
    for (int probe = 0; probe < CLASS_SLOTS && !in; probe++) {
      unsigned long long old = class_fp(t, q);
      if (old == 0) {
        old = atomicCAS(&t->fp[q], 0ull, f);
        if (old == 0) {
          t->rec[q] = rec;
          if (atomicAdd(&t->count, 1) >= MAX_CLASSES) atomicExch(&t->failed, 1);
          old = f;
        }
      }
      in = old == f;
      if (!in) q = (q + 1) % CLASS_SLOTS;
    }
    if (!in) atomicExch(&t->failed, 1);
  }
}

__device__ __forceinline__ bool class_less(const ClassRec& a, const ClassRec& b) {
  const int da = (int)a.v[0], db = (int)b.v[0];
  if (da != db) return da < db;
  for (int k = 1; k < 5; k++)
    if (a.v[k] != b.v[k]) return a.v[k] < b.v[k];
  return false;
}

// one block: the rank of every claimed slot among the claimed ones
__global__ void __launch_bounds__(1024) k_class_number(ClassScratch* t, float4* geo, int* dj) {
  __shared__ int used[MAX_CLASSES];
  __shared__ int n;
  if (t->failed || t->count > MAX_CLASSES) return;
  if (threadIdx.x == 0) n = 0;
  __syncthreads();
  for (int q = threadIdx.x; q < CLASS_SLOTS; q += blockDim.x)
    if (t->fp[q]) used[atomicAdd(&n, 1)] = q;
  __syncthreads();
  for (int a = threadIdx.x; a < n; a += blockDim.x) {
    const ClassRec me = t->rec[used[a]];
    int rank = 0;
    for (int b = 0; b < n; b++) rank += class_less(t->rec[used[b]], me);
    t->id[used[a]] = rank;
    geo[rank] = make_float4(__uint_as_float(me.v[1]), __uint_as_float(me.v[2]),
                            __uint_as_float(me.v[3]), __uint_as_float(me.v[4]));
    dj[rank] = (int)me.v[0];
  }
}

__global__ void __launch_bounds__(256) k_class_write(DevBody d, ClassScratch* t, unsigned* cls) {
  const int lane = threadIdx.x & 31;
  const long long s = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (s >= d.nslices || t->failed) return;
  const long long i = s * 32 + lane;
  const long long sbase = d.soff[s];
  const int rows = (int)((d.soff[s + 1] - sbase) >> 5);
  const int cnt = i < d.n ? (int)(d.off[i + 1] - d.off[i]) : 0;
  unsigned* out = cls + class_word0(sbase, s) + lane;
  for (int r4 = 0; r4 < rows; r4 += 4) {
    unsigned w = 0;
    for (int u = 0; u < 4 && r4 + u < cnt; u++) {
      const ClassRec rec = class_record(d, sbase + 32LL * (r4 + u) + lane, i);
      const unsigned long long f = class_print(rec);
      int q = (int)(f % CLASS_SLOTS);
      bool found = false;
      for (int probe = 0; probe < CLASS_SLOTS; probe++) {
        if (t->fp[q] == f) { found = true; break; }
        if (t->fp[q] == 0) break;
        q = (q + 1) % CLASS_SLOTS;
      }
      const ClassRec have = t->rec[q];
      for (int k = 0; k < 5; k++) found = found && have.v[k] == rec.v[k];
      if (!found) { t->failed = 2; return; }
      w |= (unsigned)t->id[q] << (8 * u);
    }
    out[8 * r4] = w;
  }
}

cudaError_t build_classes(const DevBody& d, long long nslots, unsigned** cls, float4** geo, int** dj,
                          int* ncls, cudaStream_t s) {
  *cls = nullptr;
  *geo = nullptr;
  *dj = nullptr;
  *ncls = 0;
  if (d.n == 0 || d.nb == 0 || d.lg != 1 || d.geo == nullptr) return cudaSuccess;
  ClassScratch* t = nullptr;
  const unsigned grid = (unsigned)((d.nslices + 7) / 8);
  int found[2] = {0, 0};
  cudaError_t e = cudaMalloc(&t, sizeof(ClassScratch));
  if (e == cudaSuccess) e = cudaMemsetAsync(t, 0, sizeof(ClassScratch), s);
  if (e == cudaSuccess) {
    k_class_collect<<<grid, 256, 0, s>>>(d, t);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(found, &t->count, sizeof(found), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e == cudaSuccess && found[1] == 0 && found[0] > 0) {
    const size_t words = 32 * ((size_t)(nslots >> 7) + (size_t)d.nslices + 1);
    e = cudaMalloc(cls, sizeof(unsigned) * words);
    if (e == cudaSuccess) e = cudaMalloc(geo, sizeof(float4) * MAX_CLASSES);
    if (e == cudaSuccess) e = cudaMalloc(dj, sizeof(int) * MAX_CLASSES);
    if (e == cudaSuccess) {
      k_class_number<<<1, 1024, 0, s>>>(t, *geo, *dj);
      k_class_write<<<grid, 256, 0, s>>>(d, t, *cls);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(found, &t->count, sizeof(found), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess && found[1] == 0) *ncls = found[0];
  }
  cudaFree(t);
  if (e != cudaSuccess || *ncls == 0) {
    cudaFree(*cls);
    cudaFree(*geo);
    cudaFree(*dj);
    *cls = nullptr;
    *geo = nullptr;
    *dj = nullptr;
  }
  return e;
}

}  // namespace pd
