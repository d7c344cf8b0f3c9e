// pd_stream32.cuh -- the bond stream of the packed FP32 kernels (one lane per point), two rows at
// a time and one row pair ahead: neighbour, reference vector and length, state word.
//
// CLS = false: 20 bytes a bond from the sliced arrays (nbr, geo). CLS = true: bodies whose bonds
// fall into at most 256 classes of equal (j - i, reference vector, +-length), the bodies on a
// regular lattice, store one byte a bond; the classes (20 bytes each) are kept in shared memory.
// The values are the same bits either way.
#pragma once
#include "pd_common.cuh"
#include "pd_pack.cuh"

namespace pd {

constexpr int MAX_CLASSES = 256;

// first word of slice s in the class stream: word w of a slice holds the classes of its rows 4w ..
// 4w + 3 (one byte each, row 4w lowest) of 32 lanes; R = rows of the slices before it. Slices of r
// rows take (r + 3) / 4 words a lane, which floor(R / 4) + s leaves room for.
__device__ __forceinline__ long long class_word0(long long sbase, long long s) {
  return 32 * ((sbase >> 7) + s);
}

struct ClassTable {
  float4 geo[MAX_CLASSES];
  int dj[MAX_CLASSES];
};

// the table into shared memory (all threads of the block); the block leaves together when an
// earlier kernel recorded an error
template <bool CLS>
__device__ __forceinline__ bool stream_begin(const DevBody& d, ClassTable* t) {
  const int err = *(volatile const int*)&d.ctrl->err;
  if constexpr (CLS) {
    for (int k = threadIdx.x; k < d.ncls; k += blockDim.x) {
      t->geo[k] = d.cls_geo[k];
      t->dj[k] = d.cls_dj[k];
    }
    return __syncthreads_or(err) == 0;
  } else {
    return err == 0;
  }
}

// OWNED: the kernel rewrites its state words, which are therefore loaded plainly
template <bool CLS, bool OWNED>
struct Stream32 {
  const ClassTable* tab;
  const unsigned* pw;
  const int* pn;
  const float4* pg;
  const unsigned* pc;
  int rows, lane, self;
  unsigned nw0, nw1;
  int nj0, nj1;      // CLS: the class words of this and of the next four rows
  float4 ng0, ng1;

  __device__ __forceinline__ Stream32(const DevBody& d, const ClassTable* t, long long s,
                                      long long sbase, int rows_, int lane_, int self_)
      : tab(t), pw(d.bits + (sbase >> 5)), rows(rows_), lane(lane_), self(self_) {
    if constexpr (CLS) {
      pc = d.cls + class_word0(sbase, s) + lane;
    } else {
      pn = d.nbr + sbase + lane;
      pg = d.geo + sbase + lane;
    }
    nj0 = nj1 = CLS ? 0 : self;
    if constexpr (!CLS) ng0 = ng1 = make_float4(0.f, 0.f, 0.f, 1.f);
    nw0 = nw1 = 0u;
    if (rows > 0) {
      if constexpr (CLS) nj1 = (int)pack::ld_stream(pc);
      load(0);
    }
  }

  // the records of rows r (even) and r + 1
  __device__ __forceinline__ void load(int r) {
    const bool two = r + 1 < rows;
    if constexpr (OWNED) {
      nw0 = pw[r];
      nw1 = two ? pw[r + 1] : 0u;
    } else {
      nw0 = pack::ld_stream(pw + r);
      nw1 = two ? pack::ld_stream(pw + r + 1) : 0u;
    }
    if constexpr (CLS) {
      if ((r & 2) == 0) {
        nj0 = nj1;
        if (r + 4 < rows) nj1 = (int)pack::ld_stream(pc + 8 * (r + 4));
      }
    } else {
      nj0 = pack::ld_stream(pn + 32 * r);
      ng0 = pack::ld_stream(pg + 32 * r);
      if (two) { nj1 = pack::ld_stream(pn + 32 * r + 32); ng1 = pack::ld_stream(pg + 32 * r + 32); }
      else { nj1 = self; ng1 = make_float4(0.f, 0.f, 0.f, 1.f); }
    }
  }

  // the records loaded by load(r): states, neighbours (the point itself where the bond is not
  // active) and reference vectors
  __device__ __forceinline__ void take(int r, unsigned& w0, unsigned& w1, bool& a0, bool& a1, int& j0,
                                       int& j1, float4& g0, float4& g1) const {
    w0 = nw0;
    w1 = nw1;
    a0 = (w0 >> lane) & 1u;
    a1 = (w1 >> lane) & 1u;
    if constexpr (CLS) {
      const unsigned c = (unsigned)nj0 >> ((r & 2) << 3);
      const int c0 = c & 255u, c1 = (c >> 8) & 255u;
      j0 = a0 ? self + tab->dj[c0] : self;
      j1 = a1 ? self + tab->dj[c1] : self;
      g0 = tab->geo[c0];
      g1 = tab->geo[c1];
    } else {
      j0 = a0 ? nj0 : self;
      j1 = a1 ? nj1 : self;
      g0 = ng0;
      g1 = ng1;
    }
  }
};

}  // namespace pd
