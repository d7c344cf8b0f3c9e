// pd_static.cu -- an ordinary state-based force evaluation that allocates no device memory.
//
// Some callers cannot allocate GPU memory at the moment they need forces: a Julia host that
// manages every device buffer through its own memory pool and forbids the library to call
// cudaMalloc (the reference asserts that its force loop allocates nothing, test/perf/perf.jl),
// a time loop that must not stall on the allocator, or an application that hands the library
// memory it carved out of a fixed arena. For them pd_osb_force_static takes every input and
// output as a device pointer owned by the caller and keeps its one piece of scratch state --
// the two force coefficients, the volume and the place of the bond list of every point, which the
// gather phase reads for the neighbours in one 32-byte record -- in the file-scope device array below. The array
// is part of the library image: every GPU that loads the library holds it until the process
// exits, which is why it is kept to PD_STATIC_MAX_POINTS points (8 MiB).
//
// The arithmetic is that of the FP64 kernels off the serial order (pd_bond64.cuh), on the reference's
// CSR bond arrays instead of the sliced layout.
#include <cuda.h>

#include <cfloat>
#include <mutex>
#include <string>
#include <vector>

#include "pdcuda.h"
#include "pd_bond64.cuh"
#include "pd_common.cuh"

namespace pd {

constexpr long long PD_STATIC_MAX_POINTS = 1LL << 18;

// What bounds it: the gathers of the neighbours' positions, which reach L1 as three 8-byte loads of
// records 24 bytes apart, and (phase B) the search for the reverse bond, which bounds jittered bodies.
// us a call, one thread a point before / now: 1,380 points 481 / 42, 30,659 655 / 150, 147,420 1296 / 730.

// {c1, c2, volume, place of the bond list} per point, shared by every call of pd_osb_force_static on this device
static __device__ __align__(256) double4 g_osb_state[PD_STATIC_MAX_POINTS];

struct StaticArgs {
  long long n;
  const double* X;    // [3n] reference positions
  const double* x;    // [3n] current positions
  const double* vol;  // [n]
  const long long* off;
  const int* nbr;
  const double* L;
  const unsigned char* fail_permit;
  unsigned char* bond_active;  // in / out
  double delta, G, K, epsc;
  int kernel;
  double* b_int;      // [3n] out
  long long* n_active; // [n] out
  double4* state;     // g_osb_state, through the address looked up on the host
};

// the end of a point's bond list (below 2^44) and its size (a point has at most 2^18 neighbours)
__device__ __forceinline__ double pack_list(long long b0, long long b1) {
  return __longlong_as_double((b1 << 19) | (b1 - b0));
}
__device__ __forceinline__ long long list_end(double w) { return __double_as_longlong(w) >> 19; }
__device__ __forceinline__ long long list_size(double w) { return __double_as_longlong(w) & ((1 << 19) - 1); }

__device__ __forceinline__ double s_omega(int kernel, double delta, double L) {
  if (kernel == KER_LINEAR) return delta / L;
  if (kernel == KER_CONST_ONE) return 1.0;
  const double xi = L / delta;
  if (0 < xi && xi <= 0.5) return 2.0 / 3.0 - 4 * (xi * xi) + 4 * (xi * xi * xi);
  if (0.5 < xi && xi <= 1) return 4.0 / 3.0 - 4 * xi + 4 * (xi * xi) - 4.0 / 3.0 * (xi * xi * xi);
  return 0.0;
}

// LN lanes share a point. Both phases read a point's bonds with consecutive lanes (the CSR arrays
// are then read in whole lines) and sum over the lanes in a fixed tree, so results do not depend on
// the schedule. One thread a point left 958 warps for the chip on a 30,659-point body, each with 122
// bonds in a row and every load of a bond in a line of its own.
template <int LN>
__device__ __forceinline__ double lane_sum(double v) {
#pragma unroll
  for (int o = LN / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// the place of a thread: its point, its lane of the point and whether the point exists; lanes of
// points beyond the last one run along with no bonds
template <int LN>
struct Place {
  long long i, b0, b1;
  int lane;
  bool valid;
  __device__ __forceinline__ Place(const StaticArgs& a) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    i = t / LN;
    lane = (int)(t % LN);
    valid = i < a.n;
    if (!valid) i = 0;
    b0 = a.off[i];
    b1 = valid ? a.off[i + 1] : b0;
  }
};

__device__ __forceinline__ void s_diff(const double* p, const double (&q)[3], long long j, double (&d)[3]) {
  d[0] = p[3 * j] - q[0];
  d[1] = p[3 * j + 1] - q[1];
  d[2] = p[3 * j + 2] - q[2];
}

// calc_failure! (ordinary_state_based.jl:107-126), calc_weighted_volume (:176-189),
// calc_dilatation (:191-204), c1 and c2 (:135-136): one pass over the bonds, the dilatation's factor
// 3 / m taken out of its sum
template <int LN>
__global__ void __launch_bounds__(256) k_static_osb_a(StaticArgs a) {
  const Place<LN> t(a);
  const long long i = t.i;
  const double xi[3] = {a.x[3 * i], a.x[3 * i + 1], a.x[3 * i + 2]};
  const double Xi[3] = {a.X[3 * i], a.X[3 * i + 1], a.X[3 * i + 2]};
  const double thr = fail_threshold(a.epsc);
  int na = 0;
  double m = 0.0, th = 0.0;
#pragma unroll 2
  for (long long b = t.b0 + t.lane; b < t.b1; b += LN) {
    const long long j = a.nbr[b];
    const double L = a.L[b];
    unsigned act = a.bond_active[b];
    double d[3], D[3];
    s_diff(a.x, xi, j, d);
    s_diff(a.X, Xi, j, D);
    const double l2 = (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2];
    // DBL_MIN: two points in one place have no reciprocal of the length, but a dilatation
    const double e = sqrt_of(l2, rsqrt3(l2 + DBL_MIN)) - L;
    if (!(L > 0 && e < thr * L) && (sqrt(l2) - L) / L > a.epsc && a.fail_permit[b]) {
      a.bond_active[b] = 0;
      act = 0;
    }
    na += (int)act;
    const double w = act ? s_omega(a.kernel, a.delta, L) * a.vol[j] : 0.0;
    m = fma(w, (D[0] * D[0] + D[1] * D[1]) + D[2] * D[2], m);
    th = fma(w * L, e, th);
  }
  m = lane_sum<LN>(m);
  th = lane_sum<LN>(th);
#pragma unroll
  for (int o = LN / 2; o > 0; o >>= 1) na += __shfl_xor_sync(0xffffffffu, na, o);
  if (!t.valid || t.lane) return;
  double c1 = 0.0, c2 = 0.0;
  if (m != 0.0) {
    c1 = 15.0 * a.G / m;
    c2 = 3.0 / m * th * (3.0 * a.K / m - c1 / 3.0);
  }
  a.state[i] = make_double4(c1, c2, a.vol[i], pack_list(t.b0, t.b1));
  a.n_active[i] = na;
}

// position of point i in the sorted bond list of point j at [lo, hi) (the reverse bond j -> i), or -1;
// k: the bond's place in the list of i. In a body whose points lie alike the reverse of a list's k-th
// bond is the k-th from the end of the other list: that place is tried first.
__device__ __forceinline__ long long s_reverse(const StaticArgs& a, long long lo, long long hi, long long i,
                                               long long k) {
  const long long end = hi, g = hi - 1 - k;
  if (g >= lo) {
    const int q = a.nbr[g];
    if (q == i) return g;
    if (q < i) lo = g + 1; else hi = g;
  }
  while (lo < hi) {
    const long long mid = (lo + hi) >> 1;
    if (a.nbr[mid] < i) lo = mid + 1; else hi = mid;
  }
  return (lo < end && a.nbr[lo] == i) ? lo : -1;
}

// force_density_point! (ordinary_state_based.jl:128-149), gathered: a bond's own term and the one
// that its neighbour's loop scatters into i (of the bond j -> i: its bond state and its length), so
// bond states need not be the same in both directions.
template <int LN>
__global__ void __launch_bounds__(256) k_static_osb_b(StaticArgs a) {
  const Place<LN> t(a);
  const long long i = t.i;
  const double4 ci = a.state[i];
  const double xi[3] = {a.x[3 * i], a.x[3 * i + 1], a.x[3 * i + 2]};
  const bool own = ci.x != 0.0 || ci.y != 0.0;
  double f[3] = {0.0, 0.0, 0.0};
#pragma unroll 2
  for (long long b = t.b0 + t.lane; b < t.b1; b += LN) {
    const long long j = a.nbr[b];
    const double L = a.L[b];
    const double4 cj = a.state[j];
    double d[3];
    s_diff(a.x, xi, j, d);
    const double l2 = (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2];
    const double rl = rsqrt3(l2), l = sqrt_of(l2, rl);
    const double om = s_omega(a.kernel, a.delta, L);
    double s = (a.bond_active[b] ? om : 0.0) * (ci.y * L + ci.x * (l - L));
    const long long end = list_end(cj.w), r = s_reverse(a, end - list_size(cj.w), end, i, b - t.b0);
    if (r >= 0) {  // else j scatters nothing into i
      const double Lr = a.L[r];
      const double omr = !a.bond_active[r] ? 0.0 : (Lr == L ? om : s_omega(a.kernel, a.delta, Lr));
      s += omr * (cj.y * Lr + cj.x * (l - Lr));
    }
    // neither point has bonds left: no force, whatever the bond's length
    if (!(own || (r >= 0 && (cj.x != 0.0 || cj.y != 0.0)))) continue;
    s *= rl * cj.z;
    f[0] = fma(s, d[0], f[0]);
    f[1] = fma(s, d[1], f[1]);
    f[2] = fma(s, d[2], f[2]);
  }
#pragma unroll
  for (int c = 0; c < 3; c++) f[c] = lane_sum<LN>(f[c]);
  if (!t.valid || t.lane) return;
  a.b_int[3 * i] = f[0];
  a.b_int[3 * i + 1] = f[1];
  a.b_int[3 * i + 2] = f[2];
}

}  // namespace pd

using namespace pd;

template <int LN>
static void launch_static(const StaticArgs& a, cudaStream_t s) {
  const int blocks = (int)((a.n * LN + 255) / 256);
  k_static_osb_a<LN><<<blocks, 256, 0, s>>>(a);
  k_static_osb_b<LN><<<blocks, 256, 0, s>>>(a);
}

static thread_local std::string g_static_err;

// Device address of g_osb_state in each CUDA context that called, looked up once per context
// with it current. The context is read through the driver's cuCtxGetCurrent (taken from the
// runtime's driver entry points, so the library needs no link to libcuda); where that is not
// available the key is the device's primary context, identified by the device index.
struct StaticSlot {
  CUcontext ctx;
  int dev;
  void* ptr;
};
static std::mutex g_static_mutex;
static std::vector<StaticSlot> g_static_slots;
typedef CUresult (*CtxGetCurrentFn)(CUcontext*);

static CtxGetCurrentFn ctx_get_current() {
  static CtxGetCurrentFn fn = nullptr;
  static bool looked = false;
  if (!looked) {
    looked = true;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (CtxGetCurrentFn)p;
  }
  return fn;
}

extern "C" const char* pd_static_last_error(void) { return g_static_err.c_str(); }

extern "C" pd_status pd_osb_force_static(int64_t n, const double* ref_position, const double* position,
                                         const double* volume, const int64_t* bond_offsets,
                                         const int32_t* neighbors, const double* bond_length,
                                         const uint8_t* fail_permit, uint8_t* bond_active,
                                         const pd_point_params* params, int32_t kernel,
                                         double* b_int, int64_t* n_active, void* stream) {
  if (n < 0 || !params) { g_static_err = "n < 0 or params is NULL"; return PD_ERR_ARG; }
  if (n > PD_STATIC_MAX_POINTS) {
    g_static_err = "pd_osb_force_static handles at most " + std::to_string(PD_STATIC_MAX_POINTS) +
                   " points (the size of its static scratch array); got " + std::to_string(n);
    return PD_ERR_ARG;
  }
  if (kernel < PD_KERNEL_CONST_ONE || kernel > PD_KERNEL_CUBIC_BSPLINE) {
    g_static_err = "unknown kernel";
    return PD_ERR_ARG;
  }
  if (n == 0) return PD_OK;
  if (!ref_position || !position || !volume || !bond_offsets || !neighbors || !bond_length ||
      !fail_permit || !bond_active || !b_int || !n_active) {
    g_static_err = "every array must be a device pointer";
    return PD_ERR_ARG;
  }
  // an error left by earlier CUDA work of this thread would be reported as this call's after
  // the launches: report it now, launch nothing, and leave it pending for its owner
  cudaError_t e = cudaPeekAtLastError();
  if (e != cudaSuccess) {
    g_static_err = std::string("a CUDA error from before this call is pending (") +
                   cudaGetErrorString(e) + "); no kernel was launched";
    return PD_ERR_CUDA;
  }
  int dev = 0;
  e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    g_static_err = std::string("cudaGetDevice: ") + cudaGetErrorString(e);
    return PD_ERR_CUDA;
  }
  CUcontext ctx = nullptr;
  if (CtxGetCurrentFn get = ctx_get_current()) {
    if (get(&ctx) != CUDA_SUCCESS) ctx = nullptr;
  }
  void* state = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_static_mutex);
    for (const StaticSlot& sl : g_static_slots)
      if (sl.dev == dev && sl.ctx == ctx) { state = sl.ptr; break; }
    if (!state) {
      // set-up in this context (the current one): the host-side name of the array is not a
      // device address, so its device address is looked up once
      e = cudaGetSymbolAddress(&state, g_osb_state);
      if (e != cudaSuccess) {
        g_static_err = std::string("cudaGetSymbolAddress of the scratch array on device ") +
                       std::to_string(dev) + ": " + cudaGetErrorString(e);
        return PD_ERR_CUDA;
      }
      if (ctx == nullptr && ctx_get_current() != nullptr) {
        // cudaGetSymbolAddress made the primary context current
        CUcontext now = nullptr;
        if (ctx_get_current()(&now) == CUDA_SUCCESS) ctx = now;
      }
      g_static_slots.push_back({ctx, dev, state});
    }
  }
  StaticArgs a;
  a.n = n;
  a.X = ref_position;
  a.x = position;
  a.vol = volume;
  a.off = reinterpret_cast<const long long*>(bond_offsets);
  a.nbr = neighbors;
  a.L = bond_length;
  a.fail_permit = fail_permit;
  a.bond_active = bond_active;
  a.delta = params->delta;
  a.G = params->G;
  a.K = params->K;
  a.epsc = params->epsilon_c;
  a.kernel = kernel;
  a.b_int = b_int;
  a.n_active = reinterpret_cast<long long*>(n_active);
  a.state = (double4*)state;
  cudaStream_t s = (cudaStream_t)stream;
  // Small bodies want a point's bonds spread over many lanes, large ones few idle lanes and short sums
  // over lanes. us a call with 32 / 16 / 8 lanes: 1,380 points 42 / 50 / 70, 4,095 44 / 54 / 76, 9,768
  // 76 / 75 / 84, 30,659 168 / 150 / 158, 47,196 294 / 243 / 233, 147,420 1000 / 815 / 730
  if (n <= (1 << 13)) launch_static<32>(a, s);
  else if (n <= 5 * (1 << 13)) launch_static<16>(a, s);
  else launch_static<8>(a, s);
  e = cudaGetLastError();
  if (e != cudaSuccess) {
    g_static_err = std::string("kernel launch: ") + cudaGetErrorString(e);
    return PD_ERR_CUDA;
  }
  return PD_OK;
}
