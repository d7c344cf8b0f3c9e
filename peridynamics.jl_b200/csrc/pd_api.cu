// pd_api.cu -- C ABI of libpdcuda: handle lifecycle, uploads, boundary conditions, the
// Velocity Verlet step loop (eager or CUDA-graph captured), exports and the autotuner.
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstring>
#include <string>
#include <vector>

#include "pdcuda.h"
#include "pd_common.cuh"
#include "pd_launch.h"
#include "pd_bonds.h"
#include "pd_handle.h"

using namespace pd;

static thread_local std::string g_err;

pd_status pd_fail(pd_status code, const std::string& msg) {
  g_err = msg;
  return code;
}
static inline pd_status fail(pd_status code, const std::string& msg) { return pd_fail(code, msg); }

static pd_status set_ctrl(pd_handle* h, size_t off, const void* src, size_t bytes) {
  PD_CUDA(cudaMemcpyAsync(reinterpret_cast<char*>(h->d.ctrl) + off, src, bytes,
                          cudaMemcpyHostToDevice, h->stream));
  return PD_OK;
}

// Copies between host and device ordered on the stream `s` and complete on return. The
// handles' streams are non-blocking: a plain cudaMemcpy from pageable memory may return before
// its DMA has landed, and nothing orders a kernel on such a stream after it.
static cudaError_t h2d(void* dst, const void* src, size_t bytes, cudaStream_t s) {
  if (bytes == 0) return cudaSuccess;
  cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s);
  return e != cudaSuccess ? e : cudaStreamSynchronize(s);
}
static cudaError_t d2h(void* dst, const void* src, size_t bytes, cudaStream_t s) {
  if (bytes == 0) return cudaSuccess;
  cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s);
  return e != cudaSuccess ? e : cudaStreamSynchronize(s);
}

static pd_status upload_meta(pd_handle* h) {
  PD_CUDA(cudaMemcpyAsync(h->d.meta, h->hmeta.data(), sizeof(unsigned) * h->n,
                          cudaMemcpyHostToDevice, h->stream));
  return PD_OK;
}

static pd_status upload_params(pd_handle* h) {
  PD_CUDA(cudaMemcpyAsync(h->dparams, h->hp.data(), sizeof(DevParam) * h->hp.size(),
                          cudaMemcpyHostToDevice, h->stream));
  PD_CUDA(cudaStreamSynchronize(h->stream));
  return PD_OK;
}

static void destroy_graph(pd_handle* h) {
  if (h->gexec) cudaGraphExecDestroy(h->gexec);
  h->gexec = nullptr;
  h->gkey = GraphKey();
}

// Other kernels than before: weighted volumes and shape tensors stored by one kind of FP32 kernels carry its
// roundings (a body tuned on the staged variants and left on the packed ones: velocity error after 200 steps of
// a 1M-point pulse 1.5e-6, 4.1e-7 with its own)
static void sum_anew(pd_handle* h) { h->kfull = true; }

// what a captured step holds (bond arrays, bond-state mode, parameters) changed: the handle's graph
// goes, and the graphs of the groups that the handle belongs to no longer match its version
static void drop_graphs(pd_handle* h) {
  destroy_graph(h);
  h->version++;
}

extern "C" const char* pd_last_error(void) { return g_err.c_str(); }
extern "C" const char* pd_version(void) { return "0.1.0"; }

static DevParam make_param(const pd_point_params& p, double cs) {
  DevParam q{};
  q.delta = p.delta; q.rho = p.rho; q.bc = p.bc; q.epsc = p.epsilon_c; q.G = p.G; q.K = p.K;
  q.lambda = p.lambda; q.mu = p.mu;
  q.beta = cs * p.bc / p.delta;
  q.zwa = (1 - p.nu) * p.lambda / p.nu;  // get_hooke_matrix_voigt, constitutive_models.jl:107-118
  q.dt = 0; q.dth = 0;
  q.deltaf = (float)p.delta; q.bcf = (float)p.bc; q.epscf = (float)p.epsilon_c;
  q.Gf = (float)p.G; q.Kf = (float)p.K; q.lambdaf = (float)p.lambda; q.muf = (float)p.mu;
  q.betaf = (float)q.beta;
  q.zwaf = (float)q.zwa;
  q.inv_delta = (float)(1.0 / p.delta);
  q.vscale = (float)(1.0 / (p.delta * p.delta * p.delta));
  return q;
}

static pd_status validate_desc(const pd_body_desc* desc, bool need_bonds) {
  if (!desc) return fail(PD_ERR_ARG, "desc is NULL");
  if (desc->n_points < 0) return fail(PD_ERR_ARG, "n_points < 0");
  if (desc->n_points > 0x7fffffffLL) return fail(PD_ERR_ARG, "n_points exceeds 2^31 - 1");
  if (desc->n_points > 0 && (!desc->position || !desc->volume))
    return fail(PD_ERR_ARG, "position and volume are required");
  if (desc->n_params < 1 || desc->n_params > 65535 || !desc->params)
    return fail(PD_ERR_ARG, "1 <= n_params <= 65535 parameter sets are required");
  if (desc->material < PD_MAT_BB || desc->material > PD_MAT_CMAT)
    return fail(PD_ERR_ARG, "unknown material");
  if (desc->precision != PD_PREC_FP64 && desc->precision != PD_PREC_FP32_KAHAN)
    return fail(PD_ERR_ARG, "unknown precision");
  if (desc->kernel < PD_KERNEL_CONST_ONE || desc->kernel > PD_KERNEL_CUBIC_BSPLINE)
    return fail(PD_ERR_ARG, "unknown kernel");
  if (desc->material == PD_MAT_CMAT && desc->zem != PD_ZEM_SILLING && desc->zem != PD_ZEM_WAN)
    return fail(PD_ERR_ARG, "unknown zero-energy mode stabilisation");
  if (desc->cmodel < PD_CM_SVK || desc->cmodel > PD_CM_NEOHOOKE_PENALTY)
    return fail(PD_ERR_ARG, "unknown constitutive model");
  for (int k = 0; k < desc->n_params; k++) {
    const pd_point_params& p = desc->params[k];
    if (!(p.delta > 0)) return fail(PD_ERR_ARG, "`horizon` should be larger than zero!");
    if (!(p.rho > 0)) return fail(PD_ERR_ARG, "`rho` should be larger than zero!");
  }
  const long long n = desc->n_points;
  if (desc->param_id)
    for (long long i = 0; i < n; i++)
      if (desc->param_id[i] >= desc->n_params) return fail(PD_ERR_ARG, "param_id out of range");
  for (long long i = 0; i < n; i++)
    if (!(desc->volume[i] > 0) && desc->volume[i] != 0)
      return fail(PD_ERR_ARG, "volume must be finite and >= 0");
  if (need_bonds) {
    if (desc->n_bonds < 0) return fail(PD_ERR_ARG, "n_bonds < 0");
    if (desc->n_bonds > 0x7fffffffLL) return fail(PD_ERR_ARG, "n_bonds exceeds 2^31 - 1");
    if (!desc->bond_offsets) return fail(PD_ERR_ARG, "bond_offsets is NULL");
    if (desc->n_bonds > 0 && !desc->neighbors) return fail(PD_ERR_ARG, "neighbors is NULL");
    if (desc->bond_offsets[0] != 0 || desc->bond_offsets[n] != desc->n_bonds)
      return fail(PD_ERR_ARG, "bond_offsets must start at 0 and end at n_bonds");
    for (long long i = 0; i < n; i++)
      if (desc->bond_offsets[i + 1] < desc->bond_offsets[i])
        return fail(PD_ERR_ARG, "bond_offsets must be non-decreasing");
    for (long long b = 0; b < desc->n_bonds; b++)
      if (desc->neighbors[b] < 0 || desc->neighbors[b] >= n)
        return fail(PD_ERR_ARG, "neighbor index out of range");
  }
  return PD_OK;
}

// symmetric-pair mode of the state-based materials: every bond has a reverse, both directions
// share one state and one critical stretch. Otherwise the kernels read the reverse bond.
static pd_status check_symmetry(pd_handle* h) {
  if (h->material == PD_MAT_BB || h->nb == 0 || !h->d.rev) { h->d.sym = 1; return PD_OK; }
  int hf[4] = {0, 0, 0, 0};
  PD_CUDA(cudaMemsetAsync(h->flags, 0, sizeof(int) * 4, h->stream));
  launch_check_sym(h->d, h->flags, h->stream);
  PD_CUDA(cudaMemcpyAsync(hf, h->flags, sizeof(hf), cudaMemcpyDeviceToHost, h->stream));
  PD_CUDA(cudaStreamSynchronize(h->stream));
  h->d.sym = (hf[1] == 0 && hf[2] == 0) ? 1 : 0;
  return PD_OK;
}

// Whether the points of the one-lane layout take places that suit tiles (pd_tiles.cu). The kernels that
// know no tiles are slower in that order (us a step, places / the points' own order, OSB 192,000 points: two
// parameter sets 651 / 547, the staged stream of variant 2 510 / 457, surface correction 426 / 359). ZEMWan
// and directed bond states have their first phase on tiles and are not (variant 0, 192,000 points, against
// the one-row kernels on the points' own order: 417 / 466 and 446 / 466).
static bool wants_places(const pd_handle* h) {
  if (h->multi || h->d.sc32 || h->d.sc64 || h->esc) return false;
  if (h->cfg.pipe >= 1 && h->cfg.pipe <= 3) return false;
  return h->precision != PD_PREC_FP64 || h->material != PD_MAT_CMAT;
}

// Bodies with one lane per point gather from tiles in shared memory (FP64: BB and OSB) and, in FP32
// on a regular lattice, read a bond's geometry as one byte. Both are made once per layout; a body without tiles,
// or without the memory for them, gathers from global memory, one without classes reads 16 bytes.
static pd_status ensure_tiles(pd_handle* h) {
  if (h->tiles_tried || h->d.lg != 1 || h->d.pt == nullptr || h->multi)
    return PD_OK;
  h->tiles_tried = true;
  TileArrays t;
  cudaError_t e = build_tiles(h->d, h->nslots, &t, h->stream);
  if (e != cudaErrorMemoryAllocation) PD_CUDA(e);
  else cudaGetLastError();
  if (t.pt == nullptr) return PD_OK;
  for (void* p : {(void*)t.pt, (void*)t.n, (void*)t.lidx, (void*)t.lown}) h->allocs.push_back(p);
  h->d.tile_pt = t.pt;
  h->d.tile_n = t.n;
  h->d.lidx = t.lidx;
  h->d.lown = t.lown;
  h->d.tile_cap = t.cap;
  if (h->precision == PD_PREC_FP64) return PD_OK;
  unsigned* cls = nullptr;
  float4* geo = nullptr;
  int ncls = 0;
  e = build_classes(h->d, h->nslots, &cls, &geo, &ncls, h->stream);
  if (e != cudaErrorMemoryAllocation) PD_CUDA(e);
  else cudaGetLastError();
  if (ncls == 0) return PD_OK;
  h->allocs.push_back(cls);
  h->allocs.push_back(geo);
  h->d.cls = cls;
  h->d.cls_geo = geo;
  h->d.ncls = ncls;
  return PD_OK;
}

// CSR bond lists (device) -> sliced layout with one lane per point, bond geometry, reverse
// positions, all bonds active; then the point state.
static pd_status finish_create(pd_handle* h, int* dnbr_csr, const double* dL, const unsigned char* dfp) {
  const long long n = h->n, nb = h->nb;
  int* revk_csr = nullptr;
  if (h->material != PD_MAT_BB && nb > 0) {
    int hf = 0;
    PD_TRY(dalloc(h, &revk_csr, nb));
    PD_CUDA(cudaMemsetAsync(h->flags, 0, sizeof(int) * 4, h->stream));
    launch_reverse(n, h->d.off, dnbr_csr, revk_csr, h->flags, h->stream);
    PD_CUDA(cudaMemcpyAsync(&hf, h->flags, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    PD_CUDA(cudaStreamSynchronize(h->stream));
    if (hf)
      return fail(PD_ERR_UNSUPPORTED,
                  "bond lists are not symmetric (a bond i->j without j->i): the gather form of the "
                  "state-based materials needs symmetric bond lists (equal horizons)");
  }
  long long* soff = nullptr;
  long long ns = 0, nslots = 0;
  if (wants_places(h)) {
    PD_CUDA(build_places(h->d, h->grid, &h->pt, &h->place, h->stream));
    h->allocs.push_back(h->pt);
    h->allocs.push_back(h->place);
    h->d.pt = h->pt;
    h->d.place = h->place;
  }
  PD_CUDA(build_slices(n, h->d.off, h->d.pt, 1, &soff, &ns, &nslots, h->stream));
  h->allocs.push_back(soff);
  h->d.soff = soff;
  h->d.nslices = ns;
  h->d.lg = 1;
  h->nslots = nslots;
  int* nbr = nullptr;
  PD_TRY(dalloc(h, &nbr, nslots));
  PD_CUDA(cudaMemsetAsync(nbr, 0, sizeof(int) * (nslots > 0 ? nslots : 1), h->stream));
  if (nb) launch_scatter_i32(h->d, dnbr_csr, nbr, h->stream);
  h->d.nbr = nbr;
  if (revk_csr) {
    int* rev = nullptr;
    PD_TRY(dalloc(h, &rev, nslots));
    PD_CUDA(cudaMemsetAsync(rev, 0, sizeof(int) * nslots, h->stream));
    launch_scatter_i32(h->d, revk_csr, rev, h->stream);
    h->d.rev = rev;
  }
  if (h->precision == PD_PREC_FP64) {
    double* len = nullptr;
    PD_TRY(dalloc(h, &len, nslots));
    PD_CUDA(cudaMemsetAsync(len, 0, sizeof(double) * (nslots > 0 ? nslots : 1), h->stream));
    if (nb) launch_build_len64(h->d, dnbr_csr, dL, dfp, len, h->stream);
    h->d.len64 = len;
  } else {
    float4* geo = nullptr;
    PD_TRY(dalloc(h, &geo, nslots));
    PD_CUDA(cudaMemsetAsync(geo, 0, sizeof(float4) * (nslots > 0 ? nslots : 1), h->stream));
    if (nb) launch_build_geo(h->d, dnbr_csr, dL, dfp, geo, h->stream);
    h->d.geo = geo;
  }
  unsigned* bits = nullptr;
  PD_TRY(dalloc(h, &bits, nslots / 32 + 1));
  PD_CUDA(cudaMemsetAsync(bits, 0, sizeof(unsigned) * (nslots / 32 + 1), h->stream));
  h->d.bits = bits;
  launch_pack_bits(h->d, nullptr, h->stream);
  PD_CUDA(cudaGetLastError());
  PD_CUDA(cudaStreamSynchronize(h->stream));
  if (revk_csr) dfree(h, revk_csr);
  // point state
  PD_TRY(dalloc(h, &h->d.n_active, n));
  PD_TRY(dalloc(h, &h->g.vh, 3 * n));
  PD_TRY(dalloc(h, &h->g.v, 3 * n));
  PD_TRY(dalloc(h, &h->g.a, 3 * n));
  PD_TRY(dalloc(h, &h->g.bext, 3 * n));
  PD_CUDA(cudaMemsetAsync(h->g.vh, 0, sizeof(double) * 3 * n, h->stream));
  PD_CUDA(cudaMemsetAsync(h->g.v, 0, sizeof(double) * 3 * n, h->stream));
  PD_CUDA(cudaMemsetAsync(h->g.a, 0, sizeof(double) * 3 * n, h->stream));
  PD_CUDA(cudaMemsetAsync(h->g.bext, 0, sizeof(double) * 3 * n, h->stream));
  if (h->precision == PD_PREC_FP64) {
    PD_TRY(dalloc(h, &h->g.u, 3 * n));
    PD_TRY(dalloc(h, &h->d.b64, 3 * n));
    PD_CUDA(cudaMemsetAsync(h->g.u, 0, sizeof(double) * 3 * n, h->stream));
    PD_CUDA(cudaMemsetAsync(h->d.b64, 0, sizeof(double) * 3 * n, h->stream));
    h->g.fp32 = 0;
  } else {
    PD_TRY(dalloc(h, &h->d.b32, 3 * n));
    PD_CUDA(cudaMemsetAsync(h->d.b32, 0, sizeof(float) * 3 * n, h->stream));
    PD_TRY(dalloc(h, &h->d.uhi, n));
    PD_TRY(dalloc(h, &h->d.ulo, n));
    h->g.fp32 = 1;
    launch_split_u(h->d, h->stream);
  }
  if (h->material == PD_MAT_OSB) {
    if (h->precision == PD_PREC_FP64) {
      PD_TRY(dalloc(h, &h->d.coef64, n));
      PD_CUDA(cudaMemsetAsync(h->d.coef64, 0, sizeof(double4) * n, h->stream));
    } else {
      PD_TRY(dalloc(h, &h->d.cc32, n));
      PD_TRY(dalloc(h, &h->d.cm32, n));
      PD_TRY(dalloc(h, &h->d.mlo32, n));
      PD_CUDA(cudaMemsetAsync(h->d.mlo32, 0, sizeof(float) * n, h->stream));
      PD_CUDA(cudaMemsetAsync(h->d.cc32, 0, sizeof(float2) * n, h->stream));
      PD_CUDA(cudaMemsetAsync(h->d.cm32, 0, sizeof(float2) * n, h->stream));
    }
  } else if (h->material == PD_MAT_CMAT) {
    if (h->precision == PD_PREC_FP64) {
      PD_TRY(dalloc(h, &h->d.F64, 9 * n));
      PD_TRY(dalloc(h, &h->d.PK64, 9 * n));
      PD_CUDA(cudaMemsetAsync(h->d.F64, 0, sizeof(double) * 9 * n, h->stream));
      PD_CUDA(cudaMemsetAsync(h->d.PK64, 0, sizeof(double) * 9 * n, h->stream));
      if (h->zem == PD_ZEM_WAN) {
        PD_TRY(dalloc(h, &h->d.C164, 9 * n));
        PD_CUDA(cudaMemsetAsync(h->d.C164, 0, sizeof(double) * 9 * n, h->stream));
      }
      const long long planes = h->zem == PD_ZEM_WAN ? 8 : 5;
      PD_TRY(dalloc(h, &h->d.cst64, planes * n));
      PD_CUDA(cudaMemsetAsync(h->d.cst64, 0, sizeof(double2) * planes * n, h->stream));
    } else {
      PD_TRY(dalloc(h, &h->d.H32, 9 * n));
      PD_TRY(dalloc(h, &h->d.cst32, 3 * n));
      PD_TRY(dalloc(h, &h->d.K32, 6 * n));
      PD_CUDA(cudaMemsetAsync(h->d.H32, 0, sizeof(float) * 9 * n, h->stream));
      PD_CUDA(cudaMemsetAsync(h->d.cst32, 0, sizeof(float4) * 3 * n, h->stream));
      PD_CUDA(cudaMemsetAsync(h->d.K32, 0, sizeof(float) * 6 * n, h->stream));
      if (h->zem == PD_ZEM_WAN) {
        PD_TRY(dalloc(h, &h->d.zw32, 2 * n));
        PD_CUDA(cudaMemsetAsync(h->d.zw32, 0, sizeof(float4) * 2 * n, h->stream));
      }
    }
  }
  launch_count_active(h->d, h->stream);
  PD_CUDA(cudaGetLastError());
  PD_TRY(check_symmetry(h));
  PD_TRY(ensure_tiles(h));
  PD_CUDA(cudaStreamSynchronize(h->stream));
  return PD_OK;
}

// every bond array in the layout with G lanes per point, places: in the order of the tiles
static pd_status move_bonds(pd_handle* h, int G, bool places) {
  PD_CUDA(cudaStreamSynchronize(h->stream));
  DevBody a = h->d, b = h->d;
  long long* soff = nullptr;
  long long ns = 0, nslots = 0;
  b.pt = places ? h->pt : nullptr;
  b.place = places ? h->place : nullptr;
  PD_CUDA(build_slices(h->n, h->d.off, b.pt, G, &soff, &ns, &nslots, h->stream));
  h->allocs.push_back(soff);
  b.soff = soff;
  b.nslices = ns;
  b.lg = G;
  int* nbr = nullptr;
  PD_TRY(dalloc(h, &nbr, nslots));
  PD_CUDA(cudaMemsetAsync(nbr, 0, sizeof(int) * (nslots > 0 ? nslots : 1), h->stream));
  launch_relayout_i32(a, b, a.nbr, nbr, h->stream);
  b.nbr = nbr;
  if (a.rev) {
    int* rev = nullptr;
    PD_TRY(dalloc(h, &rev, nslots));
    PD_CUDA(cudaMemsetAsync(rev, 0, sizeof(int) * (nslots > 0 ? nslots : 1), h->stream));
    launch_relayout_i32(a, b, a.rev, rev, h->stream);
    b.rev = rev;
  }
  if (a.len64) {
    double* len = nullptr;
    PD_TRY(dalloc(h, &len, nslots));
    PD_CUDA(cudaMemsetAsync(len, 0, sizeof(double) * (nslots > 0 ? nslots : 1), h->stream));
    launch_relayout_f64(a, b, a.len64, len, h->stream);
    b.len64 = len;
  } else {
    float4* geo = nullptr;
    PD_TRY(dalloc(h, &geo, nslots));
    PD_CUDA(cudaMemsetAsync(geo, 0, sizeof(float4) * (nslots > 0 ? nslots : 1), h->stream));
    launch_relayout_f4(a, b, a.geo, geo, h->stream);
    b.geo = geo;
  }
  if (a.sc64) {  // surface correction factors follow the bond slots
    double* sc = nullptr;
    PD_TRY(dalloc(h, &sc, nslots));
    PD_CUDA(cudaMemsetAsync(sc, 0, sizeof(double) * (nslots > 0 ? nslots : 1), h->stream));
    launch_relayout_f64(a, b, a.sc64, sc, h->stream);
    b.sc64 = sc;
  }
  if (a.sc32) {
    float* sc = nullptr;
    PD_TRY(dalloc(h, &sc, nslots));
    PD_CUDA(cudaMemsetAsync(sc, 0, sizeof(float) * (nslots > 0 ? nslots : 1), h->stream));
    launch_relayout_i32(a, b, reinterpret_cast<const int*>(a.sc32), reinterpret_cast<int*>(sc), h->stream);
    b.sc32 = sc;
  }
  unsigned* bits = nullptr;
  unsigned char* bytes = nullptr;
  PD_TRY(dalloc(h, &bits, nslots / 32 + 1));
  PD_CUDA(cudaMemsetAsync(bits, 0, sizeof(unsigned) * (nslots / 32 + 1), h->stream));
  PD_TRY(dalloc(h, &bytes, h->nb));
  launch_export_bond_active(a, bytes, 1, h->stream);
  b.bits = bits;
  launch_pack_bits(b, bytes, h->stream);
  PD_CUDA(cudaGetLastError());
  PD_CUDA(cudaStreamSynchronize(h->stream));
  dfree(h, bytes);
  dfree(h, (void*)a.soff); dfree(h, (void*)a.nbr); dfree(h, (void*)a.rev);
  dfree(h, (void*)a.len64); dfree(h, (void*)a.geo); dfree(h, a.bits);
  dfree(h, (void*)a.sc64); dfree(h, (void*)a.sc32);
  for (const void* p : {(const void*)a.tile_pt, (const void*)a.tile_n, (const void*)a.lidx,
                        (const void*)a.lown, (const void*)a.cls, (const void*)a.cls_geo})
    dfree(h, const_cast<void*>(p));
  b.tile_pt = nullptr;
  b.tile_n = nullptr;
  b.lidx = nullptr;
  b.lown = nullptr;
  b.cls = nullptr;
  b.cls_geo = nullptr;
  b.ncls = 0;
  h->tiles_tried = false;
  h->d = b;
  h->nslots = nslots;
  return PD_OK;
}

// the layout with G lanes per point, one lane in the order that the handle's kernels want. On failure, for want
// of memory among others, the body keeps its layout and what was allocated for the other is given back
static pd_status relayout(pd_handle* h, int G) {
  const bool places = G == 1 && wants_places(h) && h->pt != nullptr;
  if (G == h->d.lg && places == (h->d.pt != nullptr)) return PD_OK;
  const size_t kept = h->allocs.size();
  const pd_status st = move_bonds(h, G, places);
  if (st != PD_OK) {
    cudaStreamSynchronize(h->stream);
    while (h->allocs.size() > kept) {
      cudaFree(h->allocs.back());
      h->allocs.pop_back();
    }
    cudaGetLastError();  // the caller has st; the next check of a launch is not to find it
    return st;
  }
  drop_graphs(h);
  return ensure_tiles(h);
}

// The lattice that the places of the points are laid out on: the bounding box's corner, the spacing
// that the mean volume implies, and first the axis on which consecutive points lie (of the first
// few thousand). Only the speed of the kernels depends on how well it fits the body.
static PlaceGrid place_grid(long long n, const double* X, const double* V) {
  PlaceGrid g{};
  double vol = 0;
  int steps[3] = {0, 0, 0};
  for (int a = 0; a < 3; a++) { g.lo[a] = n > 0 ? X[a] : 0.0; g.axis[a] = a; }
  for (long long i = 0; i < n; i++) {
    for (int a = 0; a < 3; a++) g.lo[a] = std::min(g.lo[a], X[3 * i + a]);
    vol += V[i];
  }
  for (long long i = 1; i < std::min<long long>(n, 4096); i++) {
    int m = 0;
    for (int a = 1; a < 3; a++)
      if (std::fabs(X[3 * i + a] - X[3 * i - 3 + a]) > std::fabs(X[3 * i + m] - X[3 * i - 3 + m])) m = a;
    steps[m]++;
  }
  const int first = (int)(std::max_element(steps, steps + 3) - steps);
  std::swap(g.axis[0], g.axis[first]);
  const double h = n > 0 ? std::cbrt(vol / n) : 1.0;
  g.inv = h > 0 && std::isfinite(h) ? 1.0 / h : 1.0;
  return g;
}

static pd_status begin_create(const pd_body_desc* desc, pd_handle** out, pd_handle** hp) {
  if (!out) return fail(PD_ERR_ARG, "out is NULL");
  *out = nullptr;
  PD_CUDA(cudaSetDevice(desc->device));
  pd_handle* h = new pd_handle();
  *hp = h;
  h->device = desc->device;
  h->n = desc->n_points;
  h->material = desc->material;
  h->kernel = desc->kernel;
  h->cmodel = desc->cmodel;
  h->precision = desc->precision;
  h->cs = desc->zem_cs;
  h->zem = desc->material == PD_MAT_CMAT ? desc->zem : PD_ZEM_SILLING;
  h->maxdmg = desc->maxdmg;
  h->multi = desc->multi_params ? 1 : 0;
  PD_CUDA(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking));
  h->own_stream = h->stream;
  for (int k = 0; k < desc->n_params; k++) h->hp.push_back(make_param(desc->params[k], h->cs));
  PD_TRY(dalloc(h, &h->dparams, h->hp.size()));
  PD_TRY(upload_params(h));
  PD_TRY(dalloc(h, &h->d.ctrl, 1));
  PD_CUDA(cudaMemsetAsync(h->d.ctrl, 0, sizeof(Ctrl), h->stream));
  PD_TRY(dalloc(h, &h->flags, 4));
  const long long n = h->n;
  h->hmeta.assign(n, 0u);
  for (long long i = 0; i < n; i++) h->hmeta[i] = desc->param_id ? desc->param_id[i] : 0u;
  PD_TRY(dalloc(h, &h->d.meta, n));
  PD_TRY(upload_meta(h));
  // reference positions and volumes
  std::vector<double4> X0(n > 0 ? n : 1), cur(n > 0 ? n : 1);
  for (long long i = 0; i < n; i++) {
    X0[i] = make_double4(desc->position[3 * i], desc->position[3 * i + 1], desc->position[3 * i + 2],
                         desc->volume[i]);
    cur[i] = h->precision == PD_PREC_FP64 ? X0[i] : make_double4(0, 0, 0, desc->volume[i]);
  }
  h->grid = place_grid(n, desc->position, desc->volume);
  double4 *dX0 = nullptr, *dcur = nullptr;
  PD_TRY(dalloc(h, &dX0, n));
  PD_TRY(dalloc(h, &dcur, n));
  PD_CUDA(h2d(dX0, X0.data(), sizeof(double4) * n, h->stream));
  PD_CUDA(h2d(dcur, cur.data(), sizeof(double4) * n, h->stream));
  h->d.X0 = dX0;
  h->d.cur = dcur;
  h->d.n = n;
  h->d.params = h->dparams;
  h->d.material = h->material;
  h->d.kernel = h->kernel;
  h->d.cmodel = h->cmodel;
  h->d.multi = h->multi;
  h->d.maxdmg = h->maxdmg;
  h->d.cs = h->cs;
  h->d.zem = h->zem;
  h->d.sym = 1;
  h->cfg.group = 1;
  h->cfg.block = 256;
  h->cfg.exact = false;
  h->cfg.pipe = 0;
  return PD_OK;
}

extern "C" pd_status pd_create(const pd_body_desc* desc, pd_handle** out) {
  PD_TRY(validate_desc(desc, true));
  pd_handle* h = nullptr;
  pd_status st = begin_create(desc, out, &h);
  if (st != PD_OK) { if (h) pd_destroy(h); return st; }
  h->nb = desc->n_bonds;
  h->d.nb = h->nb;
  const long long n = h->n, nb = h->nb;
  long long* doff = nullptr;
  int* dnbr = nullptr;
  double* dL = nullptr;
  unsigned char* dfp = nullptr;
  st = dalloc(h, &doff, n + 1);
  if (st == PD_OK) st = dalloc(h, &dnbr, nb);
  if (st == PD_OK && desc->bond_length) st = dalloc(h, &dL, nb);
  if (st == PD_OK && desc->fail_permit) st = dalloc(h, &dfp, nb);
  if (st != PD_OK) { pd_destroy(h); return st; }
  cudaError_t e = h2d(doff, desc->bond_offsets, sizeof(long long) * (n + 1), h->stream);
  if (e == cudaSuccess && nb) e = h2d(dnbr, desc->neighbors, sizeof(int) * nb, h->stream);
  if (e == cudaSuccess && dL) e = h2d(dL, desc->bond_length, sizeof(double) * nb, h->stream);
  if (e == cudaSuccess && dfp) e = h2d(dfp, desc->fail_permit, nb, h->stream);
  if (e != cudaSuccess) { pd_destroy(h); return fail(PD_ERR_CUDA, cudaGetErrorString(e)); }
  h->d.off = doff;
  st = finish_create(h, dnbr, dL, dfp);
  dfree(h, dnbr);
  if (dL) dfree(h, dL);
  if (dfp) dfree(h, dfp);
  if (st != PD_OK) { std::string m = g_err; pd_destroy(h); return fail(st, m); }
  *out = h;
  return PD_OK;
}

// device search; fills the cell grid from the host positions
static pd_status search_grid(long long n, const double* position, const double* delta, double lo[3],
                             double& hcell, long long nc[3]) {
  double dmax = 0;
  for (long long i = 0; i < n; i++) dmax = std::max(dmax, delta[i]);
  if (!(dmax > 0)) return fail(PD_ERR_ARG, "horizons must be > 0");
  hcell = dmax;
  long double ncell = 1;
  for (int k = 0; k < 3; k++) {
    double a = INFINITY, b = -INFINITY;
    for (long long i = 0; i < n; i++) { a = std::min(a, position[3 * i + k]); b = std::max(b, position[3 * i + k]); }
    if (n == 0) { a = 0; b = 0; }
    lo[k] = a;
    nc[k] = (long long)std::floor((b - a) / dmax) + 1;
    if (nc[k] < 1) nc[k] = 1;
    ncell *= nc[k];
  }
  if (ncell > 256.0L * 1024 * 1024)
    return fail(PD_ERR_ARG, "the bounding box holds more than 2^28 horizon-sized cells");
  return PD_OK;
}

static pd_status pack_masks(long long n, int32_t nf, const uint8_t* fa, const uint8_t* fb,
                            std::vector<unsigned short>& m) {
  if (nf < 0 || nf > 8) return fail(PD_ERR_ARG, "at most 8 filter-mode pre-cracks are supported");
  m.assign(n, 0);
  for (int k = 0; k < nf; k++)
    for (long long i = 0; i < n; i++) {
      if (fa[(size_t)k * n + i] && fb[(size_t)k * n + i])
        return fail(PD_ERR_ARG, "pre-crack point sets intersect");
      m[i] |= (unsigned short)((fa[(size_t)k * n + i] ? 1u : 0u) << (2 * k));
      m[i] |= (unsigned short)((fb[(size_t)k * n + i] ? 1u : 0u) << (2 * k + 1));
    }
  return PD_OK;
}

extern "C" pd_status pd_find_bonds(int64_t n, const double* position, const double* delta,
                                   const uint8_t* fp_point, int32_t n_filters, const uint8_t* filter_a,
                                   const uint8_t* filter_b, int64_t capacity, int64_t* bond_offsets,
                                   int32_t* neighbors, double* bond_length, uint8_t* fail_permit,
                                   int64_t* n_bonds, int32_t device) {
  if (n < 0 || !n_bonds || (n > 0 && (!position || !delta)))
    return fail(PD_ERR_ARG, "invalid arguments");
  PD_CUDA(cudaSetDevice(device));
  double lo[3], hc;
  long long nc[3];
  PD_TRY(search_grid(n, position, delta, lo, hc, nc));
  std::vector<unsigned short> mask;
  if (n_filters > 0) PD_TRY(pack_masks(n, n_filters, filter_a, filter_b, mask));
  cudaStream_t s;
  PD_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  double *dX = nullptr, *dd = nullptr, *dL = nullptr;
  unsigned short* dm = nullptr;
  long long* doff = nullptr;
  int* dnbr = nullptr;
  unsigned char *dfp = nullptr, *dfpb = nullptr;
  long long nb = 0;
  int dup = 0;
  pd_status st = PD_OK;
  cudaError_t e = cudaSuccess;
  auto ok = [&](cudaError_t x) { if (e == cudaSuccess) e = x; return e == cudaSuccess; };
  ok(cudaMalloc(&dX, sizeof(double) * 3 * (n ? n : 1)));
  ok(cudaMalloc(&dd, sizeof(double) * (n ? n : 1)));
  ok(cudaMalloc(&doff, sizeof(long long) * (n + 1)));
  if (n_filters > 0) ok(cudaMalloc(&dm, sizeof(unsigned short) * (n ? n : 1)));
  if (e == cudaSuccess) {
    ok(h2d(dX, position, sizeof(double) * 3 * n, s));
    ok(h2d(dd, delta, sizeof(double) * n, s));
    if (dm) ok(h2d(dm, mask.data(), sizeof(unsigned short) * n, s));
  }
  if (e == cudaSuccess) ok(device_find_bonds_grid(n, dX, dd, dm, nullptr, lo, hc, nc, doff, &dnbr, &nb, &dup, s));
  if (e == cudaSuccess && dup) st = fail(PD_ERR_ARG, "point duplicate found!");
  if (e == cudaSuccess && st == PD_OK) {
    *n_bonds = nb;
    if (capacity >= nb && bond_offsets && (nb == 0 || (neighbors && bond_length && fail_permit))) {
      ok(cudaMalloc(&dL, sizeof(double) * (nb ? nb : 1)));
      ok(cudaMalloc(&dfp, n ? n : 1));
      ok(cudaMalloc(&dfpb, nb ? nb : 1));
      if (e == cudaSuccess) {
        std::vector<unsigned char> fp(n, 1);
        if (fp_point) std::copy(fp_point, fp_point + n, fp.begin());
        ok(h2d(dfp, fp.data(), n, s));
        if (nb) launch_bond_props(n, dX, dfp, doff, dnbr, dL, dfpb, s);
        ok(cudaStreamSynchronize(s));
        ok(d2h(bond_offsets, doff, sizeof(long long) * (n + 1), s));
        if (nb) {
          ok(d2h(neighbors, dnbr, sizeof(int) * nb, s));
          ok(d2h(bond_length, dL, sizeof(double) * nb, s));
          ok(d2h(fail_permit, dfpb, nb, s));
        }
      }
    }
  }
  cudaFree(dX); cudaFree(dd); cudaFree(dm); cudaFree(doff); cudaFree(dnbr); cudaFree(dL);
  cudaFree(dfp); cudaFree(dfpb);
  cudaStreamDestroy(s);
  if (e != cudaSuccess) return fail(PD_ERR_CUDA, std::string("pd_find_bonds: ") + cudaGetErrorString(e));
  return st;
}

// the body's own neighbour search on the device; owned (may be null) restricts the bonds of
// the points outside it to owned neighbours and marks them halo rows
static pd_status create_search(const pd_body_desc* desc, const double* search_position,
                               const uint8_t* fp_point, int32_t n_filters, const uint8_t* filter_a,
                               const uint8_t* filter_b, const uint8_t* owned, pd_handle** out) {
  PD_TRY(validate_desc(desc, false));
  const long long n = desc->n_points;
  const double* spos = search_position ? search_position : desc->position;
  std::vector<double> delta(n);
  for (long long i = 0; i < n; i++) delta[i] = desc->params[desc->param_id ? desc->param_id[i] : 0].delta;
  double lo[3], hc;
  long long nc[3];
  PD_TRY(search_grid(n, spos, delta.data(), lo, hc, nc));
  std::vector<unsigned short> mask;
  if (n_filters > 0) PD_TRY(pack_masks(n, n_filters, filter_a, filter_b, mask));
  pd_handle* h = nullptr;
  pd_status st = begin_create(desc, out, &h);
  if (st != PD_OK) { if (h) pd_destroy(h); return st; }
  if (owned) {
    for (long long i = 0; i < n; i++)
      if (!owned[i]) h->hmeta[i] |= pd::META_HALO;
    st = upload_meta(h);
    if (st != PD_OK) { std::string m = g_err; pd_destroy(h); return fail(st, m); }
  }
  double *dX = nullptr, *dXs = nullptr, *dd = nullptr;
  unsigned short* dm = nullptr;
  long long* doff = nullptr;
  unsigned char *dfp = nullptr, *dfpb = nullptr, *down = nullptr;
  std::vector<double> X(desc->position, desc->position + 3 * n);
  st = dalloc(h, &dX, 3 * n);
  if (st == PD_OK && search_position) st = dalloc(h, &dXs, 3 * n);
  if (st == PD_OK) st = dalloc(h, &dd, n);
  if (st == PD_OK) st = dalloc(h, &doff, n + 1);
  if (st == PD_OK && n_filters > 0) st = dalloc(h, &dm, n);
  if (st == PD_OK) st = dalloc(h, &dfp, n);
  if (st == PD_OK && owned) st = dalloc(h, &down, n);
  if (st != PD_OK) { std::string m = g_err; pd_destroy(h); return fail(st, m); }
  std::vector<unsigned char> fp(n, 1);
  if (fp_point) std::copy(fp_point, fp_point + n, fp.begin());
  cudaError_t e = h2d(dX, X.data(), sizeof(double) * 3 * n, h->stream);
  if (e == cudaSuccess && dXs) e = h2d(dXs, search_position, sizeof(double) * 3 * n, h->stream);
  if (e == cudaSuccess) e = h2d(dd, delta.data(), sizeof(double) * n, h->stream);
  if (e == cudaSuccess && dm) e = h2d(dm, mask.data(), sizeof(unsigned short) * n, h->stream);
  if (e == cudaSuccess) e = h2d(dfp, fp.data(), n, h->stream);
  if (e == cudaSuccess && down) e = h2d(down, owned, n, h->stream);
  int* dnbr = nullptr;
  long long nb = 0;
  int dup = 0;
  if (e == cudaSuccess)
    e = device_find_bonds_grid(n, dXs ? dXs : dX, dd, dm, down, lo, hc, nc, doff, &dnbr, &nb, &dup, h->stream);
  if (e != cudaSuccess) { pd_destroy(h); return fail(PD_ERR_CUDA, cudaGetErrorString(e)); }
  if (dup) { pd_destroy(h); return fail(PD_ERR_ARG, "point duplicate found!"); }
  h->allocs.push_back(dnbr);
  h->nb = nb;
  h->d.nb = nb;
  h->d.off = doff;
  double* dL = nullptr;
  st = dalloc(h, &dL, nb);
  if (st == PD_OK) st = dalloc(h, &dfpb, nb);
  if (st != PD_OK) { std::string m = g_err; pd_destroy(h); return fail(st, m); }
  if (nb) launch_bond_props(n, dX, dfp, doff, dnbr, dL, dfpb, h->stream);
  dfree(h, dX); dfree(h, dXs); dfree(h, dd); dfree(h, dm); dfree(h, dfp); dfree(h, down);
  st = finish_create(h, dnbr, dL, dfpb);
  dfree(h, dnbr); dfree(h, dL); dfree(h, dfpb);
  if (st != PD_OK) { std::string m = g_err; pd_destroy(h); return fail(st, m); }
  *out = h;
  return PD_OK;
}

extern "C" pd_status pd_create_search(const pd_body_desc* desc, const double* search_position,
                                      const uint8_t* fp_point, int32_t n_filters,
                                      const uint8_t* filter_a, const uint8_t* filter_b,
                                      pd_handle** out) {
  return create_search(desc, search_position, fp_point, n_filters, filter_a, filter_b, nullptr, out);
}

extern "C" pd_status pd_create_partition(const pd_body_desc* desc, const double* search_position,
                                         const uint8_t* fp_point, int32_t n_filters,
                                         const uint8_t* filter_a, const uint8_t* filter_b,
                                         const uint8_t* owned, pd_handle** out) {
  if (!owned) return fail(PD_ERR_ARG, "owned is NULL");
  return create_search(desc, search_position, fp_point, n_filters, filter_a, filter_b, owned, out);
}

extern "C" pd_status pd_destroy(pd_handle* h) {
  if (!h) return PD_OK;
  cudaSetDevice(h->device);
  if (h->stream) cudaStreamSynchronize(h->stream);
  destroy_graph(h);
  pd::nk_release(h);
  pd::dr_release(h);
  for (void* p : h->allocs) cudaFree(p);
  h->allocs.clear();
  if (h->own_stream) cudaStreamDestroy(h->own_stream);
  delete h;
  return PD_OK;
}

static pd_status clear_error(pd_handle* h) {
  const int z = 0;
  PD_TRY(set_ctrl(h, offsetof(Ctrl, err), &z, sizeof(int)));
  h->nan_step = -1;
  return PD_OK;
}

// the handle's transfer staging buffer, at least `bytes` long (a point field: 9 doubles a point
// at most)
static pd_status staging(pd_handle* h, size_t bytes, void** p) {
  if (h->xfer_bytes < bytes) {
    dfree(h, h->xfer);
    h->xfer = nullptr;
    h->xfer_bytes = 0;
    unsigned char* q = nullptr;
    PD_TRY(dalloc(h, &q, bytes));
    h->xfer = q;
    h->xfer_bytes = bytes;
  }
  *p = h->xfer;
  return PD_OK;
}

// cur[i].xyz = in[3i..3i+2] (- X0[i].xyz with sub_x0); the fourth component is kept
__global__ void k_set_cur(double4* cur, const double4* X0, const double* in, long long n, int sub_x0) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double4 c = cur[i];
  c.x = in[3 * i];
  c.y = in[3 * i + 1];
  c.z = in[3 * i + 2];
  if (sub_x0) {
    const double4 x = X0[i];
    c.x = c.x - x.x;
    c.y = c.y - x.y;
    c.z = c.z - x.z;
  }
  cur[i] = c;
}

extern "C" pd_status pd_set_state(pd_handle* h, const double* position, const double* displacement,
                                  const double* velocity, const double* velocity_half,
                                  const double* acceleration, const double* b_ext,
                                  const uint8_t* bond_active) {
  if (!h) return fail(PD_ERR_ARG, "handle is NULL");
  PD_CUDA(cudaSetDevice(h->device));
  PD_CUDA(cudaStreamSynchronize(h->stream));
  const long long n = h->n, nb = h->nb;
  if (n == 0) return PD_OK;
  // the packed point state (FP64: current position; FP32: displacement) from a 3n host array,
  // packed on the device
  const double* src = nullptr;
  int sub_x0 = 0;
  // every copy and kernel is ordered on the handle's stream (from page-locked host memory the
  // copies run at full PCIe rate); one synchronize at the end
  const size_t vec = sizeof(double) * 3 * n;
  const cudaMemcpyKind kh2d = cudaMemcpyHostToDevice;
  if (h->precision == PD_PREC_FP64) {
    src = position;
    if (displacement) PD_CUDA(cudaMemcpyAsync(h->g.u, displacement, vec, kh2d, h->stream));
  } else if (displacement) {
    src = displacement;
  } else if (position) {
    src = position;
    sub_x0 = 1;
  }
  if (src) {
    void* tmp = nullptr;
    PD_TRY(staging(h, vec, &tmp));
    PD_CUDA(cudaMemcpyAsync(tmp, src, vec, kh2d, h->stream));
    k_set_cur<<<(unsigned)((n + 255) / 256), 256, 0, h->stream>>>(h->d.cur, h->d.X0, (const double*)tmp,
                                                                  n, sub_x0);
    PD_CUDA(cudaGetLastError());
    launch_split_u(h->d, h->stream);
    PD_CUDA(cudaGetLastError());
  }
  if (velocity) PD_CUDA(cudaMemcpyAsync(h->g.v, velocity, vec, kh2d, h->stream));
  if (velocity_half) PD_CUDA(cudaMemcpyAsync(h->g.vh, velocity_half, vec, kh2d, h->stream));
  if (acceleration) PD_CUDA(cudaMemcpyAsync(h->g.a, acceleration, vec, kh2d, h->stream));
  PD_CUDA(cudaStreamSynchronize(h->stream));
  if (b_ext) {
    PD_CUDA(h2d(h->g.bext, b_ext, vec, h->stream));
    for (long long i = 0; i < n; i++) {
      const bool nz = b_ext[3 * i] != 0 || b_ext[3 * i + 1] != 0 || b_ext[3 * i + 2] != 0 ||
                      std::signbit(b_ext[3 * i]) || std::signbit(b_ext[3 * i + 1]) || std::signbit(b_ext[3 * i + 2]);
      const bool bc = !h->bext_pt.empty() && h->bext_pt[i];
      if (nz || bc) h->hmeta[i] |= META_HAS_BEXT; else h->hmeta[i] &= ~META_HAS_BEXT;
    }
    PD_TRY(upload_meta(h));
  }
  if (bond_active && nb > 0) {
    void* tmp = nullptr;
    PD_TRY(staging(h, (size_t)nb, &tmp));
    cudaError_t e = h2d(tmp, bond_active, nb, h->stream);
    if (e == cudaSuccess) {
      launch_pack_bits(h->d, (const unsigned char*)tmp, h->stream);
      h->kfull = true;
      e = cudaStreamSynchronize(h->stream);
    }
    if (e != cudaSuccess) return fail(PD_ERR_CUDA, cudaGetErrorString(e));
    launch_count_active(h->d, h->stream);
    h->damage_valid = true;
    PD_TRY(check_symmetry(h));
    drop_graphs(h);
  }
  PD_TRY(clear_error(h));
  PD_CUDA(cudaStreamSynchronize(h->stream));
  return PD_OK;
}

extern "C" pd_status pd_get_field(pd_handle* h, int32_t field, void* out, size_t bytes) {
  if (!h || !out) return fail(PD_ERR_ARG, "handle or output is NULL");
  PD_CUDA(cudaSetDevice(h->device));
  PD_CUDA(cudaStreamSynchronize(h->stream));
  const long long n = h->n, nb = h->nb;
  size_t need = 0;
  switch (field) {
    case PD_FIELD_POSITION: case PD_FIELD_DISPLACEMENT: case PD_FIELD_VELOCITY:
    case PD_FIELD_VELOCITY_HALF: case PD_FIELD_ACCELERATION: case PD_FIELD_B_INT:
    case PD_FIELD_B_EXT: need = sizeof(double) * 3 * n; break;
    case PD_FIELD_DAMAGE: need = sizeof(double) * n; break;
    case PD_FIELD_N_ACTIVE_BONDS: case PD_FIELD_N_NEIGHBORS: need = sizeof(int64_t) * n; break;
    case PD_FIELD_BOND_ACTIVE: need = nb; break;
    case PD_FIELD_DEFGRAD: case PD_FIELD_CAUCHY_STRESS:
      if (h->material != PD_MAT_CMAT) return fail(PD_ERR_ARG, "field only exists for CMaterial");
      need = sizeof(double) * 9 * n; break;
    default: return fail(PD_ERR_ARG, "unknown field");
  }
  if (bytes != need) return fail(PD_ERR_ARG, "output size is " + std::to_string(bytes) + " bytes, need " + std::to_string(need));
  if (n == 0) return PD_OK;
  // device -> host on the handle's stream; exported point fields go through the staging buffer
  auto copy = [&](const void* src) -> pd_status {
    PD_CUDA(cudaMemcpyAsync(out, src, need, cudaMemcpyDeviceToHost, h->stream));
    PD_CUDA(cudaStreamSynchronize(h->stream));
    return PD_OK;
  };
  void* tmp = nullptr;
  pd_status st = PD_OK;
  switch (field) {
    case PD_FIELD_POSITION: case PD_FIELD_DISPLACEMENT:
      PD_TRY(staging(h, need, &tmp));
      launch_export_position(h->d, h->g, (double*)tmp, field == PD_FIELD_POSITION ? 0 : 1, h->stream);
      PD_CUDA(cudaGetLastError());
      st = copy(tmp);
      break;
    case PD_FIELD_VELOCITY: st = copy(h->g.v); break;
    case PD_FIELD_VELOCITY_HALF: st = copy(h->g.vh); break;
    case PD_FIELD_ACCELERATION: st = copy(h->g.a); break;
    case PD_FIELD_B_EXT: st = copy(h->g.bext); break;
    case PD_FIELD_B_INT:
      if (h->precision == PD_PREC_FP64) st = copy(h->d.b64);
      else {
        std::vector<float> f(3 * n);
        PD_CUDA(d2h(f.data(), h->d.b32, sizeof(float) * 3 * n, h->stream));
        double* o = (double*)out;
        for (long long k = 0; k < 3 * n; k++) o[k] = f[k];
      }
      break;
    case PD_FIELD_DAMAGE:
      PD_TRY(staging(h, need, &tmp));
      launch_export_damage(h->d, h->damage_valid ? 1 : 0, (double*)tmp, h->stream);
      PD_CUDA(cudaGetLastError());
      st = copy(tmp);
      break;
    case PD_FIELD_N_ACTIVE_BONDS: {
      std::vector<int> na(n);
      PD_CUDA(d2h(na.data(), h->d.n_active, sizeof(int) * n, h->stream));
      int64_t* o = (int64_t*)out;
      for (long long i = 0; i < n; i++) o[i] = na[i];
      break;
    }
    case PD_FIELD_N_NEIGHBORS: {
      std::vector<long long> off(n + 1);
      PD_CUDA(d2h(off.data(), h->d.off, sizeof(long long) * (n + 1), h->stream));
      int64_t* o = (int64_t*)out;
      for (long long i = 0; i < n; i++) o[i] = off[i + 1] - off[i];
      break;
    }
    case PD_FIELD_BOND_ACTIVE: {
      if (nb == 0) break;
      // one byte a bond: a temporary, not kept
      PD_CUDA(cudaMalloc(&tmp, need));
      launch_export_bond_active(h->d, (unsigned char*)tmp, 0, h->stream);
      cudaError_t e = cudaGetLastError();
      if (e == cudaSuccess) e = cudaMemcpyAsync(out, tmp, need, cudaMemcpyDeviceToHost, h->stream);
      if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
      cudaFree(tmp);
      if (e != cudaSuccess) return fail(PD_ERR_CUDA, cudaGetErrorString(e));
      break;
    }
    case PD_FIELD_DEFGRAD:
      if (h->precision == PD_PREC_FP64) st = copy(h->d.F64);
      else {
        std::vector<float> f(9 * n);
        PD_CUDA(d2h(f.data(), h->d.H32, sizeof(float) * 9 * n, h->stream));
        double* o = (double*)out;
        for (long long i = 0; i < n; i++)
          for (int k = 0; k < 9; k++) o[9 * i + k] = (double)f[9 * i + k] + ((k % 4) == 0 ? 1.0 : 0.0);
      }
      break;
    case PD_FIELD_CAUCHY_STRESS:
      PD_TRY(staging(h, need, &tmp));
      launch_cauchy64(h->d, h->d.F64, h->precision == PD_PREC_FP64 ? 0 : 1, (double*)tmp, h->stream);
      PD_CUDA(cudaGetLastError());
      st = copy(tmp);
      break;
  }
  PD_CUDA(cudaGetLastError());
  return st;
}

extern "C" pd_status pd_set_bcs(pd_handle* h, int32_t n_bcs, const pd_bc_desc* bcs) {
  if (!h) return fail(PD_ERR_ARG, "handle is NULL");
  if (n_bcs < 0 || (n_bcs > 0 && !bcs)) return fail(PD_ERR_ARG, "invalid boundary conditions");
  PD_CUDA(cudaSetDevice(h->device));
  const long long n = h->n;
  std::vector<BCInfo> info(n_bcs);
  std::vector<std::vector<BCEntry>> per_point(n);
  std::vector<double> data;
  long long col = 0;
  h->needs_table = false;
  h->bext_pt.assign(n, 0);
  for (int k = 0; k < n_bcs; k++) {
    const pd_bc_desc& b = bcs[k];
    if (b.field != PD_BC_VELOCITY_HALF && b.field != PD_BC_B_EXT) return fail(PD_ERR_ARG, "unknown boundary condition field");
    if (b.dim < 0 || b.dim > 2) return fail(PD_ERR_ARG, "dimension must be 0, 1 or 2");
    if (b.kind < PD_BC_KIND_TIME || b.kind > PD_BC_KIND_DATA) return fail(PD_ERR_ARG, "unknown boundary condition kind");
    if (b.n_points < 0 || (b.n_points > 0 && !b.points)) return fail(PD_ERR_ARG, "boundary condition point list missing");
    if (b.kind == PD_BC_KIND_DATA && b.n_points > 0 && !b.data) return fail(PD_ERR_ARG, "DataBC values missing");
    info[k].field = b.field;
    info[k].dim = b.dim;
    info[k].kind = b.kind;
    if (b.kind == PD_BC_KIND_TIME) { info[k].col = (int)col; col += 1; h->needs_table = true; }
    else if (b.kind == PD_BC_KIND_POINT_TIME) { info[k].col = (int)col; col += b.n_points; h->needs_table = true; }
    else { info[k].col = (int)data.size(); data.insert(data.end(), b.data, b.data + b.n_points); }
    for (int q = 0; q < b.n_points; q++) {
      const int p = b.points[q];
      if (p < 0 || p >= n) return fail(PD_ERR_ARG, "boundary condition point out of range");
      per_point[p].push_back(BCEntry{k, q});
      if (b.field == PD_BC_B_EXT) h->bext_pt[p] = 1;
    }
  }
  std::vector<int> pts, eoff(1, 0);
  std::vector<BCEntry> ent;
  for (long long i = 0; i < n; i++) {
    h->hmeta[i] &= ~META_HAS_BC;
    if (per_point[i].empty()) continue;
    pts.push_back((int)i);
    for (auto& e : per_point[i]) ent.push_back(e);
    eoff.push_back((int)ent.size());
    h->hmeta[i] |= META_HAS_BC;
    if (h->bext_pt[i]) h->hmeta[i] |= META_HAS_BEXT;
  }
  PD_TRY(upload_meta(h));
  PD_CUDA(cudaStreamSynchronize(h->stream));
  // free the previous lists
  dfree(h, (void*)h->bc.point); dfree(h, (void*)h->bc.entry_off); dfree(h, (void*)h->bc.entry);
  dfree(h, (void*)h->bc.info); dfree(h, (void*)h->bc.data); dfree(h, (void*)h->bc.slot);
  h->bc = BCDev{};
  h->bc.table = h->table;
  // the position of every constrained point in the condition list (-1: none)
  std::vector<int> slot(n, -1);
  for (size_t p = 0; p < pts.size(); p++) slot[pts[p]] = (int)p;
  int* ds = nullptr;
  PD_TRY(dalloc(h, &ds, n));
  if (n > 0) PD_CUDA(h2d(ds, slot.data(), sizeof(int) * n, h->stream));
  h->bc.slot = ds;
  int *dp = nullptr, *de = nullptr;
  BCEntry* den = nullptr;
  BCInfo* di = nullptr;
  double* dd = nullptr;
  PD_TRY(dalloc(h, &dp, pts.size()));
  PD_TRY(dalloc(h, &de, eoff.size()));
  PD_TRY(dalloc(h, &den, ent.size()));
  PD_TRY(dalloc(h, &di, info.size()));
  PD_TRY(dalloc(h, &dd, data.size()));
  if (!pts.empty()) PD_CUDA(h2d(dp, pts.data(), sizeof(int) * pts.size(), h->stream));
  PD_CUDA(h2d(de, eoff.data(), sizeof(int) * eoff.size(), h->stream));
  if (!ent.empty()) PD_CUDA(h2d(den, ent.data(), sizeof(BCEntry) * ent.size(), h->stream));
  if (!info.empty()) PD_CUDA(h2d(di, info.data(), sizeof(BCInfo) * info.size(), h->stream));
  if (!data.empty()) PD_CUDA(h2d(dd, data.data(), sizeof(double) * data.size(), h->stream));
  h->bc.n_points = (int)pts.size();
  h->bc.point = dp;
  h->bc.entry_off = de;
  h->bc.entry = den;
  h->bc.info = di;
  h->bc.data = dd;
  h->bc.per_step = col;
  h->per_step = col;
  h->bcinfo = info;
  const long long zero = 0;
  PD_TRY(set_ctrl(h, offsetof(Ctrl, table_n), &zero, sizeof(long long)));
  PD_CUDA(cudaStreamSynchronize(h->stream));
  drop_graphs(h);
  return PD_OK;
}

extern "C" pd_status pd_set_bc_values(pd_handle* h, int64_t first_step, int64_t n_steps,
                                      const double* values, int64_t n_values) {
  if (!h) return fail(PD_ERR_ARG, "handle is NULL");
  if (n_steps < 0) return fail(PD_ERR_ARG, "n_steps < 0");
  if (n_values != n_steps * h->per_step)
    return fail(PD_ERR_ARG, "expected " + std::to_string(n_steps * h->per_step) + " values");
  PD_CUDA(cudaSetDevice(h->device));
  if (n_values > h->table_cap) {
    PD_CUDA(cudaStreamSynchronize(h->stream));
    dfree(h, h->table);
    h->table = nullptr;
    PD_TRY(dalloc(h, &h->table, n_values));
    h->table_cap = n_values;
    h->bc.table = h->table;
    h->version++;
  }
  if (n_values > 0)
    PD_CUDA(cudaMemcpyAsync(h->table, values, sizeof(double) * n_values, cudaMemcpyHostToDevice, h->stream));
  long long v[2] = {first_step, n_steps};
  PD_TRY(set_ctrl(h, offsetof(Ctrl, table_first), v, sizeof(v)));
  PD_CUDA(cudaStreamSynchronize(h->stream));
  return PD_OK;
}

extern "C" pd_status pd_stable_timestep(pd_handle* h, double safety_factor, double* dt,
                                        double* dt_per_param) {
  if (!h || !dt) return fail(PD_ERR_ARG, "handle or dt is NULL");
  PD_CUDA(cudaSetDevice(h->device));
  const long long n = h->n;
  double* tmp = nullptr;
  std::vector<double> dtp(n);
  if (n > 0) {
    PD_CUDA(cudaMalloc(&tmp, sizeof(double) * n));
    launch_timestep(h->d, tmp, h->stream);
    cudaError_t e = cudaStreamSynchronize(h->stream);
    if (e == cudaSuccess) e = d2h(dtp.data(), tmp, sizeof(double) * n, h->stream);
    cudaFree(tmp);
    if (e != cudaSuccess) return fail(PD_ERR_CUDA, cudaGetErrorString(e));
  }
  double m = INFINITY;
  std::vector<double> mp(h->hp.size(), INFINITY);
  for (long long i = 0; i < n; i++) {
    m = std::min(m, dtp[i]);
    const unsigned p = h->hmeta[i] & META_PID_MASK;
    mp[p] = std::min(mp[p], dtp[i]);
  }
  *dt = m * safety_factor;
  if (dt_per_param)
    for (size_t k = 0; k < mp.size(); k++) dt_per_param[k] = mp[k] * safety_factor;
  return PD_OK;
}

extern "C" pd_status pd_set_param_timesteps(pd_handle* h, const double* dtp) {
  if (!h || !dtp) return fail(PD_ERR_ARG, "handle or dt_per_param is NULL");
  PD_CUDA(cudaSetDevice(h->device));
  for (size_t k = 0; k < h->hp.size(); k++) { h->hp[k].dt = dtp[k]; h->hp[k].dth = 0.5 * dtp[k]; }
  PD_TRY(upload_params(h));
  drop_graphs(h);
  return PD_OK;
}

// bond-stream variants 1 to 3 where they apply
static bool runs_tma(const pd_handle* h) {
  return h->cfg.pipe >= 1 && h->cfg.pipe <= 3 && !h->d.sc32 && tma_supported(h->d);
}

static int launch_force(pd_handle* h, int kstep, int phase) {
  int k;
  // FP32 OSB / CMat: the first phase-A launch after bond states changed outside the kernels sums
  // the weighted volumes / shape tensors in full; graphs captured with that launch are
  // captured again
  const bool fullk = h->kfull && h->material != PD_MAT_BB && h->precision != PD_PREC_FP64 && phase != 2;
  h->cfg.fullk = fullk ? 1 : 0;
  if (fullk) { h->kfull = false; h->version++; }
  if (h->precision == PD_PREC_FP64) k = launch_force64(h->d, h->cfg, kstep, phase, h->stream);
  else if (runs_tma(h))
    k = launch_force32_tma(h->d, h->cfg.pipe, kstep, phase, h->stream);
  else k = launch_force32(h->d, h->cfg, kstep, phase, h->stream);
  h->launches += k;
  return k;
}

static pd_status check_err(pd_handle* h) {
  Ctrl c;
  PD_CUDA(cudaMemcpyAsync(&c, h->d.ctrl, sizeof(Ctrl), cudaMemcpyDeviceToHost, h->stream));
  PD_CUDA(cudaStreamSynchronize(h->stream));
  if (c.err == 1) {
    h->nan_step = c.err_step;
    return fail(PD_ERR_NAN, "NaN values detected in force density field! step: " + std::to_string(c.err_step));
  }
  if (c.err == 3) return fail(PD_ERR_TIMEOUT, "a bounded wait of a force kernel gave up");
  if (c.err == 4) return fail(PD_ERR_ARG, "a halo row index outside the body (pd_halo_pack)");
  if (c.err == 2)
    return fail(PD_ERR_ARG, "boundary condition values missing for step " + std::to_string(c.err_step) +
                                " (call pd_set_bc_values)");
  return PD_OK;
}

extern "C" pd_status pd_force(pd_handle* h, double t, double dt) {
  if (!h) return fail(PD_ERR_ARG, "handle is NULL");
  PD_CUDA(cudaSetDevice(h->device));
  PD_TRY(clear_error(h));
  const long long step = (t > 0 && dt > 0) ? (long long)std::floor(t / dt) : 0;
  PD_TRY(set_ctrl(h, offsetof(Ctrl, base), &step, sizeof(long long)));
  launch_force(h, 0, 0);
  PD_CUDA(cudaGetLastError());
  h->damage_valid = true;
  return check_err(h);
}

// one block of steps [kstep0, kstep0 + steps) as eager launches; timing events optional
static void issue_steps(pd_handle* h, int steps, double dto, std::vector<cudaEvent_t>* ev) {
  int e = 0;
  auto rec = [&]() { if (ev) cudaEventRecord((*ev)[e++], h->stream); };
  for (int k = 0; k < steps; k++) {
    rec();
    launch_kick_drift(h->d, h->g, h->bc, k == 0 ? 0 : 1, dto, k, h->stream);
    h->launches++;
    rec();
    launch_force(h, k, 1);
    rec();
    launch_force(h, k, 2);
    rec();
  }
  rec();
  launch_finish(h->d, h->g, dto, h->stream);
  h->launches++;
  rec();
}

static pd_status run_block_graph(pd_handle* h, int steps, double dto) {
  GraphKey key;
  key.steps = steps; key.group = h->cfg.group; key.block = h->cfg.block; key.exact = h->cfg.exact;
  key.bcpts = h->bc.n_points; key.dt = dto; key.version = h->version; key.pipe = h->cfg.pipe;
  if (!(h->gexec && key == h->gkey)) {
    destroy_graph(h);
    cudaGraph_t graph;
    long long before = h->launches;
    PD_CUDA(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
    cudaGetLastError();  // of earlier calls
    issue_steps(h, steps, dto, nullptr);
    const cudaError_t le = cudaGetLastError();  // a launch that was refused
    cudaError_t e = cudaStreamEndCapture(h->stream, &graph);
    if (e == cudaSuccess && le != cudaSuccess) { cudaGraphDestroy(graph); e = le; }
    if (e != cudaSuccess) return fail(PD_ERR_CUDA, std::string("graph capture: ") + cudaGetErrorString(e));
    h->graph_nodes = (int)(h->launches - before);
    h->launches = before;
    e = cudaGraphInstantiate(&h->gexec, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) { h->gexec = nullptr; return fail(PD_ERR_CUDA, std::string("graph instantiate: ") + cudaGetErrorString(e)); }
    h->gkey = key;
  }
  PD_CUDA(cudaGraphLaunch(h->gexec, h->stream));
  h->launches += h->graph_nodes;
  return PD_OK;
}

static pd_status run_vv(pd_handle* h, int64_t first_step, int64_t n_steps, double dt,
                        std::vector<cudaEvent_t>* ev) {
  if (!h) return fail(PD_ERR_ARG, "handle is NULL");
  if (n_steps < 0) return fail(PD_ERR_ARG, "n_steps < 0");
  if (n_steps == 0) return PD_OK;
  PD_CUDA(cudaSetDevice(h->device));
  double dto = dt > 0 ? dt : -1.0;
  if (dto < 0)
    for (auto& p : h->hp)
      if (!(p.dt > 0)) return fail(PD_ERR_ARG, "dt <= 0 and no per-parameter time steps set");
  if (h->needs_table) {
    Ctrl c;
    PD_CUDA(d2h(&c, h->d.ctrl, sizeof(Ctrl), h->stream));
    if (c.table_first > first_step || c.table_first + c.table_n < first_step + n_steps)
      return fail(PD_ERR_ARG, "boundary condition values do not cover steps " + std::to_string(first_step) +
                                  ".." + std::to_string(first_step + n_steps - 1));
  }
  PD_TRY(clear_error(h));
  int64_t done = 0;
  const int K = h->graph_steps;
  while (done < n_steps) {
    const long long base = first_step + done;
    int steps = (int)std::min<int64_t>(n_steps - done, (K > 0 && !ev) ? K : (int64_t)(1 << 30));
    PD_TRY(set_ctrl(h, offsetof(Ctrl, base), &base, sizeof(long long)));
    if (K > 0 && steps == K && !ev) {
      PD_TRY(run_block_graph(h, steps, dto));
    } else {
      issue_steps(h, steps, dto, ev);
      PD_CUDA(cudaGetLastError());
    }
    done += steps;
    if (ev) break;
  }
  h->damage_valid = true;
  return check_err(h);
}

extern "C" pd_status pd_run_vv(pd_handle* h, int64_t first_step, int64_t n_steps, double dt) {
  return run_vv(h, first_step, n_steps, dt, nullptr);
}

// ---------------------------------------------------------------------------------------
// Groups of bodies advanced together (the size classes of an ensemble): the steps of every
// body of the group in one CUDA graph, each body's launches on its own stream, forked from and
// joined into the first body's stream.
// ---------------------------------------------------------------------------------------
struct pd_group {
  std::vector<pd_handle*> hs;
  int device = 0;
  cudaEvent_t fork = nullptr;
  std::vector<cudaEvent_t> join;
  cudaGraphExec_t gexec = nullptr;
  int gsteps = 0;
  double gdt = 0;
  std::vector<GraphKey> keys;  // per body: mapping and state version the graph was made for
  std::vector<long long> nodes;  // per body: kernels of one graph launch
};

static void group_release_graph(pd_group* g) {
  if (g->gexec) cudaGraphExecDestroy(g->gexec);
  g->gexec = nullptr;
  g->keys.clear();
}

extern "C" pd_status pd_group_create(pd_handle* const* handles, int32_t n, pd_group** out) {
  if (!handles || n < 1 || !out) return fail(PD_ERR_ARG, "handles, n >= 1 and out are required");
  for (int k = 0; k < n; k++) {
    if (!handles[k]) return fail(PD_ERR_ARG, "handle is NULL");
    if (handles[k]->device != handles[0]->device)
      return fail(PD_ERR_ARG, "the bodies of a group share one device");
    for (int q = 0; q < k; q++)
      if (handles[q] == handles[k] || handles[q]->stream == handles[k]->stream)
        return fail(PD_ERR_ARG, "the bodies of a group are distinct and on distinct streams");
  }
  PD_CUDA(cudaSetDevice(handles[0]->device));
  pd_group* g = new pd_group();
  g->hs.assign(handles, handles + n);
  g->device = handles[0]->device;
  cudaError_t e = cudaEventCreateWithFlags(&g->fork, cudaEventDisableTiming);
  g->join.assign(n, nullptr);
  for (int k = 0; k < n && e == cudaSuccess; k++) e = cudaEventCreateWithFlags(&g->join[k], cudaEventDisableTiming);
  if (e != cudaSuccess) {
    pd_group_destroy(g);
    return fail(PD_ERR_CUDA, std::string("pd_group_create: ") + cudaGetErrorString(e));
  }
  *out = g;
  return PD_OK;
}

extern "C" pd_status pd_group_destroy(pd_group* g) {
  if (!g) return PD_OK;
  cudaSetDevice(g->device);
  group_release_graph(g);
  if (g->fork) cudaEventDestroy(g->fork);
  for (cudaEvent_t e : g->join)
    if (e) cudaEventDestroy(e);
  delete g;
  return PD_OK;
}

// the steps [0, steps) of every body, each on its own stream between the fork and the join
static void group_issue(pd_group* g, int steps, double dto) {
  cudaStream_t origin = g->hs[0]->stream;
  cudaEventRecord(g->fork, origin);
  for (size_t k = 1; k < g->hs.size(); k++) cudaStreamWaitEvent(g->hs[k]->stream, g->fork, 0);
  for (pd_handle* h : g->hs) issue_steps(h, steps, dto, nullptr);
  for (size_t k = 1; k < g->hs.size(); k++) {
    cudaEventRecord(g->join[k], g->hs[k]->stream);
    cudaStreamWaitEvent(origin, g->join[k], 0);
  }
}

static GraphKey group_key(const pd_handle* h, int steps, double dto) {
  GraphKey key;
  key.steps = steps; key.group = h->cfg.group; key.block = h->cfg.block; key.exact = h->cfg.exact;
  key.bcpts = h->bc.n_points; key.dt = dto; key.version = h->version; key.pipe = h->cfg.pipe;
  return key;
}

extern "C" pd_status pd_group_run_vv(pd_group* g, int64_t first_step, int64_t n_steps, double dt,
                                     int32_t steps_per_graph, double* ms_total) {
  if (!g) return fail(PD_ERR_ARG, "group is NULL");
  if (n_steps < 0 || steps_per_graph < 0 || steps_per_graph > 4096)
    return fail(PD_ERR_ARG, "n_steps >= 0 and 0 <= steps_per_graph <= 4096");
  if (ms_total) *ms_total = 0.0;
  if (n_steps == 0) return PD_OK;
  PD_CUDA(cudaSetDevice(g->device));
  const double dto = dt > 0 ? dt : -1.0;
  for (pd_handle* h : g->hs) {
    if (dto < 0)
      for (auto& p : h->hp)
        if (!(p.dt > 0)) return fail(PD_ERR_ARG, "dt <= 0 and no per-parameter time steps set");
    if (h->needs_table) {
      Ctrl c;
      PD_CUDA(d2h(&c, h->d.ctrl, sizeof(Ctrl), h->stream));
      if (c.table_first > first_step || c.table_first + c.table_n < first_step + n_steps)
        return fail(PD_ERR_ARG, "boundary condition values do not cover steps " +
                                    std::to_string(first_step) + ".." +
                                    std::to_string(first_step + n_steps - 1));
    }
    PD_TRY(clear_error(h));
    PD_CUDA(cudaStreamSynchronize(h->stream));
  }
  cudaStream_t origin = g->hs[0]->stream;
  cudaEvent_t t0 = nullptr, t1 = nullptr;
  if (ms_total) {
    PD_CUDA(cudaEventCreate(&t0));
    PD_CUDA(cudaEventCreate(&t1));
    cudaEventRecord(t0, origin);
  }
  pd_status st = PD_OK;
  const int K = steps_per_graph;
  int64_t done = 0;
  while (done < n_steps && st == PD_OK) {
    const long long base = first_step + done;
    const int steps = (int)std::min<int64_t>(n_steps - done, K > 0 ? K : (int64_t)(1 << 30));
    // every body's first step of the block, written on the origin stream before the launch
    for (pd_handle* h : g->hs) {
      cudaError_t e = cudaMemcpyAsync(reinterpret_cast<char*>(h->d.ctrl) + offsetof(Ctrl, base), &base,
                                      sizeof(long long), cudaMemcpyHostToDevice, origin);
      if (e != cudaSuccess) { st = fail(PD_ERR_CUDA, cudaGetErrorString(e)); break; }
    }
    if (st != PD_OK) break;
    if (K > 0 && steps == K) {
      std::vector<GraphKey> keys;
      for (pd_handle* h : g->hs) keys.push_back(group_key(h, steps, dto));
      if (!(g->gexec && keys == g->keys)) {
        group_release_graph(g);
        std::vector<long long> before;
        for (pd_handle* h : g->hs) before.push_back(h->launches);
        cudaGraph_t graph;
        cudaError_t e = cudaStreamBeginCapture(origin, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
          cudaGetLastError();  // of earlier calls
          group_issue(g, steps, dto);
          const cudaError_t le = cudaGetLastError();  // a launch that was refused
          e = cudaStreamEndCapture(origin, &graph);
          if (e == cudaSuccess && le != cudaSuccess) { cudaGraphDestroy(graph); e = le; }
        }
        g->nodes.assign(g->hs.size(), 0);
        for (size_t k = 0; k < g->hs.size(); k++) {
          g->nodes[k] = g->hs[k]->launches - before[k];
          g->hs[k]->launches = before[k];
        }
        if (e != cudaSuccess) { st = fail(PD_ERR_CUDA, std::string("group graph capture: ") + cudaGetErrorString(e)); break; }
        e = cudaGraphInstantiate(&g->gexec, graph, 0);
        cudaGraphDestroy(graph);
        if (e != cudaSuccess) {
          g->gexec = nullptr;
          st = fail(PD_ERR_CUDA, std::string("group graph instantiate: ") + cudaGetErrorString(e));
          break;
        }
        g->keys = keys;
      }
      cudaError_t e = cudaGraphLaunch(g->gexec, origin);
      if (e != cudaSuccess) { st = fail(PD_ERR_CUDA, std::string("group graph launch: ") + cudaGetErrorString(e)); break; }
      for (size_t k = 0; k < g->hs.size(); k++) g->hs[k]->launches += g->nodes[k];
    } else {
      group_issue(g, steps, dto);
      cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) { st = fail(PD_ERR_CUDA, cudaGetErrorString(e)); break; }
    }
    done += steps;
  }
  if (ms_total) cudaEventRecord(t1, origin);
  cudaError_t se = cudaStreamSynchronize(origin);
  if (st == PD_OK && se != cudaSuccess) st = fail(PD_ERR_CUDA, cudaGetErrorString(se));
  if (ms_total && st == PD_OK) {
    float x = 0.f;
    cudaEventElapsedTime(&x, t0, t1);
    *ms_total = x;
  }
  if (t0) cudaEventDestroy(t0);
  if (t1) cudaEventDestroy(t1);
  for (pd_handle* h : g->hs) {
    h->damage_valid = true;
    if (st == PD_OK) st = check_err(h);
  }
  return st;
}

extern "C" pd_status pd_run_vv_timed(pd_handle* h, int64_t first_step, int64_t n_steps, double dt,
                                     double* ms_total, double* ms_phase_a, double* ms_phase_b,
                                     double* ms_integrate) {
  if (!h) return fail(PD_ERR_ARG, "handle is NULL");
  if (n_steps <= 0) return fail(PD_ERR_ARG, "n_steps must be > 0");
  if (n_steps > (1 << 20)) return fail(PD_ERR_ARG, "at most 2^20 timed steps per call");
  PD_CUDA(cudaSetDevice(h->device));
  if (!ms_phase_a && !ms_phase_b && !ms_integrate) {
    // the run as pd_run_vv issues it (CUDA-graph blocks when pd_set_graph is on), between two
    // events on the handle's stream
    cudaEvent_t e0, e1;
    PD_CUDA(cudaEventCreate(&e0));
    cudaError_t ce = cudaEventCreate(&e1);
    if (ce != cudaSuccess) { cudaEventDestroy(e0); PD_CUDA(ce); }
    cudaEventRecord(e0, h->stream);
    pd_status st = run_vv(h, first_step, n_steps, dt, nullptr);
    cudaEventRecord(e1, h->stream);
    if (st == PD_OK || st == PD_ERR_NAN) {
      cudaError_t se = cudaEventSynchronize(e1);
      float x = 0.f;
      if (se == cudaSuccess) cudaEventElapsedTime(&x, e0, e1);
      if (ms_total) *ms_total = x;
      if (se != cudaSuccess && st == PD_OK)
        st = fail(PD_ERR_CUDA, std::string("pd_run_vv_timed: ") + cudaGetErrorString(se));
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return st;
  }
  const size_t nev = (size_t)4 * n_steps + 2;
  std::vector<cudaEvent_t> ev(nev);
  for (auto& e : ev) PD_CUDA(cudaEventCreate(&e));
  pd_status st = run_vv(h, first_step, n_steps, dt, &ev);
  if (st == PD_OK || st == PD_ERR_NAN) {
    PD_CUDA(cudaStreamSynchronize(h->stream));
    double ta = 0, tb = 0, ti = 0;
    float x;
    for (int64_t k = 0; k < n_steps; k++) {
      cudaEventElapsedTime(&x, ev[4 * k], ev[4 * k + 1]); ti += x;
      cudaEventElapsedTime(&x, ev[4 * k + 1], ev[4 * k + 2]); ta += x;
      cudaEventElapsedTime(&x, ev[4 * k + 2], ev[4 * k + 3]); tb += x;
    }
    cudaEventElapsedTime(&x, ev[nev - 2], ev[nev - 1]); ti += x;
    cudaEventElapsedTime(&x, ev[0], ev[nev - 1]);
    if (ms_total) *ms_total = x;
    if (ms_phase_a) *ms_phase_a = ta;
    if (ms_phase_b) *ms_phase_b = tb;
    if (ms_integrate) *ms_integrate = ti;
  }
  for (auto& e : ev) cudaEventDestroy(e);
  return st;
}

extern "C" pd_status pd_nan_step(pd_handle* h, int64_t* step) {
  if (!h || !step) return fail(PD_ERR_ARG, "handle or step is NULL");
  *step = h->nan_step;
  return PD_OK;
}

extern "C" pd_status pd_set_mapping(pd_handle* h, int32_t group, int32_t block) {
  if (!h) return fail(PD_ERR_ARG, "handle is NULL");
  if (block != 64 && block != 128 && block != 256) return fail(PD_ERR_ARG, "block must be 64, 128 or 256");
  if (group == 0) {
    if (h->precision != PD_PREC_FP64) return fail(PD_ERR_ARG, "the serial-order mapping (group 0) is FP64 only");
    PD_CUDA(cudaSetDevice(h->device));
    h->cfg.pipe = 0;
    PD_TRY(relayout(h, 1));
    h->cfg.exact = true;
    h->cfg.group = 1;
  } else {
    if (group != 1 && group != 2 && group != 4 && group != 8 && group != 16 && group != 32)
      return fail(PD_ERR_ARG, "group must be 0, 1, 2, 4, 8, 16 or 32");
    PD_CUDA(cudaSetDevice(h->device));
    PD_TRY(relayout(h, group));
    h->cfg.exact = false;
    h->cfg.group = group;
    if (group != 1) h->cfg.pipe = 0;
  }
  h->cfg.block = block;
  sum_anew(h);
  drop_graphs(h);
  return PD_OK;
}

// the phases that run on tiles: 1 for the first force kernel plus 2 for the second
static int tile_phases(const pd_handle* h) {
  int on = 0;
  for (int phase = 1; phase <= (h->material == PD_MAT_BB ? 1 : 2); phase++) {
    const bool t = h->precision == PD_PREC_FP64 ? !h->cfg.exact && tile64_supported(h->d, phase)
                                                : !runs_tma(h) && force32_on_tiles(h->d, phase);
    if (t) on |= phase;
  }
  return on;
}

extern "C" pd_status pd_tile_info(pd_handle* h, int32_t* tile_points, int32_t* classes, int32_t* phases) {
  if (!h) return fail(PD_ERR_ARG, "handle is NULL");
  if (tile_points) *tile_points = h->d.tile_pt ? h->d.tile_cap : 0;
  if (classes) *classes = h->d.ncls;
  if (phases) *phases = tile_phases(h);
  return PD_OK;
}

extern "C" pd_status pd_autotune(pd_handle* h, int32_t* group_out, int32_t* block_out) {
  if (!h) return fail(PD_ERR_ARG, "handle is NULL");
  PD_CUDA(cudaSetDevice(h->device));
  const LaunchCfg keep = h->cfg;
  cudaEvent_t e0, e1;
  PD_CUDA(cudaEventCreate(&e0));
  PD_CUDA(cudaEventCreate(&e1));
  struct Cand { float ms; LaunchCfg c; };
  std::vector<Cand> cands;
  // five evaluations of the current configuration after one warm-up
  auto time_cfg = [&](float* out) -> pd_status {
    launch_force(h, 0, 0);
    cudaEventRecord(e0, h->stream);
    for (int r = 0; r < 5; r++) launch_force(h, 0, 0);
    cudaEventRecord(e1, h->stream);
    cudaError_t e = cudaEventSynchronize(e1);
    if (e != cudaSuccess) return fail(PD_ERR_CUDA, cudaGetErrorString(e));
    cudaEventElapsedTime(out, e0, e1);
    return PD_OK;
  };
  auto give_up = [&](pd_status st) {
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return st;
  };
  // force evaluations are idempotent at fixed positions: bonds that broke stay broken and
  // every output is recomputed
  const bool f32 = h->precision == PD_PREC_FP32_KAHAN, corr = h->material == PD_MAT_CMAT;
  for (int G : {1, 4, 32}) {
    // the variants to time: plain loads, then (FP32 BB / OSB) the two-row kernels, then (one lane per point)
    // the packed kernels and the TMA-staged bond stream, which wants another order of the points
    std::vector<int> pipes{0};
    if (f32 && !corr) pipes.push_back(4);
    if (f32 && G == 1) {
      pipes.push_back(5);
      if (!corr) pipes.insert(pipes.end(), {1, 2, 3});
    }
    for (int pipe : pipes) {
      h->cfg.group = G; h->cfg.exact = false; h->cfg.pipe = pipe;
      pd_status st = relayout(h, G);
      if (st == PD_ERR_OOM) break;  // no room for a second layout
      if (st != PD_OK) return give_up(st);
      const bool tma = pipe >= 1 && pipe <= 3;
      if (tma && !tma_supported(h->d)) continue;
      if (pipe == 5 && !packed_supported(h->d, 1)) continue;
      // where every phase runs the packed kernels the plain variants are the same ones (correspondence: 0
      // has sums of its own); on tiles the block size is the tile's
      const bool bb = h->material == PD_MAT_BB;
      if (G == 1 && f32 && !corr && (pipe == 0 || pipe == 4) && packed_supported(h->d, 1) &&
          (bb || packed_supported(h->d, 2)))
        continue;
      const bool tiles = tile_phases(h) == (bb ? 1 : 3);
      for (int B : {128, 256}) {
        if (B == 256 && (tma || tiles)) continue;
        h->cfg.block = B;
        float ms;
        st = time_cfg(&ms);
        if (st != PD_OK) return give_up(st);
        cands.push_back({ms, h->cfg});
      }
    }
  }
  // the three fastest are timed twice more, interleaved, and keep their best time: one window
  // of five evaluations moves with the clocks of a power-capped GPU
  std::sort(cands.begin(), cands.end(), [](const Cand& a, const Cand& b) { return a.ms < b.ms; });
  if (cands.size() > 3) cands.resize(3);
  for (int round = 0; round < 2 && cands.size() > 1; round++)
    for (auto& c : cands) {
      h->cfg = c.c;
      if (relayout(h, c.c.group) != PD_OK) continue;
      float ms;
      pd_status ts = time_cfg(&ms);
      if (ts != PD_OK) return give_up(ts);
      c.ms = std::min(c.ms, ms);
    }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  LaunchCfg bestc = keep;
  float best = INFINITY;
  for (const auto& c : cands)
    if (c.ms < best) { best = c.ms; bestc = c.c; }
  h->cfg = bestc;
  sum_anew(h);
  PD_TRY(relayout(h, bestc.group));
  drop_graphs(h);
  if (group_out) *group_out = bestc.group;
  if (block_out) *block_out = bestc.block;
  return check_err(h);
}

extern "C" pd_status pd_set_graph(pd_handle* h, int32_t steps_per_graph) {
  if (!h) return fail(PD_ERR_ARG, "handle is NULL");
  if (steps_per_graph < 0 || steps_per_graph > 4096) return fail(PD_ERR_ARG, "0 <= steps_per_graph <= 4096");
  h->graph_steps = steps_per_graph;
  drop_graphs(h);
  return PD_OK;
}

extern "C" pd_status pd_info(pd_handle* h, int64_t* n_points, int64_t* n_bonds, int32_t* symmetric) {
  if (!h) return fail(PD_ERR_ARG, "handle is NULL");
  if (n_points) *n_points = h->n;
  if (n_bonds) *n_bonds = h->nb;
  if (symmetric) *symmetric = h->d.sym;
  return PD_OK;
}

extern "C" pd_status pd_launch_count(pd_handle* h, int64_t* count) {
  if (!h || !count) return fail(PD_ERR_ARG, "handle or count is NULL");
  *count = h->launches;
  return PD_OK;
}

extern "C" pd_status pd_stream(pd_handle* h, void** stream) {
  if (!h || !stream) return fail(PD_ERR_ARG, "handle or stream is NULL");
  *stream = (void*)h->stream;
  return PD_OK;
}

extern "C" pd_status pd_break_bonds(pd_handle* h, const uint8_t* set_a, const uint8_t* set_b) {
  if (!h || (h->n > 0 && (!set_a || !set_b))) return fail(PD_ERR_ARG, "handle or point sets are NULL");
  PD_CUDA(cudaSetDevice(h->device));
  const long long n = h->n;
  if (n == 0) return PD_OK;
  for (long long i = 0; i < n; i++)
    if (set_a[i] && set_b[i]) return fail(PD_ERR_ARG, "point sets intersect");
  unsigned char* tmp = nullptr;
  PD_CUDA(cudaMalloc(&tmp, 2 * n));
  cudaError_t e = h2d(tmp, set_a, n, h->stream);
  if (e == cudaSuccess) e = h2d(tmp + n, set_b, n, h->stream);
  if (e == cudaSuccess) {
    launch_break_sets(h->d, tmp, tmp + n, h->stream);
    h->kfull = true;
    launch_count_active(h->d, h->stream);
    e = cudaStreamSynchronize(h->stream);
  }
  cudaFree(tmp);
  if (e != cudaSuccess) return fail(PD_ERR_CUDA, cudaGetErrorString(e));
  h->damage_valid = true;
  drop_graphs(h);
  return PD_OK;
}

extern "C" pd_status pd_count_near_critical(pd_handle* h, double tol, int64_t* count) {
  if (!h || !count) return fail(PD_ERR_ARG, "NULL argument");
  if (!(tol >= 0)) return fail(PD_ERR_ARG, "tol must be >= 0");
  PD_CUDA(cudaSetDevice(h->device));
  *count = 0;
  if (h->n == 0) return PD_OK;
  unsigned long long* dc = nullptr;
  PD_CUDA(cudaMalloc(&dc, sizeof(unsigned long long)));
  cudaError_t e = cudaMemsetAsync(dc, 0, sizeof(unsigned long long), h->stream);
  if (e == cudaSuccess) {
    launch_near_critical(h->d, h->g, tol, dc, h->stream);
    e = cudaGetLastError();
  }
  unsigned long long c = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&c, dc, sizeof(c), cudaMemcpyDeviceToHost, h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  cudaFree(dc);
  if (e != cudaSuccess) return fail(PD_ERR_CUDA, cudaGetErrorString(e));
  *count = (int64_t)c;
  return PD_OK;
}

extern "C" pd_status pd_break_random_pairs(pd_handle* h, double fraction, uint64_t seed) {
  return pd_break_random_pairs_ids(h, fraction, seed, nullptr);
}

extern "C" pd_status pd_break_random_pairs_ids(pd_handle* h, double fraction, uint64_t seed,
                                               const int64_t* point_ids) {
  if (!h) return fail(PD_ERR_ARG, "handle is NULL");
  if (!(fraction >= 0 && fraction <= 1)) return fail(PD_ERR_ARG, "fraction must be in [0, 1]");
  PD_CUDA(cudaSetDevice(h->device));
  if (h->n == 0) return PD_OK;
  long long* gid = nullptr;
  if (point_ids) {
    PD_TRY(dalloc(h, &gid, h->n));
    PD_CUDA(h2d(gid, point_ids, sizeof(long long) * h->n, h->stream));
  }
  launch_break_random(h->d, fraction, (unsigned long long)seed, gid, h->stream);
  h->kfull = true;
  launch_count_active(h->d, h->stream);
  PD_CUDA(cudaStreamSynchronize(h->stream));
  dfree(h, gid);
  h->damage_valid = true;
  PD_TRY(check_symmetry(h));
  drop_graphs(h);
  return PD_OK;
}

extern "C" pd_status pd_get_mapping(pd_handle* h, int32_t* group, int32_t* block, int32_t* pipe) {
  if (!h) return fail(PD_ERR_ARG, "handle is NULL");
  if (group) *group = h->cfg.exact ? 0 : h->cfg.group;
  if (block) *block = h->cfg.block;
  if (pipe) *pipe = h->cfg.pipe;
  return PD_OK;
}

extern "C" pd_status pd_set_pipeline(pd_handle* h, int32_t pipe) {
  if (!h) return fail(PD_ERR_ARG, "handle is NULL");
  if (pipe < 0 || pipe > 5) return fail(PD_ERR_ARG, "pipe must be 0 to 5");
  if (pipe == 4 && (h->precision != PD_PREC_FP32_KAHAN || h->material == PD_MAT_CMAT))
    return fail(PD_ERR_ARG, "the two-row kernels are the FP32 BB and OSB ones");
  if (pipe == 5 && h->precision != PD_PREC_FP32_KAHAN)
    return fail(PD_ERR_ARG, "the packed-pair kernels are FP32 ones");
  if (pipe >= 1 && pipe <= 3 && (h->precision != PD_PREC_FP32_KAHAN || !tma_supported(h->d)))
    return fail(PD_ERR_ARG, "the staged bond stream needs the FP32 path, one lane per point and BB or OSB");
  PD_CUDA(cudaSetDevice(h->device));
  h->cfg.pipe = pipe;
  sum_anew(h);
  drop_graphs(h);
  const pd_status st = relayout(h, h->d.lg);
  return st == PD_ERR_OOM ? PD_OK : st;  // any order will do
}

// pd_esc_init: the bond factors have no place in the tiles
pd_status pd_without_tiles(pd_handle* h) {
  h->esc = true;
  const pd_status st = relayout(h, h->d.lg);
  return st == PD_ERR_OOM ? PD_OK : st;
}

// helpers shared with pd_nk.cu
pd_status pd_set_ctrl(pd_handle* h, size_t off, const void* src, size_t bytes) {
  return set_ctrl(h, off, src, bytes);
}
pd_status pd_clear_error(pd_handle* h) { return clear_error(h); }
pd_status pd_check_err(pd_handle* h) { return check_err(h); }
int pd_launch_force(pd_handle* h, int kstep, int phase) { return launch_force(h, kstep, phase); }
