// C-ABI implementation: device context, state upload/download, the trend and
// the RK4 stepper (one captured CUDA graph per step).
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../../include/wavetrisk_gpu.h"
#include "trisk_kernels.cuh"
#include "trisk_mixed.cuh"
#include "trisk_pipe.cuh"
#include "trisk_tma.cuh"
#include "wt_handle.cuh"

using namespace wtk;

namespace {

constexpr int TPB = 256;

inline unsigned blocks_for(int64_t n, int tpb = TPB) { return (unsigned)((n + tpb - 1) / tpb); }

}  // namespace


int wt_handle_fail(const char* where, cudaError_t e) {
  std::fprintf(stderr, "wavetrisk_gpu: %s: %s\n", where, cudaGetErrorString(e));
  return e == cudaErrorMemoryAllocation ? WT_ERR_ALLOC : WT_ERR_CUDA;
}

#define CK(x)                                         \
  do {                                                \
    cudaError_t e_ = (x);                             \
    if (e_ != cudaSuccess) return wt_handle_fail(#x, e_); \
  } while (0)

static int dev_copy(double** dst, const double* src, int64_t count) {
  CK(cudaMalloc(dst, count * sizeof(double)));
  if (src)
    CK(cudaMemcpy(*dst, src, count * sizeof(double), cudaMemcpyHostToDevice));
  else
    CK(cudaMemset(*dst, 0, count * sizeof(double)));
  return WT_OK;
}

static int dev_zero(double** dst, int64_t count) { return dev_copy(dst, nullptr, count); }

// Tensor maps of the trend inputs on the top level: dims (P, P, 10 lozenges,
// planes), boxes of TB_X x TB_Y nodes.  The encoder is taken from the driver
// through the runtime, so the library does not link libcuda directly.
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  if (!encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q{};
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
    if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !fn) {
      std::fprintf(stderr, "wavetrisk_gpu: cuTensorMapEncodeTiled unavailable\n");
      return nullptr;
    }
    encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }
  return encode;
}

// Tensor map of a top-level field of `planes` planes of NN values (double or
// float), boxes of bx x by nodes.
template <class T>
static bool top_map(wt_handle* h, CUtensorMap* m, const T* base, int planes, int bx = TB_X, int by = TB_Y) {
  PFN_cuTensorMapEncodeTiled_v12000 encode = tensor_map_encoder();
  if (!encode) return false;
  const DevLevel& D = h->top();
  const cuuint64_t sz = sizeof(T);
  const cuuint64_t dims[4] = {(cuuint64_t)D.P, (cuuint64_t)D.P, 10, (cuuint64_t)planes};
  const cuuint64_t strides[3] = {(cuuint64_t)D.P * sz, (cuuint64_t)D.P * D.P * sz, (cuuint64_t)D.NN * sz};
  const cuuint32_t box[4] = {(cuuint32_t)bx, (cuuint32_t)by, 1, 1};
  const cuuint32_t elem[4] = {1, 1, 1, 1};
  return encode(m, sz == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4,
                const_cast<T*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The step1 input maps of a top-level state (m, t, v) with the top level's means and geometry.
static bool step1_maps(wt_handle* h, const double* m, const double* t, const double* v, Step1Maps* S) {
  const DevLevel& D = h->top();
  const int nz = h->nz;
  auto mk = [&](CUtensorMap* map, const double* base, int planes) { return top_map(h, map, base, planes); };
  return mk(&S->mass, m, nz) && mk(&S->temp, t, nz) && mk(&S->velo, v, 3 * nz) && mk(&S->mean_m, h->mean_m, nz) &&
         mk(&S->mean_t, h->mean_t, nz) && mk(&S->len, D.len, 3) && mk(&S->ped, D.pedlen, 3) &&
         mk(&S->part, D.part, 6) && mk(&S->cor, D.coriolis, 2);
}

int wt_make_step1_maps(wt_handle* h, const double* m, const double* t, const double* v, wtk::Step1Maps* out) {
  if (h->trend_variant != 0) return WT_ERR_STATE;
  return step1_maps(h, m, t, v, out) ? WT_OK : WT_ERR_CUDA;
}

static bool trend_maps(wt_handle* h, const double* hfm, const double* hft, const double* qe,
                       const double* theta, const double* bern, const double* phik, TrendMaps* M) {
  const DevLevel& D = h->top();
  const int nz = h->nz;
  return top_map(h, &M->hfm, hfm, 3 * nz) && top_map(h, &M->hft, hft, 3 * nz) && top_map(h, &M->qe, qe, 3 * nz) &&
         top_map(h, &M->theta, theta, nz) && top_map(h, &M->bern, bern, nz) && top_map(h, &M->phik, phik, nz) &&
         top_map(h, &M->part, D.part, 6) && top_map(h, &M->hinv, D.hex_inv, 1);
}

int wt_make_trend_maps(wt_handle* h, const double* hfm, const double* hft, const double* qe, const double* theta,
                       const double* bern, const double* phik, wtk::TrendMaps* M) {
  if (h->trend_variant != 0) return WT_ERR_STATE;
  return trend_maps(h, hfm, hft, qe, theta, bern, phik, M) ? WT_OK : WT_ERR_CUDA;
}

// Tensor maps and launch limits of the TMA-staged kernels on the top level.
static int make_trend_maps(wt_handle* h) {
  const int nz = h->nz;
  bool ok = trend_maps(h, h->hfm, h->hft, h->qe, h->theta, h->bern, h->phik, &h->maps);
  auto mk = [&](CUtensorMap* m, const double* base, int planes) {
    return top_map(h, m, base, planes, PBX, PipeTile::BY);
  };
  TrendMapsD& M = h->pmaps;
  ok = ok && mk(&M.hfm, h->hfm, 3 * nz) && mk(&M.hft, h->hft, 3 * nz) && mk(&M.qe, h->qe, 3 * nz) &&
       mk(&M.theta, h->theta, nz) && mk(&M.bern, h->bern, nz) && mk(&M.phik, h->phik, nz);
  double* SM[3] = {h->mass, h->m1, h->m2};
  double* ST[3] = {h->temp, h->t1, h->t2};
  double* SV[3] = {h->velo, h->v1, h->v2};
  for (int b = 0; b < 3 && ok; ++b) {
    PipeStateMaps& S = h->p1maps[b];
    ok = step1_maps(h, SM[b], ST[b], SV[b], &h->s1maps[b]) && mk(&S.mass, SM[b], nz) && mk(&S.temp, ST[b], nz) &&
         mk(&S.velo, SV[b], 3 * nz) && mk(&S.mean_m, h->mean_m, nz) && mk(&S.mean_t, h->mean_t, nz) &&
         mk(&S.phik, h->phik, nz) && mk(&S.pterm, h->pterm, nz);
  }
  if (!ok) {
    std::fprintf(stderr, "wavetrisk_gpu: tensor map encoding failed\n");
    return WT_ERR_CUDA;
  }
  int dev = 0;
  CK(cudaGetDevice(&dev));
  CK(cudaDeviceGetAttribute(&h->pipe_slots, cudaDevAttrMultiProcessorCount, dev));  // one block a SM
  const auto smem = cudaFuncAttributeMaxDynamicSharedMemorySize;
  CK(cudaFuncSetAttribute(k_step1_tma, smem, STEP1_TMA_SMEM));
  CK(cudaFuncSetAttribute(k_trend_tma<MODE_RK>, smem, TREND_TMA_SMEM));
  CK(cudaFuncSetAttribute(k_trend_tma<MODE_TREND>, smem, TREND_TMA_SMEM));
  CK(cudaFuncSetAttribute(k_trend_tma<MODE_ML>, smem, TREND_TMA_SMEM));
  CK(cudaFuncSetAttribute(k_step1_pipe<double>, smem, Step1Pipe<double>::SMEM));
  CK(cudaFuncSetAttribute(k_step1_pipe<float>, smem, Step1Pipe<float>::SMEM));
  CK(cudaFuncSetAttribute(k_trend_pipe<double, MODE_RK>, smem, TrendPipe<double, MODE_RK>::SMEM));
  CK(cudaFuncSetAttribute(k_trend_pipe<double, MODE_TREND>, smem, TrendPipe<double, MODE_TREND>::SMEM));
  CK(cudaFuncSetAttribute(k_trend_pipe<float, MODE_RK>, smem, TrendPipe<float, MODE_RK>::SMEM));
  CK(cudaFuncSetAttribute(k_trend_pipe<float, MODE_TREND>, smem, TrendPipe<float, MODE_TREND>::SMEM));
  return WT_OK;
}

// The pipelined kernels' ghost lists of the top level, from its halo lists and remaps.
static int make_ghost_lists(wt_handle* h, const DevLevel& D, const std::vector<int2>& hn, const std::vector<int3>& he,
                            const std::vector<int>& nsrc, const std::vector<int>& esrc) {
  std::vector<int2> nodes, edges, outer;
  const int NN = (int)D.NN, P = D.P;
  auto within = [&](int x, int hi) {  // node slot x lies in [-1, hi]^2
    const int r = x % (P * P), i = r % P - 2, j = r / P - 2;
    return i >= -1 && j >= -1 && i <= hi && j <= hi;
  };
  for (const int2& e : hn)
    if (nsrc[e.x] != e.x && within(e.x, D.n + 1)) nodes.push_back(make_int2(e.x, 2 * nsrc[e.x]));
  for (const int3& e : he) {
    const int x = e.x % NN;
    if (esrc[e.x] == 2 * e.x || !within(x, D.n + 1)) continue;
    (within(x, D.n) ? edges : outer).push_back(make_int2(e.x, esrc[e.x]));
  }
  h->ghosts.n_f = (int)edges.size();
  edges.insert(edges.end(), outer.begin(), outer.end());
  int2 *dn = nullptr, *de = nullptr;
  CK(cudaMalloc(&dn, sizeof(int2) * std::max<size_t>(1, nodes.size())));
  h->ghosts.nodes = dn;
  CK(cudaMalloc(&de, sizeof(int2) * std::max<size_t>(1, edges.size())));
  h->ghosts.edges = de;
  CK(cudaMemcpy(dn, nodes.data(), sizeof(int2) * nodes.size(), cudaMemcpyHostToDevice));
  CK(cudaMemcpy(de, edges.data(), sizeof(int2) * edges.size(), cudaMemcpyHostToDevice));
  h->ghosts.n_nodes = (int)nodes.size();
  h->ghosts.n_edges = (int)edges.size();
  return WT_OK;
}

// The pipelined kernels copy FP32 planes only where a row of the padded level is a
// multiple of 16 bytes (from level 2 up); the L1 kernels take any level.
static bool f32_staged(wt_handle* h) { return h->trend_variant == 0 && h->top().P % 4 == 0; }

// Trend input maps of the FP32 flux arrays a (qe, hfm, hft, ke, theta).
static int make_f32_maps(wt_handle* h, float* const* a, TrendMapsF& M) {
  const int nz = h->nz;
  auto mk = [&](CUtensorMap* m, const float* base, int planes) { return top_map(h, m, base, planes, FBX, PipeTile::BY); };
  const bool ok = mk(&M.qe, a[0], 3 * nz) && mk(&M.hfm, a[1], 3 * nz) && mk(&M.hft, a[2], 3 * nz) && mk(&M.ke, a[3], nz) &&
                  mk(&M.theta, a[4], nz) && top_map(h, &M.phik, h->phik, nz, PBX, PipeTile::BY) &&
                  top_map(h, &M.pterm, h->pterm, nz, PBX, PipeTile::BY);
  if (!ok) {
    std::fprintf(stderr, "wavetrisk_gpu: tensor map encoding failed\n");
    return WT_ERR_CUDA;
  }
  return WT_OK;
}

extern "C" {

int wt_create(const wt_grid_desc* desc, wt_handle** out) {
  if (!desc || !out || !desc->levels || desc->nz < 1 || desc->level_end < desc->level_start) return WT_ERR_ARG;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return WT_ERR_NO_DEVICE;
  wt_handle* h = new wt_handle();
  h->nz = desc->nz;
  h->ph = Phys{desc->grav, desc->ref_density, desc->p_top};
  h->level_start = desc->level_start;
  h->level_end = desc->level_end;
  const int nlev = desc->level_end - desc->level_start + 1;
  h->lev.resize(nlev);
  int rc = WT_OK;
  // Kernel family: TMA-staged tiles from n = 64 up; below that the tiles are mostly
  // empty and the L1 kernels are faster (J5 x 8, 100 steps: 10.4 ms against 11.4).
  // WAVETRISK_TREND_KERNEL=tma|plain forces either.
  h->trend_variant = desc->level_end >= 6 ? 0 : 1;
  if (const char* tv = std::getenv("WAVETRISK_TREND_KERNEL")) {
    if (std::strcmp(tv, "tma") == 0) h->trend_variant = 0;
    if (std::strcmp(tv, "plain") == 0) h->trend_variant = 1;
  }
  for (int q = 0; q < nlev && rc == WT_OK; ++q) {
    const wt_level_desc& ld = desc->levels[q];
    DevLevel& D = h->lev[q];
    if (ld.n != (1 << ld.level) || ld.P != ld.n + 4 || ld.NN != (int64_t)10 * ld.P * ld.P) { rc = WT_ERR_ARG; break; }
    if (6 * ld.NN >= (int64_t)1 << 31) { rc = WT_ERR_ARG; break; }  // 32-bit offsets inside one layer
    D.level = ld.level;
    D.n = ld.n;
    D.P = ld.P;
    D.NN = ld.NN;
    const int64_t NN = ld.NN;
    if ((rc = dev_copy(&D.len, ld.len, 3 * NN))) break;
    if ((rc = dev_copy(&D.pedlen, ld.pedlen, 3 * NN))) break;
    if ((rc = dev_copy(&D.part, ld.part, 6 * NN))) break;
    if ((rc = dev_copy(&D.hex_inv, ld.hex_inv, NN))) break;
    if ((rc = dev_copy(&D.triarea, ld.triarea, 2 * NN))) break;
    if ((rc = dev_copy(&D.coriolis, ld.coriolis, 2 * NN))) break;
    if ((rc = dev_copy(&D.overl_a, ld.overl_a, 4 * NN))) break;
    if ((rc = dev_copy(&D.topo, ld.topo, NN))) break;
    if (ld.iu_wgt && (rc = dev_copy(&D.iu_wgt, ld.iu_wgt, 9 * NN))) break;
    if (ld.overl_split && (rc = dev_copy(&D.overl_split, ld.overl_split, 2 * NN))) break;
    if (ld.rf_wgt && (rc = dev_copy(&D.rf_wgt, ld.rf_wgt, 3 * NN))) break;
    std::vector<int2> hn(ld.n_halo_node);
    for (int64_t k = 0; k < ld.n_halo_node; ++k) {
      int64_t a = ld.halo_node[2 * k], b = ld.halo_node[2 * k + 1];
      if (a < 0 || b < 0 || a >= NN || b >= NN) { rc = WT_ERR_ARG; break; }
      hn[k] = make_int2((int)a, (int)b);
    }
    if (rc) break;
    std::vector<int3> he(ld.n_halo_edge);
    for (int64_t k = 0; k < ld.n_halo_edge; ++k) {
      int64_t a = ld.halo_edge[3 * k], b = ld.halo_edge[3 * k + 1], s = ld.halo_edge[3 * k + 2];
      if (a < 0 || b < 0 || a >= 3 * NN || b >= 3 * NN) { rc = WT_ERR_ARG; break; }
      he[k] = make_int3((int)a, (int)b, (int)s);
    }
    if (rc) break;
    D.n_hn = (int)hn.size();
    D.n_he = (int)he.size();
    cudaError_t e;
    if ((e = cudaMalloc(&D.hn, sizeof(int2) * std::max<size_t>(1, hn.size()))) != cudaSuccess) { rc = wt_handle_fail("halo", e); break; }
    if ((e = cudaMalloc(&D.he, sizeof(int3) * std::max<size_t>(1, he.size()))) != cudaSuccess) { rc = wt_handle_fail("halo", e); break; }
    cudaMemcpy(D.hn, hn.data(), sizeof(int2) * hn.size(), cudaMemcpyHostToDevice);
    cudaMemcpy(D.he, he.data(), sizeof(int3) * he.size(), cudaMemcpyHostToDevice);
    // read remaps: a ghost reads the node / signed edge its copy entry names
    std::vector<int> nsrc(NN), esrc(3 * NN);
    for (int64_t k = 0; k < NN; ++k) nsrc[k] = (int)k;
    for (auto& x : hn) nsrc[x.x] = x.y;
    for (int64_t k = 0; k < 3 * NN; ++k) esrc[k] = (int)(2 * k);
    for (auto& x : he) esrc[x.x] = 2 * x.y + (x.z < 0 ? 1 : 0);
    if ((e = cudaMalloc(&D.nsrc, sizeof(int) * NN)) != cudaSuccess) { rc = wt_handle_fail("remap", e); break; }
    if ((e = cudaMalloc(&D.esrc, sizeof(int) * 3 * NN)) != cudaSuccess) { rc = wt_handle_fail("remap", e); break; }
    cudaMemcpy(D.nsrc, nsrc.data(), sizeof(int) * NN, cudaMemcpyHostToDevice);
    cudaMemcpy(D.esrc, esrc.data(), sizeof(int) * 3 * NN, cudaMemcpyHostToDevice);
    if (h->trend_variant == 0 && D.level == h->level_end && (rc = make_ghost_lists(h, D, hn, he, nsrc, esrc))) break;
  }
  if (rc == WT_OK) {
    // Prognostic state and RK/trend work arrays on level_end.
    DevLevel& D = h->top();
    const int64_t NN = D.NN, nn = (int64_t)h->nz * NN, ne = 3 * nn;
    double** node_arrays[] = {&h->mass, &h->temp, &h->mean_m, &h->mean_t, &h->m1, &h->t1, &h->m2, &h->t2,
                              &h->dm, &h->dt, &h->bern, &h->phik, &h->pterm, &h->theta};
    for (double** p : node_arrays)
      if ((rc = dev_zero(p, nn))) break;
    double** edge_arrays[] = {&h->velo, &h->v1, &h->v2, &h->dv, &h->qe, &h->hfm, &h->hft};
    if (rc == WT_OK)
      for (double** p : edge_arrays)
        if ((rc = dev_zero(p, ne))) break;
    if (rc == WT_OK) {
      // The handle's stream carries the critical path of a step (the finest
      // level's step1 and trend, the restrictions, the coarser trends, the
      // velocity reconstruction); the side streams that run beside it (coarser
      // levels' step1, forward wavelets, scalar reconstruction) keep the default
      // priority, so the block scheduler serves this stream's blocks first.
      int least = 0, greatest = 0;
      cudaError_t e = cudaDeviceGetStreamPriorityRange(&least, &greatest);
      if (e == cudaSuccess) e = cudaStreamCreateWithPriority(&h->stream, cudaStreamNonBlocking, greatest);
      if (e != cudaSuccess) rc = wt_handle_fail("stream", e);
    }
    if (rc == WT_OK) {
      cudaError_t e = cudaMalloc(&h->dflag, sizeof(int));
      if (e == cudaSuccess) e = cudaMemset(h->dflag, 0, sizeof(int));
      if (e != cudaSuccess) rc = wt_handle_fail("flag", e);
    }
    if (rc == WT_OK) rc = make_trend_maps(h);
  }
  if (rc != WT_OK) {
    wt_destroy(h);
    return rc;
  }
  *out = h;
  return WT_OK;
}

int wt_destroy(wt_handle* h) {
  if (!h) return WT_OK;
  if (h->graph_exec) cudaGraphExecDestroy(h->graph_exec);
  for (auto& D : h->lev) D.release();
  double* arrays[] = {h->mass, h->temp, h->velo, h->mean_m, h->mean_t, h->m1, h->t1, h->v1, h->m2, h->t2, h->v2,
                      h->dm, h->dt, h->dv, h->qe, h->hfm, h->hft, h->bern, h->phik, h->pterm, h->theta};
  for (double* p : arrays)
    if (p) cudaFree(p);
  float* arrays32[] = {h->qe32, h->hfm32, h->hft32, h->ke32, h->theta32};
  for (float* p : arrays32)
    if (p) cudaFree(p);
  h->release_extra();
  cudaFree(const_cast<int2*>(h->ghosts.nodes));
  cudaFree(const_cast<int2*>(h->ghosts.edges));
  if (h->dflag) cudaFree(h->dflag);
  if (h->stream) cudaStreamDestroy(h->stream);
  delete h;
  return WT_OK;
}

void* wt_stream(wt_handle* h) { return h ? (void*)h->stream : nullptr; }

// WT_TUNE_FLUX_PRECISION (wt_tune): the single-level stepper's flux stencils
// in FP64 (64) or FP32 (32).  The FP32 work arrays are allocated on the first
// switch to 32; the captured step graph is dropped so the next step records
// the other kernels.
int wt_set_flux_precision(wt_handle* h, int bits) {
  if (!h || (bits != 64 && bits != 32)) return WT_ERR_ARG;
  if (bits == h->flux_bits) return WT_OK;
  if (bits == 32 && !h->qe32) {
    // all or nothing: qe32 says that the five arrays and the maps are there
    const int64_t nn = (int64_t)h->nz * h->top().NN;
    const int64_t sizes[5] = {3 * nn, 3 * nn, 3 * nn, nn, nn};
    float* a[5] = {};
    int rc = WT_OK;
    for (int q = 0; q < 5 && rc == WT_OK; ++q) {
      cudaError_t e = cudaMalloc(&a[q], sizeof(float) * sizes[q]);
      if (e == cudaSuccess) e = cudaMemset(a[q], 0, sizeof(float) * sizes[q]);
      if (e != cudaSuccess) rc = wt_handle_fail("flux fp32 arrays", e);
    }
    if (rc == WT_OK && f32_staged(h)) rc = make_f32_maps(h, a, h->fmaps);
    if (rc != WT_OK) {
      for (float* p : a) cudaFree(p);
      cudaGetLastError();  // reported: a later call must not find the failed allocation
      return rc;
    }
    h->qe32 = a[0];
    h->hfm32 = a[1];
    h->hft32 = a[2];
    h->ke32 = a[3];
    h->theta32 = a[4];
  }
  if (h->graph_exec) {
    cudaGraphExecDestroy(h->graph_exec);
    h->graph_exec = nullptr;
  }
  h->flux_bits = bits;
  return WT_OK;
}

int wt_synchronize(wt_handle* h) {
  if (!h) return WT_ERR_ARG;
  CK(cudaStreamSynchronize(h->stream));
  return WT_OK;
}

int wt_clear_status(wt_handle* h) {
  if (!h) return WT_ERR_ARG;
  CK(cudaStreamSynchronize(h->stream));
  if (h->dflag) CK(cudaMemset(h->dflag, 0, sizeof(int)));
  h->sticky = WT_OK;
  return WT_OK;
}

// Test-only: the TMA kernels of the next steps declare more bytes than their
// copies deliver and take their wait-timeout path (value 1), or run normally
// (0).  The captured step graphs hold the flag, so they are dropped here.
int wt_set_tma_inject(wt_handle* h, int value) {
  if (!h) return WT_ERR_ARG;
  if (value != 0 && value != 1) return WT_ERR_ARG;
  if (h->tma_inject == value) return WT_OK;
  CK(cudaStreamSynchronize(h->stream));
  h->tma_inject = value;
  if (h->graph_exec) {
    cudaGraphExecDestroy(h->graph_exec);
    h->graph_exec = nullptr;
  }
  return WT_OK;
}

int wt_status(wt_handle* h) {
  if (!h) return WT_ERR_ARG;
  CK(cudaStreamSynchronize(h->stream));
  CK(cudaGetLastError());
  if (h->dflag && h->sticky == WT_OK) {
    int f = 0;
    CK(cudaMemcpy(&f, h->dflag, sizeof(int), cudaMemcpyDeviceToHost));
    if (f) h->sticky = WT_ERR_TIMEOUT;
  }
  return h->sticky;
}

int wt_upload_state(wt_handle* h, const double* mass, const double* temp, const double* velo, const double* mean_m,
                    const double* mean_t) {
  if (!h || !mass || !temp || !velo) return WT_ERR_ARG;
  const int64_t nn = (int64_t)h->nz * h->top().NN;
  CK(cudaMemcpyAsync(h->mass, mass, nn * 8, cudaMemcpyHostToDevice, h->stream));
  CK(cudaMemcpyAsync(h->temp, temp, nn * 8, cudaMemcpyHostToDevice, h->stream));
  CK(cudaMemcpyAsync(h->velo, velo, 3 * nn * 8, cudaMemcpyHostToDevice, h->stream));
  if (mean_m) CK(cudaMemcpyAsync(h->mean_m, mean_m, nn * 8, cudaMemcpyHostToDevice, h->stream));
  if (mean_t) CK(cudaMemcpyAsync(h->mean_t, mean_t, nn * 8, cudaMemcpyHostToDevice, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  h->state_halo_done = false;
  return WT_OK;
}

int wt_download_state(wt_handle* h, double* mass, double* temp, double* velo) {
  if (!h || !mass || !temp || !velo) return WT_ERR_ARG;
  const int64_t nn = (int64_t)h->nz * h->top().NN;
  {
    // ghosts are read through remaps on the device; fill them for the host
    DevLevel& D = h->top();
    int64_t nt = (int64_t)(2 * D.n_hn + D.n_he) * h->nz;
    k_halo_state<<<blocks_for(nt), TPB, 0, h->stream>>>(h->nz, D.NN, D.hn, D.n_hn, D.he, D.n_he, h->mass, h->temp, h->velo);
  }
  CK(cudaMemcpyAsync(mass, h->mass, nn * 8, cudaMemcpyDeviceToHost, h->stream));
  CK(cudaMemcpyAsync(temp, h->temp, nn * 8, cudaMemcpyDeviceToHost, h->stream));
  CK(cudaMemcpyAsync(velo, h->velo, 3 * nn * 8, cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return WT_OK;
}

}  // extern "C"

// Optional per-launch timing (wt_profile_rk4): events recorded around each
// kernel on the handle's stream.
struct KTimer {
  std::vector<cudaEvent_t> ev;
  std::vector<int> ids;
  cudaStream_t s = nullptr;
  void begin(int) {
    cudaEvent_t e;
    cudaEventCreate(&e);
    cudaEventRecord(e, s);
    ev.push_back(e);
  }
  void end(int id) {
    cudaEvent_t e;
    cudaEventCreate(&e);
    cudaEventRecord(e, s);
    ev.push_back(e);
    ids.push_back(id);
  }
  ~KTimer() {
    for (auto e : ev) cudaEventDestroy(e);
  }
};
#define TB(id) \
  if (tm) tm->begin(id)
#define TE(id) \
  if (tm) tm->end(id)

// The kernels of one trend evaluation.  The pipelined tiles keep a tile's geometry over
// a group of layers, which one or two layers do not pay back; measured, us a step
// (pipelined tiles / tiles of one layer / L1 kernels):
//   FP64, 1 layer:  J6 102 / 70 / 84,   J7 164 / 124 / 152,  J8 476 / 391 / 662,  J9 1528 / 1249
//   FP64, 2 layers: J6 113 / 107 / 92,  J7 231 / 222 / 308,  J8 664 / 670 / 1217, J9 2411 / 2241
//   FP64, 3 layers: J6 125 / 126 / 145, J7 288 / 337 / 477,  J8 880 / 984 / 1777, J9 3171 / 3371
//   FP32, 1 layer:  J6 105 / - / 83,    J7 166 / - / 150,    J8 491 / - / 587,    J9 1570 / - / 2063
//   FP32, 2 layers: J6 113 / - / 92,    J7 220 / - / 263,    J8 650 / - / 1061,   J9 2262 / - / 3813
//   FP32, 3 layers: J6 125 / - / 131,   J7 276 / - / 404,    J8 838 / - / 1573,   J9 2972 / - / 5649
// FP64 takes the pipelined tiles from three layers up; FP32 fluxes, whose L1 kernels are
// further off, also below that where the blocks have eight rounds of tiles or more
// (J7: 5.5 rounds with one layer, 10.9 with two).
enum FluxKernels { FLUX_L1, FLUX_TILES, FLUX_PIPE };
static FluxKernels flux_kernels(wt_handle* h) {
  const int P = h->top().P;
  const int64_t tiles = (int64_t)10 * ((P + PX - 1) / PX) * ((P + PY - 1) / PY);
  if (h->trend_variant != 0) return FLUX_L1;
  if (h->flux_bits == 32)
    return f32_staged(h) && (h->nz >= 3 || tiles * h->nz >= 8 * (int64_t)h->pipe_slots) ? FLUX_PIPE : FLUX_L1;
  return h->nz >= 3 ? FLUX_PIPE : FLUX_TILES;
}

// Launch sequence of one trend evaluation of state (m, t, v); MODE_RK writes
// dst = base + hstep * trend, base the resident state, MODE_TREND writes the trends into
// h->dm/dt/dv.
static int launch_trend(wt_handle* h, double* m, double* t, double* v, int mode, double* om, double* ot, double* ov,
                        double hstep, KTimer* tm = nullptr) {
  DevLevel& D = h->top();
  LevelDev L = D.view();
  const int nz = h->nz;
  cudaStream_t s = h->stream;
  // block b: layer b % nz of node chunk b / nz (layer_node in trisk_kernels.cuh)
  const unsigned chunks = blocks_for(D.NN, NODE_TILE);
  const bool f32 = h->flux_bits == 32;
  const FluxKernels kernels = flux_kernels(h);
  const bool pipe = kernels == FLUX_PIPE;
  const unsigned cb = blocks_for(D.NN, COL_TILE);
  const unsigned gb = pipe ? ghost_blocks(h->ghosts.n_nodes + h->ghosts.n_edges, nz, COL_TILE) : 0;
  TB(1);
  column_batch(nz, [&](auto B) {
    if (pipe)
      k_column_halo<B.value><<<cb + gb, COL_TILE, 0, s>>>(L, h->ph, nz, gb, h->ghosts, m, t, v, h->mean_m, h->mean_t,
                                                          h->phik, h->pterm);
    else
      k_column<B.value><<<cb, COL_TILE, 0, s>>>(L, h->ph, nz, m, t, h->mean_m, h->mean_t, h->phik, h->pterm, nullptr);
  });
  TE(1);
  double* dm = mode == MODE_RK ? om : h->dm;
  double* dt = mode == MODE_RK ? ot : h->dt;
  double* dv = mode == MODE_RK ? ov : h->dv;
  const int sb = (m == h->m1) ? 1 : (m == h->m2) ? 2 : 0;  // which state buffer the stage reads
  if (pipe) {
    auto grid = [&](int nodes) {
      PipeGrid G{(nodes + PX - 1) / PX, (nodes + PY - 1) / PY, 0, 0, 0};
      const int tiles = G.nbx * G.nby * 10;
      G.group = pipe_group(tiles, nz, h->pipe_slots);
      G.ngroups = (nz + G.group - 1) / G.group;
      G.items = tiles * G.ngroups;
      return G;
    };
    const PipeGrid g1 = grid(D.n + 1), g2 = grid(D.P);
    const unsigned b1 = std::min(g1.items, h->pipe_slots), b2 = std::min(g2.items, h->pipe_slots);
    TB(2);
    if (f32)
      k_step1_pipe<float><<<b1, Step1Pipe<float>::BLOCK, Step1Pipe<float>::SMEM, s>>>(
          L, nz, g1, Step1Res<float>{h->qe32, h->hfm32, h->hft32, h->ke32, h->theta32}, h->dflag, h->tma_inject, h->p1maps[sb]);
    else
      k_step1_pipe<double><<<b1, Step1Pipe<double>::BLOCK, Step1Pipe<double>::SMEM, s>>>(
          L, nz, g1, Step1Res<double>{h->qe, h->hfm, h->hft, h->bern, h->theta}, h->dflag, h->tma_inject, h->p1maps[sb]);
    const unsigned nc = corner_blocks(nz), nb = border_blocks(D.n, nz), ng = ghost_blocks(h->ghosts.n_f, nz, GHOST_TILE);
    if (f32)
      k_step1_border<float><<<nc + nb + ng, GHOST_TILE, 0, s>>>(L, nz, nc, nb, m, v, h->mean_m, h->qe32, h->ghosts,
                                                                h->hfm32, h->hft32);
    else
      k_step1_border<double><<<nc + nb + ng, GHOST_TILE, 0, s>>>(L, nz, nc, nb, m, v, h->mean_m, h->qe, h->ghosts,
                                                                 h->hfm, h->hft);
    TE(2);
    TB(5);
    if (f32) {
      const TrendPipeIO io{dm, dt, dv, hstep};
      const auto k = mode == MODE_RK ? k_trend_pipe<float, MODE_RK> : k_trend_pipe<float, MODE_TREND>;
      const int smem = mode == MODE_RK ? TrendPipe<float, MODE_RK>::SMEM : TrendPipe<float, MODE_TREND>::SMEM;
      k<<<b2, TrendPipe<float, MODE_RK>::BLOCK, smem, s>>>(L, nz, g2, io, h->dflag, h->tma_inject, h->fmaps, h->p1maps[0]);
    } else {
      const TrendPipeIO io{dm, dt, dv, hstep};
      const auto k = mode == MODE_RK ? k_trend_pipe<double, MODE_RK> : k_trend_pipe<double, MODE_TREND>;
      const int smem = mode == MODE_RK ? TrendPipe<double, MODE_RK>::SMEM : TrendPipe<double, MODE_TREND>::SMEM;
      k<<<b2, TrendPipe<double, MODE_RK>::BLOCK, smem, s>>>(L, nz, g2, io, h->dflag, h->tma_inject, h->pmaps, h->p1maps[0]);
    }
    TE(5);
    CK(cudaGetLastError());
    return WT_OK;
  }
  if (f32) {  // FP32 flux stencils, FP64 trends and sub-step (trisk_mixed.cuh)
    TB(2);
    k_step1_f32<<<chunks * nz, NODE_TILE, 0, s>>>(L, nz, m, t, v, h->mean_m, h->mean_t,
                                                   Step1OutF{h->qe32, h->hfm32, h->hft32, h->ke32, h->theta32});
    TE(2);
    TrendIOF io{};
    io.theta = h->theta32; io.qe = h->qe32; io.hfm = h->hfm32; io.hft = h->hft32; io.ke = h->ke32;
    io.phik = h->phik; io.pterm = h->pterm;
    io.base_m = h->mass; io.base_t = h->temp; io.base_v = h->velo;
    io.dst_m = om; io.dst_t = ot; io.dst_v = ov; io.h = hstep;
    io.dm = h->dm; io.dtt = h->dt; io.dv = h->dv;
    TB(5);
    if (mode == MODE_RK)
      k_trend_mixed<MODE_RK><<<chunks * nz, NODE_TILE, 0, s>>>(L, nz, io);
    else
      k_trend_mixed<MODE_TREND><<<chunks * nz, NODE_TILE, 0, s>>>(L, nz, io);
    TE(5);
    CK(cudaGetLastError());
    return WT_OK;
  }
  Step1Out so{h->qe, h->hfm, h->hft, h->bern, h->theta};
  TB(2);
  if (kernels == FLUX_TILES) {
    const int nbx = (D.n + 1 + TT_X - 1) / TT_X, nby = (D.n + 1 + TT_Y - 1) / TT_Y;
    k_step1_tma<<<(unsigned)(nz * nbx * nby * 10), TT_X * TT_Y, STEP1_TMA_SMEM, s>>>(
        L, nz, nbx, nby, m, t, v, h->mean_m, h->phik, h->pterm, so, h->dflag, h->tma_inject, h->s1maps[sb], nullptr);
  } else {
    k_step1<<<chunks * nz, NODE_TILE, 0, s>>>(L, nz, m, t, v, h->mean_m, h->mean_t, h->phik, h->pterm, so, nullptr);
  }
  TE(2);
  TrendIO io{};
  io.theta = h->theta; io.qe = h->qe; io.hfm = h->hfm; io.hft = h->hft; io.bern = h->bern; io.phik = h->phik;
  io.base_m = h->mass; io.base_t = h->temp; io.base_v = h->velo;
  io.dst_m = om; io.dst_t = ot; io.dst_v = ov; io.h = hstep;
  io.dm = h->dm; io.dtt = h->dt; io.dv = h->dv;
  TB(5);
  if (kernels == FLUX_TILES) {
    const int nbx = (D.P + TT_X - 1) / TT_X, nby = (D.P + TT_Y - 1) / TT_Y;
    const auto k = mode == MODE_RK ? k_trend_tma<MODE_RK> : k_trend_tma<MODE_TREND>;
    k<<<(unsigned)(nz * nbx * nby * 10), TT_X * TT_Y, TREND_TMA_SMEM, s>>>(L, nz, nbx, nby, io, h->dflag, h->tma_inject,
                                                                           h->maps);
  } else if (mode == MODE_RK)
    k_trend<MODE_RK><<<chunks * nz, NODE_TILE, 0, s>>>(L, nz, io);
  else
    k_trend<MODE_TREND><<<chunks * nz, NODE_TILE, 0, s>>>(L, nz, io);
  TE(5);
  CK(cudaGetLastError());
  return WT_OK;
}

// k_trend_tma<MODE_ML> on the top level: the multi-level trend of the finest
// level with the RK sub-step, its inputs read through the maps M.
int wt_level_trend_ml_tma(wt_handle* h, const wtk::TrendIO& io, const wtk::TrendMaps& M, cudaStream_t stream) {
  const DevLevel& D = h->top();
  const int nz = h->nz;
  const int nbx = (D.P + TT_X - 1) / TT_X, nby = (D.P + TT_Y - 1) / TT_Y;
  const unsigned nblk = (unsigned)(nz * nbx * nby * 10);
  k_trend_tma<MODE_ML><<<nblk, TT_X * TT_Y, TREND_TMA_SMEM, stream ? stream : h->stream>>>(D.view(), nz, nbx, nby, io,
                                                                                           h->dflag, h->tma_inject, M);
  CK(cudaGetLastError());
  return WT_OK;
}

int wt_level_step1(wt_handle* h, int level, const double* m, const double* t, const double* v, const double* mean_m,
                   const double* mean_t, double* phik, double* pterm, double* qe, double* hfm, double* hft,
                   double* bern, double* theta, const wtk::Step1Maps* maps, cudaStream_t stream,
                   const unsigned char* need, const wtk::NodeList* list) {
  const DevLevel& D = h->at(level);
  const LevelDev L = D.view();
  const int nz = h->nz;
  cudaStream_t s = stream ? stream : h->stream;
  Step1Out so{qe, hfm, hft, bern, theta};
  const unsigned chunks = blocks_for(D.NN, NODE_TILE);
  if (list && list->ids) {  // the needed slots only, persistent blocks over the level's work list
    column_batch(nz, [&](auto B) {
      k_column_list<B.value><<<persistent_grid(k_column_list<B.value>, blocks_for(D.NN, COL_TILE), COL_TILE), COL_TILE,
                               0, s>>>(L, h->ph, nz, m, t, mean_m, mean_t, phik, pterm, *list);
    });
    k_step1_list<<<persistent_grid(k_step1_list, chunks * nz), NODE_TILE, 0, s>>>(L, nz, m, t, v, mean_m, mean_t,
                                                                                  phik, pterm, so, *list);
    CK(cudaGetLastError());
    return WT_OK;
  }
  column_batch(nz, [&](auto B) {
    k_column<B.value><<<blocks_for(D.NN, COL_TILE), COL_TILE, 0, s>>>(L, h->ph, nz, m, t, mean_m, mean_t, phik, pterm,
                                                                      need);
  });
  if (maps && level == h->level_end && h->trend_variant == 0) {
    const int nbx = (D.n + 1 + TT_X - 1) / TT_X, nby = (D.n + 1 + TT_Y - 1) / TT_Y;
    const unsigned nblk = (unsigned)(nz * nbx * nby * 10);
    k_step1_tma<<<nblk, TT_X * TT_Y, STEP1_TMA_SMEM, s>>>(L, nz, nbx, nby, m, t, v, mean_m, phik, pterm, so,
                                                           h->dflag, h->tma_inject, *maps, need);
  } else {
    k_step1<<<chunks * nz, NODE_TILE, 0, s>>>(L, nz, m, t, v, mean_m, mean_t, phik, pterm, so, need);
  }
  CK(cudaGetLastError());
  return WT_OK;
}

extern "C" {

int wt_trend(wt_handle* h) {
  if (!h) return WT_ERR_ARG;
  int rc = launch_trend(h, h->mass, h->temp, h->velo, MODE_TREND, nullptr, nullptr, nullptr, 0.0);
  if (rc) return rc;
  CK(cudaStreamSynchronize(h->stream));
  return WT_OK;
}

int wt_download_trend(wt_handle* h, double* dmass, double* dtemp, double* dvelo) {
  if (!h || !dmass || !dtemp || !dvelo) return WT_ERR_ARG;
  const int64_t nn = (int64_t)h->nz * h->top().NN;
  CK(cudaMemcpyAsync(dmass, h->dm, nn * 8, cudaMemcpyDeviceToHost, h->stream));
  CK(cudaMemcpyAsync(dtemp, h->dt, nn * 8, cudaMemcpyDeviceToHost, h->stream));
  CK(cudaMemcpyAsync(dvelo, h->dv, 3 * nn * 8, cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return WT_OK;
}

// One RK4 step (src/time_integr.f90:78-103): four trend evaluations, each
// fused with its sub-step.  WT_after_step on a uniform level is the ghost copy,
// which the kernels replace by reading ghosts through the remap tables.
static int record_rk4(wt_handle* h, double dt, KTimer* tm = nullptr) {
  const double hs[4] = {dt / 4.0, dt / 3.0, dt / 2.0, dt};
  // Stage states ping-pong between two buffers: k_trend reads the stage state at
  // neighbouring nodes while it writes the next one, so they must differ (the
  // reference finishes the whole trend before RK_sub_step).  The last stage
  // writes the solution in place, which it reads only at each thread's own node.
  double* SM[3] = {h->mass, h->m1, h->m2};
  double* ST[3] = {h->temp, h->t1, h->t2};
  double* SV[3] = {h->velo, h->v1, h->v2};
  const int qi[4] = {0, 1, 2, 1}, oi[4] = {1, 2, 1, 0};
  for (int stage = 0; stage < 4; ++stage) {
    double* qm = SM[qi[stage]];
    double* qt = ST[qi[stage]];
    double* qv = SV[qi[stage]];
    double* om = SM[oi[stage]];
    double* ot = ST[oi[stage]];
    double* ov = SV[oi[stage]];
    int rc = launch_trend(h, qm, qt, qv, MODE_RK, om, ot, ov, hs[stage], tm);
    if (rc) return rc;
  }
  CK(cudaGetLastError());
  return WT_OK;
}

int wt_rk4_step(wt_handle* h, double dt, int nsteps) {
  if (!h || nsteps < 0) return WT_ERR_ARG;
  if (nsteps == 0) return WT_OK;
  if (!h->graph_exec || h->graph_dt != dt) {
    if (h->graph_exec) { cudaGraphExecDestroy(h->graph_exec); h->graph_exec = nullptr; }
    cudaGraph_t g;
    CK(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
    int rc = record_rk4(h, dt);
    cudaError_t e = cudaStreamEndCapture(h->stream, &g);
    if (rc) return rc;
    if (e != cudaSuccess) return wt_handle_fail("capture", e);
    CK(cudaGraphInstantiate(&h->graph_exec, g, 0));
    cudaGraphDestroy(g);
    h->graph_dt = dt;
  }
  for (int s = 0; s < nsteps; ++s) CK(cudaGraphLaunch(h->graph_exec, h->stream));
  CK(cudaGetLastError());
  return WT_OK;
}

// Same steps as wt_rk4_step, launched kernel by kernel (no graph) with CUDA
// events around every launch; ms_per_launch[k] receives the average duration
// of kernel k (0 halo_state, 1 column, 2 step1, 3 post_step1, 4 halo_flux,
// 5 trend_rk) and *nkernels the number of kernel kinds.
int wt_profile_rk4(wt_handle* h, double dt, int nsteps, double* ms_per_launch, int* nkernels) {
  if (!h || nsteps < 1 || !ms_per_launch || !nkernels) return WT_ERR_ARG;
  KTimer tm;
  tm.s = h->stream;
  for (int s = 0; s < nsteps; ++s) {
    int rc = record_rk4(h, dt, &tm);
    if (rc) return rc;
  }
  CK(cudaStreamSynchronize(h->stream));
  double tot[8] = {0};
  int cnt[8] = {0};
  for (size_t q = 0; q < tm.ids.size(); ++q) {
    float ms = 0.f;
    CK(cudaEventElapsedTime(&ms, tm.ev[2 * q], tm.ev[2 * q + 1]));
    tot[tm.ids[q]] += ms;
    cnt[tm.ids[q]] += 1;
  }
  for (int k = 0; k < 6; ++k) ms_per_launch[k] = cnt[k] ? tot[k] / cnt[k] : 0.0;
  *nkernels = 6;   // kinds 0 (ghost copy), 3, 4 are no longer launched by the stepper
  return WT_OK;
}

int wt_rk4_step_host(wt_handle* h, double dt, int nsteps, double* mass, double* temp, double* velo) {
  if (!h || !mass || !temp || !velo) return WT_ERR_ARG;
  const int64_t nn = (int64_t)h->nz * h->top().NN;
  CK(cudaMemcpyAsync(h->mass, mass, nn * 8, cudaMemcpyHostToDevice, h->stream));
  CK(cudaMemcpyAsync(h->temp, temp, nn * 8, cudaMemcpyHostToDevice, h->stream));
  CK(cudaMemcpyAsync(h->velo, velo, 3 * nn * 8, cudaMemcpyHostToDevice, h->stream));
  h->state_halo_done = false;
  int rc = wt_rk4_step(h, dt, nsteps);
  if (rc) return rc;
  {
    DevLevel& D = h->top();
    int64_t nt = (int64_t)(2 * D.n_hn + D.n_he) * h->nz;
    k_halo_state<<<blocks_for(nt), TPB, 0, h->stream>>>(h->nz, D.NN, D.hn, D.n_hn, D.he, D.n_he, h->mass, h->temp, h->velo);
  }
  CK(cudaMemcpyAsync(mass, h->mass, nn * 8, cudaMemcpyDeviceToHost, h->stream));
  CK(cudaMemcpyAsync(temp, h->temp, nn * 8, cudaMemcpyDeviceToHost, h->stream));
  CK(cudaMemcpyAsync(velo, h->velo, 3 * nn * 8, cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return WT_OK;
}

}  // extern "C"
