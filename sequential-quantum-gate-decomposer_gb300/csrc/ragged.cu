// Ragged batches: one launch evaluates instances that each have their own circuit (and so
// their own qubit count, gate list and parameter count) and their own target.  A
// persistent grid (CTAs resident on every SM) pulls (instance, tile) work items from a
// queue ordered by decreasing work, so large instances start first and small ones fill
// the tail.  Tile bodies are the ones of the fixed-shape launches (tilekern.cuh).
#include <cuda_runtime.h>

#include <algorithm>
#include <numeric>
#include <string>
#include <vector>

#include "../../include/sqg.h"
#include "gates.cuh"
#include "handle.h"
#include "rotgrad.cuh"
#include "tile.cuh"
#include "tilekern.cuh"

using namespace sqg;

namespace {

constexpr int kRaggedThreads = 256;
constexpr int kRaggedStatic = 512;  // bound of the tile kernels' static shared memory

struct InstDesc {
  RotPlan plan;
  int P, n, N, cols, TC, tiles;
  // offsets of the instance in the packed arrays; gr_off counts overlaps
  long long theta_off, target_off, rec_off, ph_off, tr_off, gr_off;
};

}  // namespace

struct sqg_ragged_batch {
  int count = 0, with_grad = 0, device = 0, grid = 0, n_items = 0;
  size_t smem = 0;
  InstDesc* d_desc = nullptr;
  int2* d_items = nullptr;     // (instance, tile), decreasing work
  int2* d_cta_map = nullptr;   // (instance, CTA of runs) of the plan and gradient kernels
  int total_ctas = 0, max_overlaps = 0, sms = 1;
  long long total_rec = 0, total_ph = 0, total_tr = 0, total_gr = 0;
  std::vector<long long> theta_off, target_off;
  size_t off_rec = 0, off_ph = 0, off_tr = 0, off_gr = 0, ws_bytes = 0;
};

namespace {

inline size_t a256(size_t v) { return (v + 255) / 256 * 256; }

__global__ void __launch_bounds__(kRotThreads) k_ragged_plan(const InstDesc* __restrict__ desc,
                                                             const int2* __restrict__ cta_map,
                                                             const double* __restrict__ theta,
                                                             RotRec* __restrict__ recs, double2* __restrict__ phases,
                                                             int deal) {
  const int2 m = cta_map[blockIdx.x];
  const InstDesc d = desc[m.x];
  rot_plan_body(d.plan, m.y, theta + d.theta_off, recs + d.rec_off, phases + d.ph_off + m.y, deal);
}

// MODE 0: cost only; 1: gradient with real overlaps (FROBENIUS_NORM); 2: with complex ones.
template <int MODE>
__global__ void __launch_bounds__(kRaggedThreads, 3) k_ragged_tiles(const InstDesc* __restrict__ desc,
                                                                 const int2* __restrict__ items, int n_items,
                                                                 int* __restrict__ counter, const double2* targets,
                                                                 const RotRec* recs, const double2* phases,
                                                                 double2* ws_tr, double* ws_gr) {
  extern __shared__ double2 smem[];
  __shared__ int item_s;
  for (;;) {
    if (threadIdx.x == 0) item_s = atomicAdd(counter, 1);
    __syncthreads();
    const int item = item_s;
    __syncthreads();
    if (item >= n_items) break;
    const int2 it = items[item];
    const InstDesc d = desc[it.x];
    TileArgs a;
    a.ops = d.plan.ops;
    a.ends = d.plan.ends;
    a.nops = d.plan.nops;
    a.nrecs = d.plan.nrecs;
    a.noverlaps = d.plan.noverlaps;
    a.n = d.n; a.N = d.N;
    a.recs = recs + d.rec_off;
    a.phases = phases + d.ph_off;
    a.nphase = d.plan.ncta;
    a.mtx = const_cast<double2*>(targets) + d.target_off;
    a.bstride = 0;
    a.rstride = d.cols;
    a.cstride = 1;
    a.cols = d.cols;
    a.TC = d.TC;
    a.tiles = d.tiles;
    a.trace_offset = 0;
    a.ws_tr = ws_tr + d.tr_off;
    a.ws_gr = MODE ? ws_gr + d.gr_off * MODE : nullptr;
    a.ckpt = nullptr;
    a.ckpt_interval = 0;
    a.nck = 0;
    a.fixed = 1;
    if constexpr (MODE == 0)
      tile_forward_body<false, true, kRotFwd>(a, 0, it.y, smem);
    else
      tile_adjoint_body<MODE == 2>(a, 0, it.y, smem);
    __syncthreads();
  }
}

// blockIdx.x: instance, blockIdx.y and so on: 32 of its overlaps, W doubles each.
template <int W>
__global__ void __launch_bounds__(32 * kSumGroups) k_ragged_sum(const InstDesc* __restrict__ desc, double2* ws_tr,
                                                                double* ws_gr, int with_grad, int variant,
                                                                double* __restrict__ cost) {
  const InstDesc d = desc[blockIdx.x];
  const int nov = with_grad ? d.plan.noverlaps : 0;
  for (int part = blockIdx.y; part == 0 || part < (nov + 31) / 32; part += gridDim.y) {
    tile_sum_body<W>(part, ws_tr + d.tr_off, ws_gr + d.gr_off * W, d.tiles, nov, d.cols, variant, cost + blockIdx.x);
    __syncthreads();  // its sums are no longer read
  }
}

template <bool CPLX>
__global__ void __launch_bounds__(kRotThreads) k_ragged_grad(const InstDesc* __restrict__ desc,
                                                             const int2* __restrict__ cta_map,
                                                             const double* __restrict__ theta,
                                                             const RotRec* __restrict__ recs,
                                                             const double2* __restrict__ ws_tr,
                                                             const double* __restrict__ ws_gr, int variant,
                                                             double* __restrict__ grad) {
  const int2 m = cta_map[blockIdx.x];
  const InstDesc d = desc[m.x];
  rot_grad_body<CPLX>(d.plan, m.y, theta + d.theta_off, recs + d.rec_off, ws_tr + d.tr_off,
                      ws_gr + d.gr_off * (CPLX ? 2 : 1), d.cols, variant, grad + d.theta_off);
}

int cerr(cudaError_t e, const char* where) {
  return e == cudaSuccess ? SQG_OK : set_error(SQG_ERR_CUDA, std::string(where) + ": " + cudaGetErrorString(e));
}

void free_batch(sqg_ragged_batch* r) {
  if (!r) return;
  cudaFree(r->d_desc);
  cudaFree(r->d_items);
  cudaFree(r->d_cta_map);
  delete r;
}

}  // namespace

// Work of an item: pairs of amplitudes times gates.
static double item_work(const sqg_circuit* c, int tile_cols) {
  return (double)std::max(c->L, 1) * c->N * tile_cols;
}

// Default tile width: as many columns as 100 KB take, then halved, down to a pair for every thread of
// four warps, while one item is more than 1.3 times a resident CTA's share of the batch: the launch
// would wait for a few items.  Measured on GB300, full width against narrowed: 20 instances of 3 to 8
// qubits 2.05 against 1.55 ms, 10 of 3 to 7 1.13 against 0.51 ms, 60 of 3 to 6 0.86 against 0.43 ms,
// 40 of 3 to 5 379 against 249 us.  Batches with enough items lose by it (60 instances of 3 to 8
// qubits 2.69 against 2.87 ms, 400 12.4 against 13.2 ms) and stay as they are.
static int default_tile_cols(const sqg_circuit* c, int cols, bool with_grad, double share) {
  const size_t per = (size_t)c->N * sizeof(double2) * (with_grad ? 2 : 1);
  const int most = (int)std::max<size_t>(1, (size_t)100 * 1024 / per);
  int tc = 1;
  while (tc * 2 <= most) tc *= 2;
  tc = std::min(tc, cols);
  while (tc > 1 && (tc / 2) * (c->N / 2) >= 128 && item_work(c, tc) > 1.3 * share) tc /= 2;
  return tc;
}

extern "C" {

int sqg_ragged_create(const sqg_circuit* const* circuits, const int* cols, int count, int with_grad,
                      const int* tile_cols, sqg_ragged_batch** out) {
  if (!out) return set_error(SQG_ERR_INVALID_ARGUMENT, "null output handle");
  *out = nullptr;
  if (!circuits || !cols || count <= 0 || count > 65535)
    return set_error(SQG_ERR_INVALID_ARGUMENT, "need 1..65535 circuits and target widths");
  auto* r = new sqg_ragged_batch();
  r->count = count;
  r->with_grad = with_grad ? 1 : 0;
  cudaGetDevice(&r->device);
  std::vector<InstDesc> desc(count);
  std::vector<int2> cta_map;
  std::vector<std::pair<double, int2>> work;
  long long th = 0, tg = 0;
  size_t smem = 0;
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, r->device);
  double share = 0.0;  // of a resident CTA (three per SM) of the batch's work
  for (int i = 0; i < count; i++)
    if (circuits[i] && cols[i] > 0) share += item_work(circuits[i], cols[i]) / (3.0 * std::max(sms, 1));
  for (int i = 0; i < count; i++) {
    const sqg_circuit* c = circuits[i];
    if (!c || c->device != r->device || cols[i] <= 0 || cols[i] > (c ? c->N : 0)) {
      free_batch(r);
      return set_error(SQG_ERR_INVALID_ARGUMENT, "instance " + std::to_string(i) + ": bad circuit or target width");
    }
    if (c->n > 13) {
      free_batch(r);
      return set_error(SQG_ERR_UNSUPPORTED, "ragged batches hold whole columns on chip: qbit_num <= 13");
    }
    if (with_grad && c->n > 12) {
      free_batch(r);
      return set_error(SQG_ERR_UNSUPPORTED, "gradient supports qbit_num <= 12");
    }
    InstDesc& d = desc[i];
    d.plan = c->plan;
    d.P = c->P; d.n = c->n; d.N = c->N; d.cols = cols[i];
    const int tc = tile_cols && tile_cols[i] > 0 ? std::min(tile_cols[i], cols[i])
                                                 : default_tile_cols(c, cols[i], with_grad, share);
    if (tile_smem_bytes(tc, c->N, with_grad) > 220 * 1024) {
      free_batch(r);
      return set_error(SQG_ERR_UNSUPPORTED, "instance " + std::to_string(i) + ": tile does not fit in shared memory");
    }
    d.TC = tc;
    d.tiles = (cols[i] + tc - 1) / tc;
    d.theta_off = th;
    d.target_off = tg;
    d.rec_off = r->total_rec;
    d.ph_off = r->total_ph;
    d.tr_off = r->total_tr;
    d.gr_off = r->total_gr;
    r->theta_off.push_back(th);
    r->target_off.push_back(tg);
    th += c->P;
    tg += (long long)c->N * cols[i];
    r->total_rec += c->plan.nrecs;
    r->total_ph += c->plan.ncta;
    r->total_tr += d.tiles;
    if (with_grad) r->total_gr += (long long)d.tiles * c->plan.noverlaps;
    r->max_overlaps = std::max(r->max_overlaps, c->plan.noverlaps);
    smem = std::max(smem, tile_smem_bytes(tc, c->N, with_grad));
    for (int k = 0; k < c->plan.ncta; k++) cta_map.push_back(make_int2(i, k));
    const double w = item_work(c, tc);
    for (int t = 0; t < d.tiles; t++) work.push_back({w, make_int2(i, t)});
  }
  r->theta_off.push_back(th);
  r->target_off.push_back(tg);
  std::stable_sort(work.begin(), work.end(), [](const auto& a, const auto& b) { return a.first > b.first; });
  std::vector<int2> items(work.size());
  for (size_t k = 0; k < work.size(); k++) items[k] = work[k].second;
  r->n_items = (int)items.size();
  r->total_ctas = (int)cta_map.size();
  r->smem = smem;
  r->off_rec = 256;
  r->off_ph = a256(r->off_rec + sizeof(RotRec) * r->total_rec);
  r->off_tr = a256(r->off_ph + sizeof(double2) * r->total_ph);
  r->off_gr = a256(r->off_tr + sizeof(double2) * r->total_tr);
  r->ws_bytes = a256(r->off_gr + sizeof(double2) * std::max<long long>(r->total_gr, 1));
  cudaError_t e = cudaMalloc(&r->d_desc, sizeof(InstDesc) * count);
  if (e == cudaSuccess) e = cudaMalloc(&r->d_items, sizeof(int2) * std::max<size_t>(items.size(), 1));
  if (e == cudaSuccess) e = cudaMalloc(&r->d_cta_map, sizeof(int2) * std::max<size_t>(cta_map.size(), 1));
  if (e == cudaSuccess) e = cudaMemcpy(r->d_desc, desc.data(), sizeof(InstDesc) * count, cudaMemcpyHostToDevice);
  if (e == cudaSuccess && !items.empty())
    e = cudaMemcpy(r->d_items, items.data(), sizeof(int2) * items.size(), cudaMemcpyHostToDevice);
  if (e == cudaSuccess && !cta_map.empty())
    e = cudaMemcpy(r->d_cta_map, cta_map.data(), sizeof(int2) * cta_map.size(), cudaMemcpyHostToDevice);
  // kernel attributes are set here, at planning time and to the device's opt-in maximum
  // (the attribute is per kernel, shared by every batch), so that launches can be captured
  // in CUDA graphs
  int optin = 0;
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, r->device);
  if (e == cudaSuccess && smem + kRaggedStatic > (size_t)optin) {
    free_batch(r);
    return set_error(SQG_ERR_UNSUPPORTED, "work item does not fit in shared memory");
  }
  for (auto k : {k_ragged_tiles<0>, k_ragged_tiles<1>, k_ragged_tiles<2>})
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - kRaggedStatic);
  int per_sm = 0;
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &per_sm, with_grad ? k_ragged_tiles<1> : k_ragged_tiles<0>, kRaggedThreads, smem);
  if (e != cudaSuccess) {
    int st = cerr(e, "sqg_ragged_create");
    free_batch(r);
    return st;
  }
  r->sms = sms;
  r->grid = std::max(1, std::min(r->n_items, std::max(per_sm, 1) * sms));
  *out = r;
  return SQG_OK;
}

int sqg_ragged_destroy(sqg_ragged_batch* r) {
  free_batch(r);
  return SQG_OK;
}

size_t sqg_ragged_workspace_bytes(const sqg_ragged_batch* r) { return r ? r->ws_bytes : 0; }

int sqg_ragged_layout(const sqg_ragged_batch* r, long long* theta_offsets, long long* target_offsets) {
  if (!r) return set_error(SQG_ERR_INVALID_ARGUMENT, "null batch");
  for (int i = 0; i <= r->count; i++) {
    if (theta_offsets) theta_offsets[i] = r->theta_off[i];
    if (target_offsets) target_offsets[i] = r->target_off[i];
  }
  return SQG_OK;
}

int sqg_ragged_cost_grad(const sqg_ragged_batch* r, const double* theta, const void* targets, int variant,
                         double* cost, double* grad, void* workspace, size_t ws_bytes, void* stream) {
  if (!r || !targets || !cost) return set_error(SQG_ERR_INVALID_ARGUMENT, "null batch, targets or cost");
  int dev = -1;
  cudaGetDevice(&dev);
  if (dev != r->device) return set_error(SQG_ERR_INVALID_ARGUMENT, "batch belongs to another device");
  if (variant != SQG_FROBENIUS_NORM && variant != SQG_HILBERT_SCHMIDT_TEST && variant != SQG_INFIDELITY)
    return set_error(SQG_ERR_UNSUPPORTED, "cost function variant not implemented by the engine");
  if (grad && !r->with_grad) return set_error(SQG_ERR_INVALID_ARGUMENT, "batch was planned without gradients");
  if (!workspace || ws_bytes < r->ws_bytes)
    return set_error(SQG_ERR_WORKSPACE, "workspace too small: need " + std::to_string(r->ws_bytes));
  if (r->theta_off.back() > 0 && !theta) return set_error(SQG_ERR_INVALID_ARGUMENT, "null parameter array");
  cudaStream_t s = (cudaStream_t)stream;
  char* ws = (char*)workspace;
  int* counter = (int*)ws;
  RotRec* recs = (RotRec*)(ws + r->off_rec);
  double2* ph = (double2*)(ws + r->off_ph);
  double2* tr = (double2*)(ws + r->off_tr);
  double* gr = (double*)(ws + r->off_gr);
  const double2* tg = (const double2*)targets;
  int st;
  if ((st = cerr(cudaMemsetAsync(counter, 0, sizeof(int), s), "cudaMemsetAsync"))) return st;
  if (r->total_ctas > 0) {
    k_ragged_plan<<<r->total_ctas, kRotThreads, 0, s>>>(r->d_desc, r->d_cta_map, theta, recs, ph,
                                                        r->total_ctas > 2 * r->sms ? 2 : 4);
    if ((st = cerr(cudaGetLastError(), "k_ragged_plan"))) return st;
  }
  const int mode = !grad ? 0 : variant == SQG_FROBENIUS_NORM ? 1 : 2;
  auto tiles = mode == 0 ? k_ragged_tiles<0> : mode == 1 ? k_ragged_tiles<1> : k_ragged_tiles<2>;
  tiles<<<r->grid, kRaggedThreads, r->smem, s>>>(r->d_desc, r->d_items, r->n_items, counter, tg, recs, ph, tr, gr);
  if ((st = cerr(cudaGetLastError(), "k_ragged_tiles"))) return st;
  const dim3 sgrid(r->count, grad ? std::min(std::max(1, (r->max_overlaps + 31) / 32), 65535) : 1);
  if (mode < 2)
    k_ragged_sum<1><<<sgrid, 32 * kSumGroups, 0, s>>>(r->d_desc, tr, gr, grad != nullptr, variant, cost);
  else
    k_ragged_sum<2><<<sgrid, 32 * kSumGroups, 0, s>>>(r->d_desc, tr, gr, 1, variant, cost);
  if (grad && r->total_ctas > 0) {
    if (mode == 1)
      k_ragged_grad<false><<<r->total_ctas, kRotThreads, 0, s>>>(r->d_desc, r->d_cta_map, theta, recs, tr, gr, variant, grad);
    else
      k_ragged_grad<true><<<r->total_ctas, kRotThreads, 0, s>>>(r->d_desc, r->d_cta_map, theta, recs, tr, gr, variant, grad);
  }
  return cerr(cudaGetLastError(), "ragged sums and gradients");
}

}  // extern "C"
