// GB300 engine for the SQUANDER decomposition hot path: cost and adjoint gradient of a
// parametric circuit applied to a 2^n x cols complex128 target, plus forward/right
// application and the combined-unitary parity API.  Entry points are declared in
// include/sqg.h.
//
// Design (GB300-first, one GPU):
//  * Column tiles.  Gates mix rows only, so every column of U^dagger is an independent
//    state vector.  A CTA loads a tile of TC columns into shared memory (column-major:
//    each column contiguous), applies the whole circuit there, and reads HBM once, whatever
//    qubits it touches (n <= 13 fits a column in 128 KB).
//  * The circuit is applied as its rotation plan (rot.cuh): runs of single-qubit gates as one
//    rotation, CNOTs as a change of places.
//  * Adjoint gradient per column: psi = C u_j is undone operation by operation while the
//    co-state lambda (starting at e_{j+offset}) is taken back with it; for each run two or three
//    Pauli overlaps are summed over the tile, from which rotgrad.cuh makes the derivatives of its
//    gates.  O(L) passes in shared memory replace the reference's (P+1) dense derivative matrices.
//  * FP64 is the scarcest resource on GB300.  Cost and gradient, which are sums, are swept in 64-bit
//    fixed point on the integer multiplier (fx.cuh); matrices and states that go back to the caller
//    stay in FP64.
//  * Deterministic reductions: per-tile partial traces go to the caller's workspace and
//    are summed in a fixed order by a second kernel.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/sqg.h"
#include "gates.cuh"
#include "gatetile.cuh"
#include "handle.h"
#include "rotgrad.cuh"
#include "rotplan.h"
#include "tile.cuh"
#include "tilekern.cuh"

using namespace sqg;

namespace {
thread_local std::string g_last_error;
}  // namespace

int sqg::set_error(int status, const std::string& msg) {
  g_last_error = msg;
  return status;
}

namespace {

int fail(int status, const std::string& msg) { return sqg::set_error(status, msg); }

int cuda_status(cudaError_t e, const char* where) {
  if (e == cudaSuccess) return SQG_OK;
  g_last_error = std::string(where) + ": " + cudaGetErrorString(e);
  return SQG_ERR_CUDA;
}

constexpr int kMaxThreads = 256;
constexpr size_t kSmemBudgetFwd = 100 * 1024;   // column tile budget, forward only (n = 12: one column, 3 CTAs/SM)
constexpr size_t kSmemBudgetGrad = 100 * 1024;  // psi + lambda tiles

inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// -------------------------------------------------------------------------------------
// Gate-matrix preparation: one thread per (instance, gate).  Each parameter belongs to
// exactly one gate, so sin/cos of each stored parameter is evaluated once
// (Gates_block.cpp:269-279 evaluates them the same way, per parameter).
// -------------------------------------------------------------------------------------
__global__ void k_prep(const Gate* __restrict__ gates, int L, int P, const double* __restrict__ theta,
                       long long theta_stride, int B, GateMat* __restrict__ gm, double2* __restrict__ sc) {
  int g = blockIdx.x * blockDim.x + threadIdx.x;
  int b = blockIdx.y;
  if (g >= L || b >= B) return;
  Gate gt = gates[g];
  const double* th = theta + (long long)b * theta_stride + gt.pstart;
  GateMat m;
  m.u[0] = m.u[1] = m.u[2] = m.u[3] = make_double2(0.0, 0.0);
  double2* scb = sc + (long long)b * P + gt.pstart;
  if (gt.type == G_U3) {
    double st, ct, sp, cp, sl, cl;
    sincos(th[0], &st, &ct);
    sincos(th[1], &sp, &cp);
    sincos(th[2], &sl, &cl);
    scb[0] = make_double2(st, ct);
    scb[1] = make_double2(sp, cp);
    scb[2] = make_double2(sl, cl);
    double spl = sp * cl + cp * sl, cpl = cp * cl - sp * sl;
    // gate_kernel_templates.h:509-521
    m.u[0] = make_double2(ct, 0.0);
    m.u[1] = make_double2(-st * cl, -st * sl);
    m.u[2] = make_double2(st * cp, st * sp);
    m.u[3] = make_double2(ct * cpl, ct * spl);
  } else if (gate_param_num(gt.type) == 1) {
    double s, c;
    sincos(th[0], &s, &c);
    scb[0] = make_double2(s, c);
    m.u[0] = make_double2(c, s);
  }
  gm[(long long)b * L + g] = m;
}

// Numbers of the plan's operations, one CTA per (CTA of runs, instance).
__global__ void __launch_bounds__(kRotThreads) k_rot_plan(RotPlan pl, const double* __restrict__ theta,
                                                          long long theta_stride, RotRec* __restrict__ recs,
                                                          double2* __restrict__ phases, int deal) {
  const long long b = blockIdx.y;
  rot_plan_body(pl, blockIdx.x, theta + b * theta_stride, recs + b * pl.nrecs, phases + b * pl.ncta + blockIdx.x, deal);
}

// The same for many vectors in three launches.
__global__ void __launch_bounds__(kRotThreads) k_rot_matrices(RotPlan pl, const double* __restrict__ theta,
                                                              long long theta_stride, RotRec* recs) {
  const long long b = blockIdx.y;
  batch_matrices_body(pl, blockIdx.x, theta + b * theta_stride, recs + b * pl.nrecs);
}
// A warp per (chain, 32 vectors), counted in one dimension: circuits have more chains than a grid is
// high.  The chains of two and more runs come first for all vectors.
__global__ void __launch_bounds__(32) k_rot_chains(RotPlan pl, int B, int groups, RotRec* recs) {
  const long long b = (blockIdx.x % groups) * 32LL + threadIdx.x;
  if (b < B) batch_chain_body(pl, blockIdx.x / groups, recs + b * pl.nrecs);
}
__global__ void __launch_bounds__(kRotThreads) k_rot_finish(RotPlan pl, RotRec* recs, double2* __restrict__ phases) {
  const long long b = blockIdx.y;
  batch_finish_body(pl, blockIdx.x, recs + b * pl.nrecs, phases + b * pl.ncta + blockIdx.x);
}

template <bool WRITE_BACK, bool TRACE, int DIR>
__global__ void __launch_bounds__(kMaxThreads, 3) k_tile_forward(TileArgs a) {
  extern __shared__ double2 smem[];
  tile_forward_body<WRITE_BACK, TRACE, DIR>(a, blockIdx.y, blockIdx.x, smem);
}

// MINB: CTAs per SM that the registers are cut to where the launch fills the device with tiles: the sweeps
// wait on the integer pipes' latencies.  Three for real overlaps (80 registers, 196 bytes of them stored and
// 240 loaded again), two for complex ones (three: 232 and 844 bytes).  One where it does not fill the device.
// GB300, three against two: real, 8 qubits, 360 blocks, 64 vectors 40.1, 41.5 ms; 10 qubits, 6 vectors 17.5, 18.2 ms;
// 4 qubits, 1024 vectors 725, 699 us; 6 qubits, 300 vectors 1.32, 1.30 ms; complex, 8 qubits 50.7, 50.1 ms; 9 qubits,
// 300 gates of all kinds, 8 vectors 5.08, 4.89 ms.
template <bool CPLX, int MINB>
__global__ void __launch_bounds__(kMaxThreads, MINB) k_tile_adjoint(TileArgs a) {
  extern __shared__ double2 smem[];
  tile_adjoint_body<CPLX>(a, blockIdx.y, blockIdx.x, smem);
}

// Sums the per-tile partials in a fixed order and writes the cost; W doubles per overlap.
template <int W>
__global__ void __launch_bounds__(32 * kSumGroups) k_tile_sum(double2* ws_tr, double* ws_gr, int tiles, int noverlaps,
                                                              int cols, int variant, double* __restrict__ cost) {
  const long long b = blockIdx.y;
  tile_sum_body<W>(blockIdx.x, ws_tr + b * tiles, ws_gr + b * tiles * noverlaps * W, tiles, noverlaps, cols, variant,
                   cost + b);
}

template <bool CPLX>
__global__ void __launch_bounds__(kRotThreads) k_rot_grad(RotPlan pl, const double* __restrict__ theta,
                                                          const RotRec* __restrict__ recs,
                                                          const double2* __restrict__ ws_tr,
                                                          const double* __restrict__ ws_gr, int tiles, int P, int cols,
                                                          int variant, double* __restrict__ grad) {
  const long long b = blockIdx.y;
  rot_grad_body<CPLX>(pl, blockIdx.x, theta + b * P, recs + b * pl.nrecs, ws_tr + b * tiles,
                      ws_gr + b * tiles * pl.noverlaps * (CPLX ? 2 : 1), cols, variant, grad + b * P);
}

// The optimizer loops' evaluation (gatetile.cuh) and the sum of its tiles in their order.
__global__ void __launch_bounds__(kMaxThreads) k_gate_adjoint(GateTileArgs a) {
  extern __shared__ double2 smem[];
  gate_adjoint_body(a, blockIdx.x, smem);
}
__global__ void k_gate_finish(const double2* __restrict__ ws_tr, const double2* __restrict__ ws_gr, int tiles, int P,
                              int cols, int variant, double* __restrict__ cost, double* __restrict__ grad) {
  double2 tr = make_double2(0.0, 0.0);
  for (int t = 0; t < tiles; t++) tr = cadd(tr, ws_tr[t]);
  if (blockIdx.x == 0 && threadIdx.x == 0) *cost = cost_from_trace(variant, tr, cols);
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P) return;
  double2 dt = make_double2(0.0, 0.0);
  for (int t = 0; t < tiles; t++) dt = cadd(dt, ws_gr[(long long)t * P + p]);
  grad[p] = grad_from_trace(variant, tr, dt, cols);
}

// -------------------------------------------------------------------------------------
// One pass over an HBM-resident matrix per gate (unfused application and the
// combined-unitary parity API).  Thread = one amplitude pair x one column; consecutive
// threads take consecutive columns, so every access is a coalesced 16-byte load.
// deriv_k < 0: forward gate from gm; deriv_k >= 0: derivative kernel of parameter
// deriv_k built from the stored sin/cos, with the pairs whose control bit is clear
// zeroed (apply_kernel_to_input.cpp:93-97).
// -------------------------------------------------------------------------------------
__global__ void k_gate_hbm(double2* __restrict__ mtx, long long bstride, long long rstride, int cols, int logN,
                           Gate gt, const GateMat* __restrict__ gmp, const double2* __restrict__ scp, int deriv_k,
                           int nmat) {
  const bool ctrl = gate_controlled(gt.type);
  const bool deriv = deriv_k >= 0;
  const int lognp = (!deriv && ctrl) ? logN - 2 : logN - 1;
  const long long items = (long long)cols << lognp;
  const int step = 1 << gt.target;
  PairOp op;
  double2 D[4];
  if (deriv) {
    deriv_kernel(gt.type, scp + gt.pstart, deriv_k, D);
  } else {
    op = make_op(gt.type, *gmp, ORIENT_FWD);
  }
  // items < 2^31 (at most 2^29 pairs of a 30-qubit state, 2^12 x 2^13 pairs of a matrix);
  // a power-of-two column count splits an item with a shift instead of a division
  const int logc = (__popc(cols) == 1) ? __ffs(cols) - 1 : -1;
  for (int b = blockIdx.y; b < nmat; b += gridDim.y) {
    double2* base = mtx + (long long)b * bstride;
    for (unsigned it = blockIdx.x * blockDim.x + threadIdx.x; it < (unsigned)items; it += gridDim.x * blockDim.x) {
      int p, c;
      if (logc >= 0) {
        p = (int)(it >> logc);
        c = (int)(it & (unsigned)(cols - 1));
      } else {
        p = (int)(it / (unsigned)cols);
        c = (int)(it - (unsigned)p * (unsigned)cols);
      }
      int i;
      bool active = true;
      if (!deriv) {
        i = ctrl ? pair_index2(p, gt.target, gt.control) : pair_index1(p, gt.target);
      } else {
        i = pair_index1(p, gt.target);
        active = !ctrl || ((i >> gt.control) & 1);
      }
      double2* px = base + (long long)i * rstride + c;
      double2* py = base + (long long)(i + step) * rstride + c;
      if (!active) {
        *px = make_double2(0.0, 0.0);
        *py = make_double2(0.0, 0.0);
        continue;
      }
      double2 x = *px, y = *py;
      if (!deriv) {
        apply_op(op, x, y);
      } else {
        double2 nx, ny;
        nx.x = D[0].x * x.x - D[0].y * x.y + D[1].x * y.x - D[1].y * y.y;
        nx.y = D[0].x * x.y + D[0].y * x.x + D[1].x * y.y + D[1].y * y.x;
        ny.x = D[2].x * x.x - D[2].y * x.y + D[3].x * y.x - D[3].y * y.y;
        ny.y = D[2].x * x.y + D[2].y * x.x + D[3].x * y.y + D[3].y * y.x;
        x = nx;
        y = ny;
      }
      *px = x;
      *py = y;
    }
  }
}

// CNOT and CZ on an HBM-resident matrix or state (one pass per gate, no FP64 instruction, so
// the pass is bound by HBM alone).  An item is one element of a touched row; consecutive
// threads take consecutive elements, so every load and store instruction of a warp covers
// 512 contiguous bytes.  A thread handles 4 items a grid-stride apart and issues all their loads
// before its stores (8 loads in flight for CNOT).  CNOT exchanges the two rows of every pair
// whose control bit is set (half of the rows); CZ negates, by flipping sign bits, only the
// target = 1 row of those pairs (a quarter of the rows) and reads nothing else.
// `col_shift` = log2(cols) when cols is a power of two, else -1.
template <int KIND>  // 0: CNOT, 1: CZ
__global__ void __launch_bounds__(256) k_perm_hbm(double2* __restrict__ mtx, long long rstride, int cols,
                                                  int col_shift, long long items, int target, int control) {
  constexpr int U = 4;
  const int step = 1 << target;
  const unsigned long long sign = 0x8000000000000000ULL;
  const long long T = (long long)gridDim.x * blockDim.x;
  for (long long it0 = blockIdx.x * (long long)blockDim.x + threadIdx.x; it0 < items; it0 += U * T) {
    double2* px[U];
    double2* py[U];
    double2 a[U], b[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const long long it = it0 + k * T;
      px[k] = py[k] = nullptr;
      if (it < items) {
        const int pr = col_shift >= 0 ? (int)(it >> col_shift) : (int)(it / cols);
        const int c = (int)(it - (long long)pr * cols);
        const int i = pair_index2(pr, target, control);
        px[k] = mtx + (long long)i * rstride + c;
        py[k] = mtx + (long long)(i + step) * rstride + c;
      }
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      if (py[k]) {
        b[k] = *py[k];
        if (KIND == 0) a[k] = *px[k];
      }
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      if (!py[k]) continue;
      if (KIND == 0) {
        *px[k] = b[k];
        *py[k] = a[k];
      } else {
        *py[k] = make_double2(__longlong_as_double(__double_as_longlong(b[k].x) ^ (long long)sign),
                              __longlong_as_double(__double_as_longlong(b[k].y) ^ (long long)sign));
      }
    }
  }
}

int hbm_blocks(long long items) { return (int)std::min<long long>((items + 255) / 256, 152LL * 16); }

// ---- launch helpers ------------------------------------------------------------------
struct TilePlan {
  int TC, tiles, threads;
  size_t smem;
};

int choose_threads(int tc, int N, bool grad) {
  int items = tc * (N / 2);
  int t = std::min(kMaxThreads, std::max(32, (items + 31) / 32 * 32));
  (void)grad;
  return t;
}

int device_sms() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 1;
  return std::max(sms, 1);
}

// Column tiles of a launch over B instances of `cols` columns.  A tile holds as many columns
// as the shared-memory budget takes (a power of two); when the whole launch would then not
// give every SM two CTAs (small batches: a single decomposition's evaluation), tiles are
// narrowed down to one column each, so the work of one instance spreads over the GPU.  even: one
// step more for a launch of two to three CTAs per SM, which are two on some SMs and three on others,
// while that leaves 128 pairs per tile.  Measured on GB300, gradient, without and with: 5 qubits, 40
// blocks, 310 vectors 864, 741 us; 6 qubits, 160 vectors 1506, 1063 us; 7 qubits, 30 blocks, 40 vectors
// 1194, 832 us, 10 vectors 412, 384 us; 8 qubits, 10 vectors 1212, 841 us, 3 vectors 420, 410 us.  With 64
// pairs 7 qubits, 5 vectors 277, 294 us; 4 qubits, 400 vectors 366, 397 us.  The cost alone gains as
// often as it loses.
TilePlan plan_tiles(int N, int cols, bool grad, int B = 0, bool even = false) {
  const size_t per = (size_t)N * sizeof(double2) * (grad ? 2 : 1);
  size_t budget = grad ? kSmemBudgetGrad : kSmemBudgetFwd;
  int tc = (int)std::max<size_t>(1, budget / per);
  // prefer powers of two, never more than the vectors available
  int p2 = 1;
  while (p2 * 2 <= tc) p2 *= 2;
  tc = std::min(p2, cols);
  if (B > 0) {
    const long long sms = device_sms();
    auto ctas = [&] { return (long long)B * ((cols + tc - 1) / tc); };
    while (tc > 1 && ctas() < 2 * sms) tc >>= 1;
    if (even && ctas() < 3 * sms && (tc / 2) * (N / 2) >= 128) tc >>= 1;
  }
  TilePlan pl;
  pl.TC = tc;
  pl.tiles = (cols + tc - 1) / tc;
  pl.threads = choose_threads(tc, N, grad);
  pl.smem = tile_smem_bytes(tc, N, grad);
  return pl;
}

// Threads of a fixed-point evaluation: up to four pairs each, so that an operation's numbers are
// decoded for more than one, and more tiles are resident, while every SM keeps a warp per
// scheduler.  Measured on GB300 with one, two and four pairs per thread (40 blocks; gradient): four
// qubits, 1024 vectors 788, 669, 682 us, 200 vectors 269, 301, 301 us; five qubits, 200 vectors 690,
// 629, 522 us, 2500 vectors 3.69, 3.69, 3.45 ms; seven qubits, 30 blocks, 32 vectors 789, 789, 703 us,
// one vector 191, 236, 236 us.  One warp per tile was never better than two.
int eval_threads(const TilePlan& pl, int N, int B) {
  const int items = pl.TC * (N / 2);
  int t = pl.threads;
  for (int pairs = 2; pairs <= 4; pairs *= 2) {
    const int fewer = std::max(64, (items / pairs + 31) / 32 * 32);
    if (fewer >= t) continue;
    if ((long long)B * pl.tiles * (fewer / 32) < 4LL * device_sms()) break;
    t = fewer;
  }
  return t;
}

// Raises a kernel's dynamic shared memory limit to the device's opt-in maximum (never
// lowers it: the attribute is shared by every caller of the kernel).
template <typename K>
int set_smem(K kernel, size_t bytes) {
  if (bytes > 48 * 1024) {
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncAttributes fa;
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, kernel);
    const size_t dyn_max = e == cudaSuccess ? (size_t)optin - fa.sharedSizeBytes : 0;  // minus static shared memory
    if (e == cudaSuccess && bytes > dyn_max) return fail(SQG_ERR_UNSUPPORTED, "tile exceeds shared memory");
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn_max);
    if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute");
  }
  return SQG_OK;
}

// Workspace of the per-gate kernels: gate matrices and (sin, cos) of every parameter.
struct PrepLayout {
  size_t gm_off, sc_off, end;
};
PrepLayout prep_layout(const sqg_circuit* c, int B, size_t start) {
  PrepLayout l;
  l.gm_off = align_up(start, 256);
  l.sc_off = align_up(l.gm_off + (size_t)B * std::max(c->L, 1) * sizeof(GateMat), 256);
  l.end = align_up(l.sc_off + (size_t)B * std::max(c->P, 1) * sizeof(double2), 256);
  return l;
}

// Workspace of the plan's numbers (at most prep_layout's: no more operations than gates, no
// more CTAs than parameters).
struct RotLayout {
  size_t rec_off, ph_off, end;
};
RotLayout rot_layout(const RotPlan& p, int B, size_t start) {
  RotLayout l;
  l.rec_off = align_up(start, 256);
  l.ph_off = align_up(l.rec_off + (size_t)B * p.nrecs * sizeof(RotRec), 256);
  l.end = align_up(l.ph_off + (size_t)B * p.ncta * sizeof(double2), 256);
  return l;
}

// Vectors from which the plan's numbers are made in three launches.  Below, warps of k_rot_chains
// would idle.
constexpr int kRotBatch = 32;

// Makes the plan's numbers for B parameter vectors in the workspace and points `a` at them.
int launch_plan(const sqg_circuit* c, const RotPlan& p, const double* theta, long long theta_stride, int B, const RotLayout& l, char* ws,
                TileArgs& a, cudaStream_t st) {
  RotRec* recs = (RotRec*)(ws + l.rec_off);
  double2* ph = (double2*)(ws + l.ph_off);
  a.ops = p.ops;
  a.ends = p.ends;
  a.nops = p.nops;
  a.nrecs = p.nrecs;
  a.noverlaps = p.noverlaps;
  a.n = c->n;
  a.N = c->N;
  a.recs = recs;
  a.phases = ph;
  a.nphase = p.ncta;
  if (p.ncta == 0) return SQG_OK;
  if (B >= kRotBatch) {
    k_rot_matrices<<<dim3(p.ncta, B), kRotThreads, 0, st>>>(p, theta, theta_stride, recs);
    const int groups = (B + 31) / 32;
    k_rot_chains<<<(unsigned)groups * p.nheads, 32, 0, st>>>(p, B, groups, recs);
    k_rot_finish<<<dim3(p.ncta, B), kRotThreads, 0, st>>>(p, recs, ph);
  } else {
    k_rot_plan<<<dim3(p.ncta, B), kRotThreads, 0, st>>>(p, theta, theta_stride, recs, ph,
                                                         p.ncta * B > 2 * device_sms() ? 2 : 4);
  }
  return cuda_status(cudaGetLastError(), "k_rot_plan");
}

// The plan of a launch of so many tiles: with short chains where it waits for them.  Sweeps in fixed point do
// while they do not fill the device (three tiles per SM), those in FP64 while an SM has no more than one tile:
// GB300, chains of 16 against 4, 60 U3-CNOT blocks on 8 qubits, 75 tiles 751, 735 us; 38 gates on 9 qubits, 306
// tiles 281, 292 us.
const RotPlan& launch_plan_of(const sqg_circuit* c, long long tiles, int per_sm) {
  return tiles < (long long)per_sm * device_sms() ? c->short_plan : c->plan;
}
constexpr int kShortPlanFx = 3, kShortPlanFp64 = 1;

struct EvalLayout {
  const RotPlan* rp;
  RotLayout rot;
  size_t tr_off, gr_off, ck_off, end;
  TilePlan plan;
  int nck;
};
// The overlaps take two doubles each, whatever the cost variant: FROBENIUS_NORM, which needs
// only their imaginary parts, uses half of that.
EvalLayout eval_layout(const sqg_circuit* c, int B, int cols, bool grad, int ckpt_interval, bool even = true) {
  EvalLayout l;
  l.plan = plan_tiles(c->N, cols, grad, B, even && grad && ckpt_interval == 0);
  if (ckpt_interval == 0) l.plan.threads = eval_threads(l.plan, c->N, B);
  l.rp = &launch_plan_of(c, (long long)B * l.plan.tiles, kShortPlanFx);
  l.rot = rot_layout(*l.rp, B, 0);
  l.tr_off = l.rot.end;
  l.gr_off = align_up(l.tr_off + (size_t)B * l.plan.tiles * sizeof(double2), 256);
  size_t gr_bytes = grad ? (size_t)B * l.plan.tiles * std::max(l.rp->noverlaps, 1) * sizeof(double2) : 0;
  l.ck_off = align_up(l.gr_off + gr_bytes, 256);
  l.nck = 0;
  if (grad && ckpt_interval > 0) l.nck = l.rp->nops / ckpt_interval;
  size_t ck_bytes = (size_t)B * l.plan.tiles * l.nck * (size_t)l.plan.TC * c->N * sizeof(double2);
  l.end = align_up(l.ck_off + ck_bytes, 256);
  return l;
}

// The layout for a workspace of ws_bytes: without the last step of plan_tiles, which takes more
// bytes, where it does not fit.
EvalLayout eval_layout_within(const sqg_circuit* c, int B, int cols, bool grad, int ckpt_interval, size_t ws_bytes) {
  const EvalLayout l = eval_layout(c, B, cols, grad, ckpt_interval);
  return l.end <= ws_bytes ? l : eval_layout(c, B, cols, grad, ckpt_interval, false);
}

int launch_prep(const sqg_circuit* c, const double* theta, long long theta_stride, int B, GateMat* gm, double2* sc,
                cudaStream_t st) {
  if (c->L == 0) return SQG_OK;
  dim3 grid((c->L + 127) / 128, B);
  k_prep<<<grid, 128, 0, st>>>(c->d_gates, c->L, c->P, theta, theta_stride, B, gm, sc);
  return cuda_status(cudaGetLastError(), "k_prep");
}

// Matrix entry points hold whole columns in shared memory: qbit_num <= kMatrixQubits.
constexpr int kMatrixQubits = 13;

int check_circuit(const sqg_circuit* c, int max_n = kMatrixQubits) {
  if (!c) return fail(SQG_ERR_INVALID_ARGUMENT, "null circuit handle");
  int dev = -1;
  cudaGetDevice(&dev);
  if (dev != c->device) return fail(SQG_ERR_INVALID_ARGUMENT, "circuit handle belongs to another device");
  if (c->n > max_n)
    return fail(SQG_ERR_UNSUPPORTED, "this entry point supports qbit_num <= " + std::to_string(max_n) +
                                         " (state vectors up to 30 qubits: sqg_apply_state)");
  return SQG_OK;
}

// ---- state vectors ---------------------------------------------------------------------
constexpr int kStateQubits = 30;   // largest register of sqg_apply_state (2^30 amplitudes, 16 GiB)
constexpr int kStateK = 12;        // qubits per chunk: 4096 amplitudes, 64 KB of shared memory
constexpr int kStateLow = 5;       // the lowest qubits belong to every chunk (512-byte coalesced runs)
constexpr int kStateThreads = 256;

// Appends bytes to a blob on a 16-byte boundary; returns their offset.
size_t blob_put(std::vector<char>& blob, const void* src, size_t bytes) {
  const size_t at = blob.size();
  blob.resize((at + bytes + 15) / 16 * 16);
  if (bytes) memcpy(blob.data() + at, src, bytes);
  return at;
}

// Groups the gates into blocks: a block grows while the qubits it touches, together with the
// lowest kStateLow ones, number at most K; each block is one pass over the state.  With
// partition ends (`cuts`, the gate index after each partition) a block grows by whole
// partitions and breaks only between them, unless one partition alone exceeds the chunk (it
// is then split gate by gate).  Fills the chunk with further qubits (lowest first), maps every
// gate of the block to chunk-local qubit positions and tabulates the global offsets of the
// chunk's high local bits and the qubits that number the chunks.
struct StatePlanHost {
  std::vector<RotOp> lops;
  std::vector<int> lends, hitab, inact;
  std::vector<sqg_state_block> blocks;
  int split = 0;  // partitions larger than a chunk
};
StatePlanHost build_state_plan(const sqg_circuit* c, int K, const std::vector<int>& cuts) {
  const int n = c->n, low = std::min(K, kStateLow);
  StatePlanHost out;
  std::vector<RotOp>& lops = out.lops;
  std::vector<int>&lends = out.lends, &hitab = out.hitab, &inact = out.inact;
  size_t done = 0;  // steps placed in blocks (they follow the order of their anchor gates)
  std::vector<int> inA(n, 0), A, loc(n);
  std::vector<RotCz> scratch;
  lops.reserve(c->h_steps.size() + 16);
  const int hb = K - low;
  int used = 0;  // qubits of the block's gates above the lowest
  auto close_block = [&](int g1) {  // its gates end before g1
    int free = K - low - used;
    for (int q = low; q < n && free > 0; q++)
      if (!inA[q]) {
        inA[q] = 1;
        free--;
      }
    A.clear();
    for (int q = 0; q < n; q++) {
      loc[q] = q < low || inA[q] ? (int)A.size() : -1;
      if (loc[q] >= 0) A.push_back(q);
    }
    const int s0 = (int)done, k0 = (int)lops.size();
    while (done < c->h_steps.size() && c->h_steps[done].anchor < g1) done++;
    lower_rot_steps(c->h_steps, s0, (int)done, K, loc, lops, lends, scratch);
    lends.resize(16 * (out.blocks.size() + 1), 0);
    const size_t h0 = hitab.size();
    hitab.resize(h0 + (size_t(1) << hb), 0);
    for (int h = 1; h < (1 << hb); h++)
      hitab[h0 + h] = hitab[h0 + (h & (h - 1))] | 1 << A[low + __builtin_ctz(h)];
    int k = 0;
    for (int q = 0; q < n; q++)
      if (loc[q] < 0) {
        inact.push_back(q);
        k++;
      }
    for (; k < 32; k++) inact.push_back(0);
    out.blocks.push_back({k0, (int)lops.size()});
    std::fill(inA.begin(), inA.end(), 0);
    used = 0;
  };
  auto take_gate = [&](int g) {  // gate by gate: break wherever the chunk would overflow
    const Gate& gt = c->h_gates[g];
    int add = 0;
    int qs[2] = {gt.target, gate_controlled(gt.type) ? gt.control : -1};
    for (int q : qs)
      if (q >= low && !inA[q]) add++;
    if (low + used + add > K) {
      close_block(g);
    }
    for (int q : qs)
      if (q >= low && !inA[q]) {
        inA[q] = 1;
        used++;
      }
  };
  if (cuts.empty()) {
    for (int g = 0; g < c->L; g++) take_gate(g);
  } else {
    std::vector<int> mark(n, 0);
    int s0 = 0;
    for (int e : cuts) {  // partition [s0, e)
      std::vector<int> fresh;
      for (int g = s0; g < e; g++) {
        const Gate& gt = c->h_gates[g];
        int qs[2] = {gt.target, gate_controlled(gt.type) ? gt.control : -1};
        for (int q : qs)
          if (q >= low && !mark[q]) {
            mark[q] = 1;
            fresh.push_back(q);
          }
      }
      int add = 0, own = (int)fresh.size();
      for (int q : fresh) {
        if (!inA[q]) add++;
        mark[q] = 0;
      }
      if (low + own > K) {  // the partition alone exceeds the chunk
        out.split++;
        for (int g = s0; g < e; g++) take_gate(g);
      } else {
        if (low + used + add > K) {
          close_block(s0);
          add = own;
        }
        for (int q : fresh) inA[q] = 1;
        used += add;
      }
      s0 = e;
    }
  }
  if (c->L > 0) close_block(c->L);
  return out;
}

// Makes the state-vector plans of the circuit: chunks of 2^12 amplitudes, and, for registers whose
// chunks are too few for the device, smaller ones down to 2^9, where they split no partition that the
// largest hold.  They are appended to the blob, their device pointers counted from null until state_plans_at.
std::vector<sqg_state_plan> make_state_plans(const sqg_circuit* c, const std::vector<int>& cuts,
                                             std::vector<char>& blob) {
  std::vector<sqg_state_plan> plans;
  const int largest = std::min(c->n, kStateK);
  int split = 0;
  for (int K = largest; K >= (c->n <= 20 ? std::min(largest, 9) : largest); K--) {
    StatePlanHost h = build_state_plan(c, K, cuts);
    if (K == largest) split = h.split;
    if (h.split > split) break;  // so would those of still smaller chunks
    sqg_state_plan p;
    p.K = K;
    p.nops = (int)h.lops.size();
    p.blocks = std::move(h.blocks);
    p.lops = blob_put(blob, h.lops.data(), h.lops.size() * sizeof(RotOp));
    p.lends = blob_put(blob, h.lends.data(), h.lends.size() * sizeof(int));
    p.hitab = blob_put(blob, h.hitab.data(), h.hitab.size() * sizeof(int));
    p.inact = blob_put(blob, h.inact.data(), h.inact.size() * sizeof(int));
    plans.push_back(std::move(p));
  }
  return plans;
}
void state_plans_at(std::vector<sqg_state_plan>& plans, const void* base) {
  const char* d = (const char*)base;
  for (sqg_state_plan& p : plans) {
    p.d_lops = (const RotOp*)(d + p.lops);
    p.d_lends = (const int*)(d + p.lends);
    p.d_hitab = (const int*)(d + p.hitab);
    p.d_inact = (const int*)(d + p.inact);
  }
}

// The blob on the device; *out is set on success only.
int blob_to_device(const std::vector<char>& blob, void** out, const char* where) {
  void* d = nullptr;
  cudaError_t e = cudaMalloc(&d, std::max<size_t>(blob.size(), 1));
  if (e == cudaSuccess) e = cudaMemcpy(d, blob.data(), blob.size(), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    if (d) cudaFree(d);
    return cuda_status(e, where);
  }
  *out = d;
  return SQG_OK;
}

// The plan for `batch` states: the least of the modelled times.  An operation takes 1 ns per
// amplitude of an SM's chunks (the FP64 pipe), at least 0.7 us (its latency and the barrier), a block
// two operations' worth for loading and storing and 2.5 us for its launch.  Measured on GB300, 300 to
// 400 gates, chunks of 2^12 against the choice: 12 qubits 1146 -> 454 us, 15 qubits, 7 states 1247 ->
// 858 us, 17 qubits 1808 -> 760 us, 20 qubits 3162 -> 2111 us (the first and the last two before the
// rotation plan).
const sqg_state_plan& choose_state_plan(const sqg_circuit* c, int batch) {
  const int sms = device_sms();
  const sqg_state_plan* best = &c->splans[0];
  double best_t = 0.0;
  for (const sqg_state_plan& p : c->splans) {
    const double ctas = (double)batch * (double)(1LL << (c->n - p.K));
    const double per_sm = ctas <= 4.0 * sms ? (double)(((long long)ctas + sms - 1) / sms) : ctas / sms;
    const double op = std::max(0.7, per_sm * (1 << p.K) * 1e-3);
    const double t = p.nops * op + p.blocks.size() * (2.0 * op + 2.5);
    if (&p == best || t < best_t) {
      best = &p;
      best_t = t;
    }
  }
  return *best;
}

// One block of gates applied to every chunk of 2^K amplitudes of a state vector.  The
// chunk's low local bits are the state's lowest qubits (a warp loads 32 consecutive
// amplitudes), its high local bits are the block's other qubits (offsets from hitab), and the
// remaining qubits number the chunks (inact).  One read and one write of the state per block.
struct StateArgs {
  double2* states;
  long long stride;
  int n, K, low, k0, k1, nrecs;
  const RotOp* lops;
  const int* ends;        // this block's places behind its last operation
  const RotRec* recs;     // [B][nrecs]
  const double2* phases;  // [B][nphase], multiplied in by this pass; null: by another one
  int nphase;
  const int* hitab;
  const int* inact;
};

__global__ void __launch_bounds__(kStateThreads) k_state_block(StateArgs a) {
  extern __shared__ double2 sv[];
  __shared__ int hit[128];
  __shared__ int ends[16 * kEndGroups];
  __shared__ StagedOp st[kRotChunk];
  const int b = blockIdx.y;
  const int KK = 1 << a.K, hb = a.K - a.low, lowmask = (1 << a.low) - 1;
  for (int h = threadIdx.x; h < (1 << hb); h += blockDim.x) hit[h] = a.hitab[h];
  fill_end_table(ends, a.ends, a.K);
  long long cbase = 0;
  for (int j = 0; j < a.n - a.K; j++)
    if ((blockIdx.x >> j) & 1u) cbase |= 1LL << a.inact[j];
  double2* base = a.states + (long long)b * a.stride + cbase;
  __syncthreads();
  for (int l = threadIdx.x; l < KK; l += blockDim.x) sv[l] = base[(l & lowmask) + hit[l >> a.low]];
  __syncthreads();  // a block of CNOTs alone has no operation, only places to exchange
  const RotRec* recs = a.recs + (long long)b * a.nrecs;
  for (int k0 = a.k0; k0 < a.k1; k0 += kRotChunk) {
    const int kn = min(kRotChunk, a.k1 - k0);
    __syncthreads();
    stage_ops<true, false>(st, a.lops, recs, k0, kn);
    __syncthreads();
    for (int j = 0; j < kn; j++) {
      rot_tile<kRotFwd>(sv, KK, a.K, 1, st[j]);
      __syncthreads();
    }
  }
  if (a.phases) {
    double2 p = make_double2(1.0, 0.0);
    bool finite;  // no matter here
    for (int k = 0; k < a.nphase; k++) p = cmul(p, phase_factor(a.phases[(long long)b * a.nphase + k], finite));
    with_phase(p, [&](auto mul) {
      for (int l = threadIdx.x; l < KK; l += blockDim.x) base[(l & lowmask) + hit[l >> a.low]] = mul(sv[end_place(ends, l)]);
    });
  } else {
    for (int l = threadIdx.x; l < KK; l += blockDim.x) base[(l & lowmask) + hit[l >> a.low]] = sv[end_place(ends, l)];
  }
}

}  // namespace

// =====================================================================================
// C ABI
// =====================================================================================
// Makes the rotation and state-vector plans of the circuit and copies them to the device with its gates,
// in one allocation.  Host time is what a handle costs: GB300's host, 42 gates on three qubits 107 us (131 us
// with two allocations, lists of lists for the runs and 128 offsets for every block), 2000 gates on twelve
// 588 us (924 us).
static int make_plans(sqg_circuit* c) {
  std::vector<char> blob;
  const size_t o_gates = blob_put(blob, c->h_gates.data(), c->h_gates.size() * sizeof(Gate));
  RotPlan* plans[2] = {&c->plan, &c->short_plan};
  size_t off[2][8];
  const int nplans = c->n <= kMatrixQubits ? 2 : 1;  // state vectors use the first alone
  const RotRuns runs = find_rot_runs(c->n, c->h_gates);
  for (int k = 0; k < nplans; k++) {
    RotPlanHost h = build_rot_plan(runs, c->h_gates, k ? kRotShortChain : kRotChain);
    std::vector<RotOp> ops;
    std::vector<int> ends;
    if (c->n <= kMatrixQubits) {  // larger registers are applied in chunks only
      std::vector<int> loc(c->n);
      std::vector<RotCz> scratch;
      ops.reserve(h.steps.size() + 16);
      for (int q = 0; q < c->n; q++) loc[q] = q;
      lower_rot_steps(h.steps, 0, (int)h.steps.size(), c->n, loc, ops, ends, scratch);
    }
    RotPlan& p = *plans[k];
    p.nops = (int)ops.size();
    p.nrecs = (int)h.steps.size();
    p.ncta = (int)h.cta.size() - 1;
    p.noverlaps = h.noverlaps;
    off[k][0] = blob_put(blob, ops.data(), ops.size() * sizeof(RotOp));
    off[k][1] = blob_put(blob, h.runs.data(), h.runs.size() * sizeof(RotRun));
    off[k][2] = blob_put(blob, h.members.data(), h.members.size() * sizeof(int));
    off[k][3] = blob_put(blob, h.cta.data(), h.cta.size() * sizeof(int));
    off[k][4] = blob_put(blob, h.params.data(), h.params.size() * sizeof(int));
    off[k][5] = blob_put(blob, h.cta_params.data(), h.cta_params.size() * sizeof(int));
    off[k][6] = blob_put(blob, ends.data(), ends.size() * sizeof(int));
    off[k][7] = blob_put(blob, h.heads.data(), h.heads.size() * sizeof(int));
    p.nheads = (int)h.heads.size();
    if (k == 0) c->h_steps = std::move(h.steps);
  }
  c->splans = make_state_plans(c, {}, blob);
  const int st = blob_to_device(blob, &c->d_plan, "circuit handle");
  if (st) return st;
  const char* d = (const char*)c->d_plan;
  state_plans_at(c->splans, d);
  c->d_gates = (Gate*)(d + o_gates);
  for (int k = 0; k < nplans; k++) {
    RotPlan& p = *plans[k];
    p.gates = c->d_gates;
    p.ops = (const RotOp*)(d + off[k][0]);
    p.runs = (const RotRun*)(d + off[k][1]);
    p.members = (const int*)(d + off[k][2]);
    p.cta = (const int*)(d + off[k][3]);
    p.params = (const int*)(d + off[k][4]);
    p.cta_params = (const int*)(d + off[k][5]);
    p.ends = (const int*)(d + off[k][6]);
    p.heads = (const int*)(d + off[k][7]);
  }
  return SQG_OK;
}

extern "C" {

const char* sqg_status_string(int status) {
  switch (status) {
    case SQG_OK: return "ok";
    case SQG_ERR_INVALID_ARGUMENT: return "invalid argument";
    case SQG_ERR_UNSUPPORTED: return "unsupported configuration";
    case SQG_ERR_WORKSPACE: return "workspace too small";
    case SQG_ERR_CUDA: return "CUDA error";
    case SQG_ERR_PARAMETER_COUNT: return "wrong number of parameters";
    default: return "unknown status";
  }
}

const char* sqg_last_error(void) { return g_last_error.c_str(); }

int sqg_circuit_create(int qbit_num, const sqg_gate* gates, int gate_num, sqg_circuit** out) {
  if (!out) return fail(SQG_ERR_INVALID_ARGUMENT, "null output handle");
  *out = nullptr;
  if (qbit_num < 1 || qbit_num > kStateQubits) return fail(SQG_ERR_UNSUPPORTED, "qbit_num must be in 1..30");
  if (gate_num < 0 || (gate_num > 0 && !gates)) return fail(SQG_ERR_INVALID_ARGUMENT, "bad gate list");
  auto* c = new sqg_circuit();
  c->n = qbit_num;
  c->N = 1 << qbit_num;
  c->L = gate_num;
  int p = 0;
  for (int i = 0; i < gate_num; i++) {
    const sqg_gate& g = gates[i];
    int t = g.type;
    bool known = t == G_CZ || t == G_CNOT || t == G_U3 || t == G_RY || t == G_RX || t == G_RZ || t == G_CRY;
    if (!known) {
      delete c;
      return fail(SQG_ERR_UNSUPPORTED, "gate " + std::to_string(i) + ": unsupported gate type " + std::to_string(t));
    }
    if (g.target < 0 || g.target >= qbit_num) {
      delete c;
      return fail(SQG_ERR_INVALID_ARGUMENT, "gate " + std::to_string(i) + ": target qubit out of range");
    }
    if (gate_controlled(t) && (g.control < 0 || g.control >= qbit_num || g.control == g.target)) {
      delete c;
      return fail(SQG_ERR_INVALID_ARGUMENT, "gate " + std::to_string(i) + ": bad control qubit");
    }
    if (g.param_start != p) {
      delete c;
      return fail(SQG_ERR_INVALID_ARGUMENT, "gate " + std::to_string(i) + ": parameters must be contiguous in gate order");
    }
    if (gate_controlled(t) && qbit_num < 2) {
      delete c;
      return fail(SQG_ERR_INVALID_ARGUMENT, "controlled gate needs two qubits");
    }
    Gate d{t, g.target, gate_controlled(t) ? g.control : -1, g.param_start};
    c->h_gates.push_back(d);
    p += gate_param_num(t);
  }
  c->P = p;
  cudaGetDevice(&c->device);
  int st = make_plans(c);
  if (st) {
    sqg_circuit_destroy(c);
    return st;
  }
  *out = c;
  return SQG_OK;
}

int sqg_circuit_set_partitions(sqg_circuit* c, const int* part_ends, int nparts) {
  if (!c) return fail(SQG_ERR_INVALID_ARGUMENT, "null circuit handle");
  if (nparts < 0 || (nparts > 0 && !part_ends)) return fail(SQG_ERR_INVALID_ARGUMENT, "bad partition list");
  std::vector<int> cuts(part_ends, part_ends + nparts);
  for (int i = 0; i < nparts; i++)
    if (cuts[i] < (i ? cuts[i - 1] : 0) || cuts[i] > c->L)
      return fail(SQG_ERR_INVALID_ARGUMENT, "partition ends must be non-decreasing gate indices <= gate_num");
  if (nparts > 0 && cuts.back() != c->L) return fail(SQG_ERR_INVALID_ARGUMENT, "the last partition must end at gate_num");
  int dev = -1;
  cudaGetDevice(&dev);
  if (dev != c->device) return fail(SQG_ERR_INVALID_ARGUMENT, "circuit handle belongs to another device");
  std::vector<char> blob;
  std::vector<sqg_state_plan> plans = make_state_plans(c, cuts, blob);
  void* d = nullptr;
  const int st = blob_to_device(blob, &d, "state plan");
  if (st) return st;  // the plan that was there stays
  state_plans_at(plans, d);
  c->splans = std::move(plans);
  cudaFree(c->d_state);
  c->d_state = d;
  return SQG_OK;
}

int sqg_circuit_destroy(sqg_circuit* c) {
  if (!c) return SQG_OK;
  if (c->d_plan) cudaFree(c->d_plan);
  if (c->d_state) cudaFree(c->d_state);
  delete c;
  return SQG_OK;
}

int sqg_circuit_param_num(const sqg_circuit* c) { return c ? c->P : -1; }
int sqg_circuit_qbit_num(const sqg_circuit* c) { return c ? c->n : -1; }
int sqg_circuit_gate_num(const sqg_circuit* c) { return c ? c->L : -1; }

size_t sqg_cost_grad_workspace_bytes(const sqg_circuit* c, int batch, int cols, int with_grad) {
  if (!c || batch <= 0 || cols <= 0) return 0;
  return eval_layout(c, batch, cols, with_grad != 0, 0).end;
}

size_t sqg_cost_grad_checkpoint_workspace_bytes(const sqg_circuit* c, int batch, int cols, int checkpoint_interval) {
  if (!c || batch <= 0 || cols <= 0) return 0;
  return eval_layout(c, batch, cols, true, checkpoint_interval).end;
}

// Argument checks of sqg_cost_grad, shared with sqg_cost_grad_noalloc.
static int cost_grad_args(const sqg_circuit* c, const double* theta, int B, const void* target, int cols,
                          int trace_offset, int variant, const double* cost, const double* grad,
                          int checkpoint_interval) {
  int st = check_circuit(c);
  if (st) return st;
  if (B <= 0 || B > 65535 || !target || !cost || cols <= 0)
    return fail(SQG_ERR_INVALID_ARGUMENT, "bad batch (1..65535), target or output");
  if (c->P > 0 && !theta) return fail(SQG_ERR_INVALID_ARGUMENT, "null parameter array");
  if (cols > c->N) return fail(SQG_ERR_INVALID_ARGUMENT, "target has more columns than rows");
  if (variant != SQG_FROBENIUS_NORM && variant != SQG_HILBERT_SCHMIDT_TEST && variant != SQG_INFIDELITY)
    return fail(SQG_ERR_UNSUPPORTED, "cost function variant not implemented by the engine");
  const int off = variant == SQG_FROBENIUS_NORM ? trace_offset : 0;
  if (off < 0 || off + cols > c->N) return fail(SQG_ERR_INVALID_ARGUMENT, "trace offset out of range");
  const bool with_grad = grad != nullptr && c->P > 0;
  if (with_grad && c->n > 12) return fail(SQG_ERR_UNSUPPORTED, "gradient supports qbit_num <= 12");
  if (checkpoint_interval < 0) return fail(SQG_ERR_INVALID_ARGUMENT, "negative checkpoint interval");
  return SQG_OK;
}

// Whether the tile kernels are faster than the environment-matrix evaluation where both can run.
// The latter takes one CTA per vector and its time grows faster with the gates, by a wave where its CTAs,
// whose shared memory grows with them, no longer are all resident (two to three per SM); the tiles pay for the
// plan's numbers first, which cost more from kRotBatch vectors on.  Each line lies where the tiles are not
// slower on either side of it.  Measured on GB300 (152 SMs), gradient, us, environment matrix / tiles:
// three qubits, 45 gates 73 / 118 (one vector), 320 / 425 (3000); 111 gates 180 / 243 (450), 331 / 335 (600), 344 /
// 371 (700), 486 / 408 (920); 123 gates 197 / 256 (450), 359 / 346 (460), 364 / 351 (600), 535 / 428 (920); 138 gates
// 223 / 277 (450), 408 / 373 (460); 153 gates 433 / 302 (310); 183 gates 266 / 289 (one), 278 / 417 (300).
// Four qubits, 22 gates 90 / 94 (one), 90 / 94 (16); 25 gates 100 / 99 (one), 101 / 100 (16), 101 / 116 (32); 31 gates
// 123 / 106 (26); 40 gates 154 / 146 (32), 160 / 163 (250), 161 / 167 (300); 43 gates 172 / 172 (250), 172 / 159 (304);
// 28 gates 127 / 145 (340), 146 / 172 (500), 243 / 241 (1024); 34 gates 159 / 157 (340), 196 / 193 (500), 254 / 234
// (800).
// Five qubits, 8 gates 103 / 69 (one), 104 / 87 (76), 107 / 128 (300), 205 / 199 (700); 11 gates 139 / 114 (160), 139 /
// 142 (304), 168 / 162 (340), 267 / 222 (700).
static bool tiles_first(const sqg_circuit* c, int B) {
  const int sms = device_sms(), L = c->L;
  if (c->n >= 6) return true;
  if (c->n == 5) return L >= 11 || 2 * B <= sms;
  if (c->n == 4) return L >= (B < kRotBatch ? 24 : B <= 2 * sms ? 43 : 34);
  return c->n == 3 && ((L >= 112 && B > 5 * sms) || (L >= 120 && B > 3 * sms) || (L >= 144 && B > 2 * sms));
}

int sqg_cost_grad(const sqg_circuit* c, const double* theta, int B, const void* target, int cols,
                  long long target_batch_stride, int trace_offset, int variant, double* cost, double* grad,
                  int checkpoint_interval, void* workspace, size_t ws_bytes, void* stream) {
  int st = cost_grad_args(c, theta, B, target, cols, trace_offset, variant, cost, grad, checkpoint_interval);
  if (st) return st;
  const int off = variant == SQG_FROBENIUS_NORM ? trace_offset : 0;
  const bool with_grad = grad != nullptr && c->P > 0;
  if (with_grad && checkpoint_interval == 0) {
    // up to five qubits: one CTA per vector with the environment-matrix evaluation, which also
    // takes the calls without a workspace
    const bool tiles = tiles_first(c, B) && workspace && ws_bytes >= eval_layout(c, B, cols, true, 0, false).end;
    st = tiles ? SQG_ERR_UNSUPPORTED
               : sqg::env_cost_grad(c, theta, B, target, cols, target_batch_stride, off, variant, cost, grad, stream);
    if (st != SQG_ERR_UNSUPPORTED) return st;
    st = SQG_OK;
  }
  EvalLayout l = eval_layout_within(c, B, cols, with_grad, with_grad ? checkpoint_interval : 0, ws_bytes);
  if (!workspace || ws_bytes < l.end) return fail(SQG_ERR_WORKSPACE, "workspace too small: need " + std::to_string(l.end));
  cudaStream_t s = (cudaStream_t)stream;
  char* ws = (char*)workspace;
  double2* wtr = (double2*)(ws + l.tr_off);
  double* wgr = (double*)(ws + l.gr_off);
  TileArgs a;
  if ((st = launch_plan(c, *l.rp, theta, c->P, B, l.rot, ws, a, s))) return st;
  a.mtx = (double2*)target;
  a.bstride = target_batch_stride;
  a.rstride = cols;
  a.cstride = 1;
  a.cols = cols;
  a.TC = l.plan.TC;
  a.tiles = l.plan.tiles;
  a.trace_offset = off;
  a.ws_tr = wtr;
  a.ws_gr = wgr;
  a.ckpt = l.nck > 0 ? (double2*)(ws + l.ck_off) : nullptr;
  a.ckpt_interval = checkpoint_interval;
  a.nck = l.nck;
  a.fixed = 1;
  const dim3 grid(l.plan.tiles, B);
  if (!with_grad) {
    if ((st = set_smem(k_tile_forward<false, true, kRotFwd>, l.plan.smem))) return st;
    k_tile_forward<false, true, kRotFwd><<<grid, l.plan.threads, l.plan.smem, s>>>(a);
    if ((st = cuda_status(cudaGetLastError(), "tile kernel"))) return st;
    k_tile_sum<1><<<dim3(1, B), 32 * kSumGroups, 0, s>>>(wtr, nullptr, l.plan.tiles, 0, cols, variant, cost);
    return cuda_status(cudaGetLastError(), "k_tile_sum");
  }
  const int nov = l.rp->noverlaps;
  const dim3 sgrid((nov + 31) / 32, B), ggrid(l.rp->ncta, B);
  // the other variants multiply the derivative of the trace by the trace: complex overlaps
  const bool cplx = variant != SQG_FROBENIUS_NORM;
  const bool full = (long long)l.plan.tiles * B >= 3LL * device_sms();
  auto adjoint = cplx ? (full ? k_tile_adjoint<true, 2> : k_tile_adjoint<true, 1>)
                      : (full ? k_tile_adjoint<false, 3> : k_tile_adjoint<false, 1>);
  if ((st = set_smem(adjoint, l.plan.smem))) return st;
  adjoint<<<grid, l.plan.threads, l.plan.smem, s>>>(a);
  if (cplx) {
    k_tile_sum<2><<<sgrid, 32 * kSumGroups, 0, s>>>(wtr, wgr, l.plan.tiles, nov, cols, variant, cost);
    k_rot_grad<true><<<ggrid, kRotThreads, 0, s>>>(*l.rp, theta, a.recs, wtr, wgr, l.plan.tiles, c->P, cols, variant, grad);
  } else {
    k_tile_sum<1><<<sgrid, 32 * kSumGroups, 0, s>>>(wtr, wgr, l.plan.tiles, nov, cols, variant, cost);
    k_rot_grad<false><<<ggrid, kRotThreads, 0, s>>>(*l.rp, theta, a.recs, wtr, wgr, l.plan.tiles, c->P, cols, variant, grad);
  }
  return cuda_status(cudaGetLastError(), "cost and gradient kernels");
}

}  // extern "C"

// ---- the optimizer loops' evaluation ---------------------------------------------------
namespace {
struct LoopEvalLayout {
  TilePlan plan;
  PrepLayout prep;
  size_t tr_off, gr_off, end;
};
LoopEvalLayout loop_eval_layout(const sqg_circuit* c, int cols) {
  LoopEvalLayout l;
  l.plan = plan_tiles(c->N, cols, true, 1);
  l.plan.smem = gate_tile_smem_bytes(l.plan.TC, c->N);
  l.prep = prep_layout(c, 1, 0);
  l.tr_off = l.prep.end;
  l.gr_off = align_up(l.tr_off + (size_t)l.plan.tiles * sizeof(double2), 256);
  l.end = align_up(l.gr_off + (size_t)l.plan.tiles * std::max(c->P, 1) * sizeof(double2), 256);
  return l;
}
}  // namespace

size_t sqg::loop_cost_grad_bytes(const sqg_circuit* c, int cols) { return loop_eval_layout(c, cols).end; }

int sqg::loop_cost_grad(const sqg_circuit* c, const double* theta, const void* target, int cols, int off, int variant,
                        double* cost, double* grad, void* workspace, size_t ws_bytes, void* stream) {
  int st = sqg::env_cost_grad(c, theta, 1, target, cols, 0, off, variant, cost, grad, stream);
  if (st != SQG_ERR_UNSUPPORTED) return st;
  const LoopEvalLayout l = loop_eval_layout(c, cols);
  if (!workspace || ws_bytes < l.end) return fail(SQG_ERR_WORKSPACE, "workspace too small: need " + std::to_string(l.end));
  cudaStream_t s = (cudaStream_t)stream;
  char* ws = (char*)workspace;
  GateMat* gm = (GateMat*)(ws + l.prep.gm_off);
  double2* sc = (double2*)(ws + l.prep.sc_off);
  if ((st = launch_prep(c, theta, c->P, 1, gm, sc, s))) return st;
  GateTileArgs a;
  a.gates = c->d_gates;
  a.gm = gm;
  a.sc = sc;
  a.target = (const double2*)target;
  a.L = c->L; a.P = c->P; a.n = c->n; a.N = c->N; a.cols = cols;
  a.TC = l.plan.TC;
  a.tiles = l.plan.tiles;
  a.trace_offset = off;
  a.ws_tr = (double2*)(ws + l.tr_off);
  a.ws_gr = (double2*)(ws + l.gr_off);
  if ((st = set_smem(k_gate_adjoint, l.plan.smem))) return st;
  k_gate_adjoint<<<l.plan.tiles, l.plan.threads, l.plan.smem, s>>>(a);
  k_gate_finish<<<(c->P + 127) / 128, 128, 0, s>>>(a.ws_tr, a.ws_gr, l.plan.tiles, c->P, cols, variant, cost, grad);
  return cuda_status(cudaGetLastError(), "optimizer loop evaluation");
}

// ---- allocation-free cost/gradient ---------------------------------------------------
// The scratch of sqg_cost_grad_noalloc: a file-scope device array of fixed size.  In host
// code its name is a host-side stand-in, not a device address; the device address is looked
// up with cudaGetSymbolAddress in the CUDA context that is current for the call, once per
// context (a device normally has one, its primary context; a cudaDeviceReset or a driver-API
// context made current gives the device another, and the array another address).
static __device__ __align__(256) unsigned char g_noalloc_scratch[SQG_NOALLOC_SCRATCH_BYTES];

namespace {
typedef CUresult (*CtxGetCurrentFn)(CUcontext*);
typedef CUresult (*CtxGetIdFn)(CUcontext, unsigned long long*);

struct NoallocSlot {
  unsigned long long ctx_id;
  void* addr;
};
constexpr int kNoallocSlots = 64;
std::mutex g_noalloc_mu;
NoallocSlot g_noalloc_slots[kNoallocSlots] = {};
int g_noalloc_used = 0;
CtxGetCurrentFn g_ctx_current = nullptr;
CtxGetIdFn g_ctx_id = nullptr;

// Unique id of the current CUDA context (*have = false when none is current).  The two
// driver functions are reached through the runtime's entry-point lookup, so the library
// does not link the driver library itself.
int current_context(unsigned long long* id, bool* have) {
  if (!g_ctx_current || !g_ctx_id) {
    cudaDriverEntryPointQueryResult q1, q2;
    cudaError_t e1 = cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", (void**)&g_ctx_current, 12000,
                                                      cudaEnableDefault, &q1);
    cudaError_t e2 = cudaGetDriverEntryPointByVersion("cuCtxGetId", (void**)&g_ctx_id, 12000, cudaEnableDefault, &q2);
    if (e1 != cudaSuccess || e2 != cudaSuccess || q1 != cudaDriverEntryPointSuccess ||
        q2 != cudaDriverEntryPointSuccess || !g_ctx_current || !g_ctx_id) {
      g_ctx_current = nullptr;
      g_ctx_id = nullptr;
      return fail(SQG_ERR_CUDA, "cannot reach cuCtxGetCurrent/cuCtxGetId through the CUDA runtime");
    }
  }
  CUcontext ctx = nullptr;
  if (g_ctx_current(&ctx) != CUDA_SUCCESS) return fail(SQG_ERR_CUDA, "cuCtxGetCurrent failed");
  *have = ctx != nullptr;
  if (!ctx) return SQG_OK;
  if (g_ctx_id(ctx, id) != CUDA_SUCCESS) return fail(SQG_ERR_CUDA, "cuCtxGetId failed");
  return SQG_OK;
}

// Device address of the scratch array in the current context.
int noalloc_scratch(void** out) {
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  unsigned long long id = 0;
  bool have = false;
  int st = current_context(&id, &have);
  if (st) return st;
  if (have) {
    for (int i = 0; i < g_noalloc_used && i < kNoallocSlots; ++i)
      if (g_noalloc_slots[i].ctx_id == id) {
        *out = g_noalloc_slots[i].addr;
        return SQG_OK;
      }
  }
  void* p = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
  if (e != cudaSuccess) return cuda_status(e, "cudaGetSymbolAddress(no-alloc scratch)");
  if (!have) {  // the runtime has just made its context current
    if ((st = current_context(&id, &have))) return st;
    if (!have) return fail(SQG_ERR_CUDA, "no CUDA context is current after cudaGetSymbolAddress");
  }
  g_noalloc_slots[g_noalloc_used % kNoallocSlots] = {id, p};
  ++g_noalloc_used;
  *out = p;
  return SQG_OK;
}
}  // namespace

extern "C" {

int sqg_cost_grad_noalloc(const sqg_circuit* c, const double* theta, int B, const void* target, int cols,
                          long long target_batch_stride, int trace_offset, int variant, double* cost, double* grad,
                          int checkpoint_interval, void* stream) {
  int st = cost_grad_args(c, theta, B, target, cols, trace_offset, variant, cost, grad, checkpoint_interval);
  if (st) return st;
  const bool with_grad = grad != nullptr && c->P > 0;
  if (with_grad && checkpoint_interval == 0) {
    // up to five qubits the environment-matrix form takes no scratch at all
    const int off = variant == SQG_FROBENIUS_NORM ? trace_offset : 0;
    st = sqg::env_cost_grad(c, theta, B, target, cols, target_batch_stride, off, variant, cost, grad, stream);
    if (st != SQG_ERR_UNSUPPORTED) return st;
  }
  const size_t need =
      eval_layout_within(c, B, cols, with_grad, with_grad ? checkpoint_interval : 0, SQG_NOALLOC_SCRATCH_BYTES).end;
  if (need > SQG_NOALLOC_SCRATCH_BYTES)
    return fail(SQG_ERR_WORKSPACE, "sqg_cost_grad_noalloc: this call needs " + std::to_string(need) +
                                       " bytes of scratch but the built-in array holds " +
                                       std::to_string((size_t)SQG_NOALLOC_SCRATCH_BYTES) +
                                       "; use sqg_cost_grad with a caller-allocated workspace or a smaller batch");
  void* ws = nullptr;
  if ((st = noalloc_scratch(&ws))) return st;
  return sqg_cost_grad(c, theta, B, target, cols, target_batch_stride, trace_offset, variant, cost, grad,
                       checkpoint_interval, ws, SQG_NOALLOC_SCRATCH_BYTES, stream);
}

size_t sqg_apply_workspace_bytes(const sqg_circuit* c, int batch) {
  if (!c || batch <= 0) return 0;
  return prep_layout(c, batch, 0).end;
}

int sqg_apply(const sqg_circuit* c, const double* theta, int B, void* mtx, int cols, long long stride,
              long long batch_stride, int fused, void* workspace, size_t ws_bytes, void* stream) {
  int st = check_circuit(c);
  if (st) return st;
  if (B <= 0 || B > 65535 || !mtx || cols <= 0 || stride < cols)
    return fail(SQG_ERR_INVALID_ARGUMENT, "bad matrix arguments");
  if (c->P > 0 && !theta) return fail(SQG_ERR_INVALID_ARGUMENT, "null parameter array");
  PrepLayout l = prep_layout(c, B, 0);
  if (!workspace || ws_bytes < l.end) return fail(SQG_ERR_WORKSPACE, "workspace too small: need " + std::to_string(l.end));
  if (c->L == 0) return SQG_OK;
  cudaStream_t s = (cudaStream_t)stream;
  char* ws = (char*)workspace;
  if (fused) {
    TilePlan pl = plan_tiles(c->N, cols, false);
    TileArgs a;
    memset(&a, 0, sizeof(a));
    const RotPlan& rp = launch_plan_of(c, (long long)B * pl.tiles, kShortPlanFp64);
    if ((st = launch_plan(c, rp, theta, c->P, B, rot_layout(rp, B, 0), ws, a, s))) return st;
    a.mtx = (double2*)mtx;
    a.bstride = batch_stride;
    a.rstride = stride;
    a.cstride = 1;
    a.cols = cols;
    a.TC = pl.TC;
    a.tiles = pl.tiles;
    if ((st = set_smem(k_tile_forward<true, false, kRotFwd>, pl.smem))) return st;
    k_tile_forward<true, false, kRotFwd><<<dim3(pl.tiles, B), pl.threads, pl.smem, s>>>(a);
    return cuda_status(cudaGetLastError(), "k_tile_forward");
  }
  GateMat* gm = (GateMat*)(ws + l.gm_off);
  double2* sc = (double2*)(ws + l.sc_off);
  if ((st = launch_prep(c, theta, c->P, B, gm, sc, s))) return st;
  // unfused: one pass over the matrix per gate
  for (int b = 0; b < B; b++) {
    double2* base = (double2*)mtx + (long long)b * batch_stride;
    for (int g = 0; g < c->L; g++) {
      const Gate& gt = c->h_gates[g];
      if ((gt.type == G_CNOT || gt.type == G_CZ) && c->n >= 2) {
        const int shift = (cols & (cols - 1)) == 0 ? __builtin_ctz((unsigned)cols) : -1;
        const long long items = (long long)cols << (c->n - 2);
        const int blocks = (int)std::min<long long>((items + 1023) / 1024, 152LL * 16);
        if (gt.type == G_CNOT)
          k_perm_hbm<0><<<blocks, 256, 0, s>>>(base, stride, cols, shift, items, gt.target, gt.control);
        else
          k_perm_hbm<1><<<blocks, 256, 0, s>>>(base, stride, cols, shift, items, gt.target, gt.control);
        continue;
      }
      long long items = (long long)cols << (gate_controlled(gt.type) ? c->n - 2 : c->n - 1);
      k_gate_hbm<<<dim3(hbm_blocks(items), 1), 256, 0, s>>>(base, 0, stride, cols, c->n, gt, gm + (long long)b * c->L + g,
                                                          sc + (long long)b * c->P, -1, 1);
    }
  }
  return cuda_status(cudaGetLastError(), "k_gate_hbm");
}

int sqg_apply_from_right(const sqg_circuit* c, const double* theta, void* mtx, int rows, long long stride,
                         void* workspace, size_t ws_bytes, void* stream) {
  int st = check_circuit(c);
  if (st) return st;
  if (!mtx || rows <= 0 || stride < c->N) return fail(SQG_ERR_INVALID_ARGUMENT, "bad matrix arguments");
  if (c->P > 0 && !theta) return fail(SQG_ERR_INVALID_ARGUMENT, "null parameter array");
  PrepLayout l = prep_layout(c, 1, 0);
  if (!workspace || ws_bytes < l.end) return fail(SQG_ERR_WORKSPACE, "workspace too small: need " + std::to_string(l.end));
  if (c->L == 0) return SQG_OK;
  cudaStream_t s = (cudaStream_t)stream;
  TilePlan pl = plan_tiles(c->N, rows, false);
  TileArgs a;
  memset(&a, 0, sizeof(a));
  const RotPlan& rp = launch_plan_of(c, pl.tiles, kShortPlanFp64);
  if ((st = launch_plan(c, rp, theta, c->P, 1, rot_layout(rp, 1, 0), (char*)workspace, a, s))) return st;
  a.mtx = (double2*)mtx;
  a.bstride = 0;
  a.rstride = stride;
  a.cstride = 0;  // vectors are rows
  a.cols = rows;
  a.TC = pl.TC;
  a.tiles = pl.tiles;
  if ((st = set_smem(k_tile_forward<true, false, kRotTrans>, pl.smem))) return st;
  k_tile_forward<true, false, kRotTrans><<<dim3(pl.tiles, 1), pl.threads, pl.smem, s>>>(a);
  return cuda_status(cudaGetLastError(), "k_tile_forward(right)");
}

int sqg_combined_unitary(const sqg_circuit* c, const double* theta, const void* target, int cols, void* out,
                         void* workspace, size_t ws_bytes, void* stream) {
  int st = check_circuit(c);
  if (st) return st;
  if (!target || !out || cols <= 0) return fail(SQG_ERR_INVALID_ARGUMENT, "bad matrix arguments");
  if (c->P > 0 && !theta) return fail(SQG_ERR_INVALID_ARGUMENT, "null parameter array");
  PrepLayout l = prep_layout(c, 1, 0);
  if (!workspace || ws_bytes < l.end) return fail(SQG_ERR_WORKSPACE, "workspace too small: need " + std::to_string(l.end));
  cudaStream_t s = (cudaStream_t)stream;
  char* ws = (char*)workspace;
  GateMat* gm = (GateMat*)(ws + l.gm_off);
  double2* sc = (double2*)(ws + l.sc_off);
  const long long msz = (long long)c->N * cols;
  double2* o = (double2*)out;
  cudaError_t e = cudaMemcpyAsync(o, target, sizeof(double2) * msz, cudaMemcpyDeviceToDevice, s);
  if (e != cudaSuccess) return cuda_status(e, "sqg_combined_unitary");
  if (c->L == 0) return SQG_OK;
  if ((st = launch_prep(c, theta, c->P, 1, gm, sc, s))) return st;
  // out[0] carries the forward state; derivative outputs out[1+k] are created from the
  // state in front of their gate and then carried through the remaining gates
  // (Gates_block::apply_derivate_to, Gates_block.cpp:1012-1150).
  int created = 0;
  for (int g = 0; g < c->L; g++) {
    const Gate& gt = c->h_gates[g];
    int np = gate_param_num(gt.type);
    for (int k = 0; k < np; k++) {
      double2* d = o + msz * (1 + gt.pstart + k);
      e = cudaMemcpyAsync(d, o, sizeof(double2) * msz, cudaMemcpyDeviceToDevice, s);
      if (e != cudaSuccess) return cuda_status(e, "sqg_combined_unitary");
      long long items = (long long)cols << (c->n - 1);
      k_gate_hbm<<<dim3(hbm_blocks(items), 1), 256, 0, s>>>(d, 0, cols, cols, c->n, gt, gm + g, sc, k, 1);
    }
    // forward gate on out[0] and on the derivative outputs created before this gate
    int nmat = 1 + created;
    long long items = (long long)cols << (gate_controlled(gt.type) ? c->n - 2 : c->n - 1);
    k_gate_hbm<<<dim3(hbm_blocks(items), std::min(nmat, 65535)), 256, 0, s>>>(o, msz, cols, cols, c->n, gt, gm + g, sc,
                                                                             -1, nmat);
    created += np;
  }
  return cuda_status(cudaGetLastError(), "sqg_combined_unitary");
}


size_t sqg_state_workspace_bytes(const sqg_circuit* c, int batch) {
  if (!c || batch <= 0) return 0;
  return prep_layout(c, batch, 0).end;
}

int sqg_state_block_count(const sqg_circuit* c) { return c ? (int)choose_state_plan(c, 1).blocks.size() : -1; }

int sqg_apply_state(const sqg_circuit* c, const double* theta, int B, void* states, long long stride, int fused,
                    void* workspace, size_t ws_bytes, void* stream) {
  int st = check_circuit(c, kStateQubits);
  if (st) return st;
  if (B <= 0 || B > 65535 || !states || stride < (long long)c->N)
    return fail(SQG_ERR_INVALID_ARGUMENT, "bad state arguments (batch 1..65535, stride >= 2^qbit_num)");
  if (c->P > 0 && !theta) return fail(SQG_ERR_INVALID_ARGUMENT, "null parameter array");
  PrepLayout l = prep_layout(c, B, 0);
  if (!workspace || ws_bytes < l.end) return fail(SQG_ERR_WORKSPACE, "workspace too small: need " + std::to_string(l.end));
  if (c->L == 0) return SQG_OK;
  cudaStream_t s = (cudaStream_t)stream;
  char* ws = (char*)workspace;
  if (fused) {
    const sqg_state_plan& sp = choose_state_plan(c, B);
    const size_t smem = sizeof(double2) << sp.K;
    if ((st = set_smem(k_state_block, sizeof(double2) << c->splans[0].K))) return st;
    TileArgs t;
    if ((st = launch_plan(c, c->plan, theta, c->P, B, rot_layout(c->plan, B, 0), ws, t, s))) return st;
    StateArgs a;
    a.states = (double2*)states;
    a.stride = stride;
    a.n = c->n;
    a.K = sp.K;
    a.low = std::min(sp.K, kStateLow);
    a.nrecs = t.nrecs;
    a.lops = sp.d_lops;
    a.recs = t.recs;
    a.nphase = t.nphase;
    for (size_t k = 0; k < sp.blocks.size(); k++) {
      a.k0 = sp.blocks[k].k0;
      a.k1 = sp.blocks[k].k1;
      a.phases = k == 0 && t.nphase > 0 ? t.phases : nullptr;
      a.ends = sp.d_lends + 16 * k;
      a.hitab = sp.d_hitab + (k << (a.K - a.low));
      a.inact = sp.d_inact + 32 * k;
      k_state_block<<<dim3(1u << (c->n - sp.K), B), kStateThreads, smem, s>>>(a);
    }
    return cuda_status(cudaGetLastError(), "k_state_block");
  }
  GateMat* gm = (GateMat*)(ws + l.gm_off);
  double2* sc = (double2*)(ws + l.sc_off);
  if ((st = launch_prep(c, theta, c->P, B, gm, sc, s))) return st;
  // unfused: one pass over the state per gate
  for (int b = 0; b < B; b++) {
    double2* base = (double2*)states + (long long)b * stride;
    for (int g = 0; g < c->L; g++) {
      const Gate& gt = c->h_gates[g];
      long long items = 1LL << (gate_controlled(gt.type) ? c->n - 2 : c->n - 1);
      k_gate_hbm<<<dim3(hbm_blocks(items), 1), 256, 0, s>>>(base, 0, 1, 1, c->n, gt, gm + (long long)b * c->L + g,
                                                          sc + (long long)b * c->P, -1, 1);
    }
  }
  return cuda_status(cudaGetLastError(), "k_gate_hbm");
}

}  // extern "C"
