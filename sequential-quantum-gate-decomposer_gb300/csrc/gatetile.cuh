// Cost and adjoint gradient gate by gate in FP64, for the device optimizer loops of registers that
// the environment-matrix evaluation does not take.
//
// BFGS and ADAM trajectories amplify the rounding of every evaluation (40 evaluations at six qubits: a
// change of the last place of cost and gradient moves the best point by 1e-8, now and then by far more), so
// which point a decomposition returns is a property of this arithmetic: the order of the gates and
// of every sum stays as it is, and the rotation plan (rot.cuh), which is faster and as accurate, is left
// to the evaluations whose result is the cost and gradient themselves.  GB300, six qubits, 20 blocks: 291 us
// per evaluation of the loop, against 212 us with the plan.  Bound by the latency of the serial
// gates: a tile is one column of one vector.
#pragma once
#include "gates.cuh"
#include "tile.cuh"

namespace sqg {

struct GateTileArgs {
  const Gate* gates;
  const GateMat* gm;   // [L]
  const double2* sc;   // [P]
  const double2* target;
  int L, P, n, N, cols, TC, tiles, trace_offset;
  double2* ws_tr;  // [tiles] trace partials
  double2* ws_gr;  // [tiles][P] derivative trace partials
};

// One tile of TC columns; all threads of the CTA.
__device__ __forceinline__ void gate_adjoint_body(const GateTileArgs& a, int tile, double2* smem) {
  const int N = a.N, logN = a.n;
  double2* psi = smem;
  double2* lam = smem + (size_t)a.TC * N;
  double* redd = reinterpret_cast<double*>(lam + (size_t)a.TC * N);  // [kTileMaxWarps][8]
  double* tot = redd + kTileMaxWarps * 8;                             // [8]
  double* scratch = tot + 8;                                          // [kTileMaxWarps]
  GateMat* gst = reinterpret_cast<GateMat*>(scratch + kTileMaxWarps);  // [kStage]
  Gate* gts = reinterpret_cast<Gate*>(gst + kStage);                  // [kStage]
  const int v0 = tile * a.TC;
  const int tc = min(a.TC, a.cols - v0);
  for (int e = threadIdx.x; e < tc * N; e += blockDim.x) {  // rows read coalesced
    const int r = e / tc, c = e - r * tc;
    psi[c * N + r] = a.target[(long long)r * a.cols + v0 + c];
  }
  for (int e = threadIdx.x; e < tc * N; e += blockDim.x) {  // lambda_j = e_{j + offset}
    const int c = e / N, r = e - c * N;
    lam[e] = make_double2(r == v0 + c + a.trace_offset ? 1.0 : 0.0, 0.0);
  }
  __syncthreads();
  for (int g = 0; g < a.L; g++) {
    const int j = g % kStage;
    if (j == 0) {
      __syncthreads();
      if ((int)threadIdx.x < min(kStage, a.L - g)) {
        gts[threadIdx.x] = a.gates[g + threadIdx.x];
        gst[threadIdx.x] = a.gm[g + threadIdx.x];
      }
      __syncthreads();
    }
    const Gate gt = gts[j];
    tile_apply(psi, N, logN, tc, gt, make_op(gt.type, gst[j], ORIENT_FWD));
    __syncthreads();
  }
  const double2 t = tile_trace(psi, N, tc, v0, a.trace_offset, scratch);
  if (threadIdx.x == 0) a.ws_tr[tile] = t;
  double2* wgr = a.ws_gr + (long long)tile * a.P;
  auto sink = [&](int, const Gate& gt, const double* R) {
    if (threadIdx.x < gate_param_num(gt.type)) wgr[gt.pstart + threadIdx.x] = contract_derivative(gt, a.sc, threadIdx.x, R);
  };
  adjoint_sweep(psi, lam, N, logN, tc, a.gates, a.gm, a.sc, a.L, redd, tot, sink, gts, gst);
}

inline size_t gate_tile_smem_bytes(int TC, int N) {
  return 2 * (size_t)N * TC * sizeof(double2) + (kTileMaxWarps * 8 + 8 + kTileMaxWarps) * sizeof(double) +
         kStage * (sizeof(Gate) + sizeof(GateMat));
}

}  // namespace sqg
