// Definition of the opaque circuit handle shared by the engine's translation units, and
// the thread-local error text behind sqg_last_error().
#pragma once
#include <string>
#include <vector>

#include "gates.cuh"
#include "rotplan.h"

// Fused state-vector passes (sqg_apply_state): consecutive gates whose qubits, together with
// the lowest ones, fit one chunk of 2^K amplitudes form a block applied in shared memory.
struct sqg_state_block {
  int k0, k1;  // operations [k0, k1) of the state-vector plan
};

// A plan of such passes: chunk qubits K, blocks, operations on chunk-local qubits, per block the
// places behind its last operation (K ints, padded to 16), the global offsets of the chunk's high
// local bits (2^(K - low) ints) and the qubits that number the chunks (padded to 32).  lops to inact: where
// these arrays are in their device allocation.
struct sqg_state_plan {
  int K = 0, nops = 0;
  std::vector<sqg_state_block> blocks;
  size_t lops = 0, lends = 0, hitab = 0, inact = 0;
  const sqg::RotOp* d_lops = nullptr;
  const int *d_lends = nullptr, *d_hitab = nullptr, *d_inact = nullptr;
};

struct sqg_circuit {
  int n = 0, N = 0, L = 0, P = 0;
  int device = 0;
  sqg::Gate* d_gates = nullptr;
  std::vector<sqg::Gate> h_gates;
  // rotation plan (rot.cuh): the host's steps, from which the operations of the state-vector
  // blocks are made, and the device arrays, one allocation with the gates and state-vector plans behind
  // d_plan.
  // short_plan: the same with short chains, for launches that wait for the chains.
  std::vector<sqg::RotStep> h_steps;
  void* d_plan = nullptr;
  sqg::RotPlan plan = {}, short_plan = {};
  // state-vector plans, the first with the largest chunks; d_state: the arrays of those that follow
  // handed-over partitions
  std::vector<sqg_state_plan> splans;
  void* d_state = nullptr;
};

namespace sqg {
// Records msg as the calling thread's last error and returns status.
int set_error(int status, const std::string& msg);
// Environment-matrix cost and gradient for qbit_num <= 5 (decompose.cu); SQG_ERR_UNSUPPORTED
// for shapes it does not take.
int env_cost_grad(const sqg_circuit* c, const double* theta, int B, const void* target, int cols, long long tstride,
                  int off, int variant, double* cost, double* grad, void* stream);
// Cost and gradient of one vector inside the device optimizer loops: env_cost_grad where it takes the
// call, else gate by gate in FP64 (gatetile.cuh).  Arguments as checked by the loops; off: the trace
// offset that the variant uses.
size_t loop_cost_grad_bytes(const sqg_circuit* c, int cols);
int loop_cost_grad(const sqg_circuit* c, const double* theta, const void* target, int cols, int off, int variant,
                   double* cost, double* grad, void* workspace, size_t ws_bytes, void* stream);
}  // namespace sqg
