// From the overlaps of the reverse sweep to the cost and the gradient.
#pragma once
#include "../../include/sqg.h"
#include "rot.cuh"
#include "tile.cuh"

namespace sqg {

// Cost of a variant from the trace tr over `cols` columns (Optimization_Interface.cpp:677-735).
__device__ __forceinline__ double cost_from_trace(int variant, double2 tr, int cols) {
  const double d = cols;
  if (variant == SQG_FROBENIUS_NORM) return 1.0 - tr.x / d;
  if (variant == SQG_HILBERT_SCHMIDT_TEST) {
    const double q = 1.0 / d;
    return 1.0 - q * q * (tr.x * tr.x + tr.y * tr.y);
  }
  return 1.0 - ((tr.x * tr.x + tr.y * tr.y) / d + 1) / (d + 1);
}

// Gradient component from the derivative dt of the trace (Optimization_Interface.cpp:1397-1458).
__device__ __forceinline__ double grad_from_trace(int variant, double2 tr, double2 dt, int cols) {
  const double d = cols;
  if (variant == SQG_FROBENIUS_NORM) return (1.0 - dt.x / d) - 1.0;
  if (variant == SQG_HILBERT_SCHMIDT_TEST) {
    const double q = 1.0 / d;
    return -2.0 * q * q * tr.x * dt.x - 2.0 * q * q * tr.y * dt.y;
  }
  return -2.0 / d / (d + 1) * tr.x * dt.x - 2.0 / d / (d + 1) * tr.y * dt.y;
}

constexpr int kSumGroups = 8;  // threads that share the tiles of one overlap

// Sums the tiles of 32 overlaps of one instance (ws_gr, W doubles each) into tile 0's place, in
// a fixed order; CTA 0 also sums the trace into tile 0's place and writes the cost.
// blockDim = 32 * kSumGroups.
template <int W>
__device__ __forceinline__ void tile_sum_body(int part, double2* tr, double* gr, int tiles, int noverlaps, int cols,
                                              int variant, double* cost) {
  __shared__ double sums[kSumGroups][32 * W];
  __shared__ double scratch[kTileMaxWarps];
  const int o = threadIdx.x & 31, grp = threadIdx.x >> 5;
  const int k = part * 32 + o;
  if (noverlaps > 0) {
    double v[W];
#pragma unroll
    for (int w = 0; w < W; w++) v[w] = 0.0;
    if (k < noverlaps)
#pragma unroll 4
      for (int t = grp; t < tiles; t += kSumGroups)
#pragma unroll
        for (int w = 0; w < W; w++) v[w] += gr[((long long)t * noverlaps + k) * W + w];
#pragma unroll
    for (int w = 0; w < W; w++) sums[grp][o * W + w] = v[w];
    __syncthreads();
    for (int j = threadIdx.x; j < 32 * W; j += blockDim.x) {
      const int kk = part * 32 * W + j;
      double s = 0.0;
      for (int g = 0; g < kSumGroups; g++) s += sums[g][j];
      if (kk < noverlaps * W) gr[kk] = s;
    }
  }
  if (part == 0) {
    double2 t = make_double2(0.0, 0.0);
    for (int i = threadIdx.x; i < tiles; i += blockDim.x) t = cadd(t, tr[i]);
    t.x = block_allsum(t.x, scratch);
    t.y = block_allsum(t.y, scratch);
    if (threadIdx.x == 0) {
      tr[0] = t;
      *cost = cost_from_trace(variant, t, cols);
    }
  }
}

// v = <P> behind a rotation about `axis` by the full angle (c, s) becomes <P> in front of it.
__device__ __forceinline__ void undo_rotation(int axis, double c, double s, double2 v[3]) {
  const int p = axis % 3, q = (axis + 1) % 3;  // X: (Y, Z), Y: (Z, X), Z: (X, Y), counted from 0
  const double2 a = v[p], b = v[q];
  v[p] = make_double2(fma(c, a.x, s * b.x), fma(c, a.y, s * b.y));
  v[q] = make_double2(fma(c, b.x, -(s * a.x)), fma(c, b.y, -(s * a.y)));
}
// The same rotation on coefficients r of <P> in front of it: they become those behind it.
__device__ __forceinline__ void undo_coeffs(int axis, double c, double s, double r[3]) {
  const int p = axis % 3, q = (axis + 1) % 3;
  const double a = r[p], b = r[q];
  r[p] = fma(c, a, -(s * b));
  r[q] = fma(s, a, c * b);
}

// (cos, sin) of the double angle.
__device__ __forceinline__ double2 twice(double2 a) {
  return make_double2((a.x - a.y) * (a.x + a.y), 2.0 * a.x * a.y);
}

// Gradient components of the gates of one CTA's runs (kRotThreads threads, thread i for run i).
// tr: the trace; gr: the summed overlaps.  The overlap along the axis that a run pushed is the
// one that the next run of its chain has in front of its gates.
template <bool CPLX>
__device__ __forceinline__ void rot_grad_body(const RotPlan& pl, int cta, const double* theta, const RotRec* recs,
                                              const double2* tr, const double* gr, int cols, int variant,
                                              double* grad) {
  __shared__ double2 sc[kRotParams];
  __shared__ double2 V[kRotThreads][3];
  __shared__ double R[kRotThreads][3];
  const int base = pl.cta[cta], n = pl.cta[cta + 1] - base, i = threadIdx.x;
  const double2 T = tr[0];
  cta_sincos(pl, cta, theta, sc);
  __syncthreads();
  RotRun run;
  double2 wrot = make_double2(1.0, 0.0);
  if (i < n) {
    run = pl.runs[base + i];
    if (run.push != kAxisNone) wrot = recs[run.rec].zo;
    double2 v[3];
    int pos = run.coff;
    for (int axis = 0; axis < 3; axis++) {
      v[axis] = make_double2(0.0, 0.0);
      if (!((run.mask >> axis) & 1)) continue;
      v[axis] = CPLX ? reinterpret_cast<const double2*>(gr)[pos] : make_double2(0.0, gr[pos]);
      if (axis == 2) v[axis] = make_double2(2.0 * v[axis].x - T.x, 2.0 * v[axis].y - T.y);
      pos++;
    }
    for (int axis = 0; axis < 3; axis++) V[i][axis] = v[axis];
    if (run.pulled) {  // <axis pulled> in front of the run from <P> behind it
      double r[3] = {0.0, 0.0, 0.0};
      r[pl.runs[base + i - 1].push - 1] = 1.0;
      int soff = run.soff;
      for (int k = 0; k < run.count; k++) {
        const Gate g = pl.gates[pl.members[run.first + k]];
        const double* th = theta + g.pstart;
        const double2 a = twice(param_sincos(sc, soff, th, 0));
        if (g.type == G_U3) {
          const double2 ph = param_sincos(sc, soff, th, 1), la = param_sincos(sc, soff, th, 2);
          undo_coeffs(kAxisZ, la.x, la.y, r);
          undo_coeffs(kAxisY, a.x, a.y, r);
          undo_coeffs(kAxisZ, ph.x, ph.y, r);
        } else {
          undo_coeffs(g.type == G_RX ? kAxisX : g.type == G_RY ? kAxisY : kAxisZ, a.x, a.y, r);
        }
        if (soff >= 0) soff += gate_param_num(g.type);
      }
      if (run.push != kAxisNone) undo_coeffs(run.push, wrot.x, -wrot.y, r);
      for (int axis = 0; axis < 3; axis++) R[i][axis] = r[axis];
    }
  }
  __syncthreads();
  if (i < n && run.pulled && run.push == kAxisNone) {
    RotRun r = run;
    for (int j = i, step = 0; r.pulled && step < kRotChain; j--, step++) {
      double2 c = make_double2(0.0, 0.0);
      for (int axis = 0; axis < 3; axis++) {
        c.x = fma(R[j][axis], V[j][axis].x, c.x);
        c.y = fma(R[j][axis], V[j][axis].y, c.y);
      }
      r = pl.runs[base + j - 1];
      V[j - 1][r.push - 1] = c;
    }
  }
  __syncthreads();
  if (i >= n) return;
  double2 v[3] = {V[i][0], V[i][1], V[i][2]};
  // behind the run's last gate the state carries the pushed rotation W too: <W^dagger P W>
  if (run.push != kAxisNone) undo_rotation(run.push, wrot.x, -wrot.y, v);
  auto put = [&](int p, double2 dt) { grad[p] = grad_from_trace(variant, T, dt, cols); };
  auto minus_i = [](double2 a) { return make_double2(a.y, -a.x); };                       // d/dangle of e^{-i angle P}
  auto half_i = [&](double2 z) { return make_double2(-0.5 * (T.y - z.y), 0.5 * (T.x - z.x)); };  // of diag(1, e^{i angle})
  int soff = run.soff;
  for (int k = 0; soff >= 0 && k < run.count; k++) soff += gate_param_num(pl.gates[pl.members[run.first + k]].type);
  for (int k = run.count - 1; k >= 0; k--) {
    const Gate g = pl.gates[pl.members[run.first + k]];
    const double* th = theta + g.pstart;
    if (soff >= 0) soff -= gate_param_num(g.type);
    if (g.type == G_U3) {
      const double2 ph = param_sincos(sc, soff, th, 1), a = twice(param_sincos(sc, soff, th, 0));
      put(g.pstart + 1, half_i(v[2]));
      undo_rotation(kAxisZ, ph.x, ph.y, v);
      put(g.pstart, minus_i(v[1]));
      undo_rotation(kAxisY, a.x, a.y, v);
      put(g.pstart + 2, half_i(v[2]));
      if (k > 0) {
        const double2 la = param_sincos(sc, soff, th, 2);
        undo_rotation(kAxisZ, la.x, la.y, v);
      }
    } else {
      const int axis = g.type == G_RX ? kAxisX : g.type == G_RZ ? kAxisZ : kAxisY;
      put(g.pstart, minus_i(v[axis - 1]));
      if (k > 0) {
        const double2 a = twice(param_sincos(sc, soff, th, 0));
        undo_rotation(axis, a.x, a.y, v);
      }
    }
  }
}

}  // namespace sqg
