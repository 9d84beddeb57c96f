// Column-tile kernel bodies shared by the fixed-shape launches (engine.cu) and the
// persistent ragged-batch launch (ragged.cu).  Each body processes one (instance, tile)
// work item with all threads of the CTA; smem holds the tile(s) plus reduction scratch.
#pragma once
#include "fx.cuh"
#include "gates.cuh"
#include "rot.cuh"
#include "tile.cuh"

namespace sqg {

struct TileArgs {
  const RotOp* ops;     // operations of the circuit's plan
  const int* ends;      // RotPlan::ends
  int nops, nrecs, noverlaps, n, N;
  const RotRec* recs;   // [B][nrecs]
  const double2* phases;  // [B][nphase]: factors of the phase common to all amplitudes
  int nphase;
  // matrix source (target or in/out matrix); element (r, c) of instance b at
  // base + b*bstride + r*rstride + c*cstride
  double2* mtx;
  long long bstride, rstride, cstride;
  int cols;          // number of vectors (columns for left application, rows for right)
  int TC;            // vectors per tile
  int tiles;         // tiles per instance
  int trace_offset;  // row offset of the traced element (left application)
  double2* ws_tr;    // [B][tiles] forward trace partials
  double* ws_gr;     // [B][tiles][noverlaps] overlaps (complex: noverlaps double2)
  double2* ckpt;     // checkpoints [B][tiles][nck][TC][N] or null
  int ckpt_interval;  // in operations
  int nck;
  int fixed;         // cost and gradient: sweep finite tiles in fixed point
};

// The instance's common phase; finite: whether the numbers of its operations are.
__device__ __forceinline__ double2 tile_phase(const TileArgs& a, int b, bool& finite) {
  double2 p = make_double2(1.0, 0.0);
  finite = true;
  for (int k = 0; k < a.nphase; k++) p = cmul(p, phase_factor(a.phases[(long long)b * a.nphase + k], finite));
  return p;
}

// ends: table of the places behind the last operation (fill_end_table).
__device__ __forceinline__ void load_tile(double2* s, const TileArgs& a, int b, int v0, int tc, const int* ends) {
  const double2* base = a.mtx + (long long)b * a.bstride;
  const int total = a.N * tc;
  if (a.cstride == 1) {
    // left application: vector = column, element r at row r; read rows coalesced
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
      int r = e / tc, c = e - r * tc;
      s[c * a.N + r] = base[(long long)r * a.rstride + v0 + c];
    }
  } else {
    // right application: vector = row (contiguous)
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
      int c = e >> a.n, r = e & (a.N - 1);
      s[c * a.N + end_place(ends, r)] = base[(long long)(v0 + c) * a.rstride + r];
    }
  }
}

// Writes the tile back times the instance's common phase.
__device__ __forceinline__ void store_tile(const double2* s, const TileArgs& a, int b, int v0, int tc, double2 phase,
                                           const int* ends) {
  double2* base = a.mtx + (long long)b * a.bstride;
  const int total = a.N * tc;
  with_phase(phase, [&](auto mul) {
    if (a.cstride == 1) {
      for (int e = threadIdx.x; e < total; e += blockDim.x) {
        int r = e / tc, c = e - r * tc;
        base[(long long)r * a.rstride + v0 + c] = mul(s[c * a.N + end_place(ends, r)]);
      }
    } else {
      for (int e = threadIdx.x; e < total; e += blockDim.x) {
        int c = e >> a.n, r = e & (a.N - 1);
        base[(long long)(v0 + c) * a.rstride + r] = mul(s[c * a.N + r]);
      }
    }
  });
}

// Operations are staged in shared memory kRotChunk at a time, so each CTA reads them from
// global memory once instead of once per warp and operation.
constexpr size_t kStageBytes = kRotChunk * sizeof(StagedOp);

// Turns a tile of tc vectors of N doubles into fixed point in place (Fx2): |amplitude| <= 2^62 under
// the power of two that the largest of the vectors' norms allows.  Returns false, and leaves the
// tile, if it holds an infinity or NaN.  unit: what a result / 2^62 is multiplied by, as two
// factors.  All threads; scratch: kTileMaxWarps doubles.
struct FxUnit {
  double a, b;
};
__device__ __forceinline__ bool fx_from_tile(double2* s, int N, int tc, double* scratch, FxUnit& unit) {
  const int total = tc * N, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  int top = 0;  // largest upper word without its sign
  __syncthreads();
  for (int e = threadIdx.x; e < total; e += blockDim.x) {
    const double2 v = s[e];
    top = max(top, max(__double2hiint(v.x) & 0x7fffffff, __double2hiint(v.y) & 0x7fffffff));
  }
  for (int o = 16; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
  int* tops = reinterpret_cast<int*>(scratch);
  if (lane == 0) tops[warp] = top;
  __syncthreads();
  for (int w = 0; w < nw; w++) top = max(top, tops[w]);
  __syncthreads();
  if (top >= 0x7ff00000) return false;
  // every component is below 2^(e0 + 1); zeros and denormals count as 2^-1023
  const int e0 = top < 0x00100000 ? -1023 : (top >> 20) - 1023;
  auto pow2 = [](int k) { return __hiloint2double((1023 + k) << 20, 0); };
  // 2^-e0 in two factors: e0 spans the whole exponent range
  const int h0 = -e0 / 2, h1 = -e0 - h0;
  const double f0 = pow2(h0), f1 = pow2(h1);
  double norm2 = 0.0;  // the largest of this warp's vectors
  for (int c = warp; c < tc; c += nw) {
    double q = 0.0;
    for (int r = lane; r < N; r += 32) {
      const double2 v = s[c * N + r];
      const double x = v.x * f0 * f1, y = v.y * f0 * f1;
      q = fma(x, x, fma(y, y, q));
    }
    for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
    norm2 = fmax(norm2, q);
  }
  if (lane == 0) scratch[warp] = norm2;
  __syncthreads();
  for (int w = 0; w < nw; w++) norm2 = fmax(norm2, scratch[w]);
  // norm < 2^e1
  const int e1 = norm2 >= 1.0 ? ((__double2hiint(norm2) >> 20) - 1023) / 2 + 1 : 1;
  const double f2 = pow2(kFxBits - e1);
  for (int e = threadIdx.x; e < total; e += blockDim.x) {
    const double2 v = s[e];
    Fx2 w;
    w.x = __double2ll_rn(v.x * f0 * f1 * f2);
    w.y = __double2ll_rn(v.y * f0 * f1 * f2);
    reinterpret_cast<Fx2*>(s)[e] = w;
  }
  __syncthreads();
  unit.a = pow2(-h0);
  unit.b = pow2(e1 - h1);
  return true;
}

// Complex trace partial sum_c s[c][place of first + c], returned to all threads.
__device__ __forceinline__ double2 tile_trace_at(const double2* s, int N, int tc, int first, const int* ends,
                                                 double* scratch, bool fixed, const FxUnit& unit) {
  double2 t = make_double2(0.0, 0.0);
  for (int c = threadIdx.x; c < tc; c += blockDim.x) {
    double2 v = s[c * N + end_place(ends, first + c)];
    if (fixed)
      v = make_double2((double)__double_as_longlong(v.x) * 0x1p-62, (double)__double_as_longlong(v.y) * 0x1p-62);
    t.x += v.x;
    t.y += v.y;
  }
  t.x = block_allsum(t.x, scratch);
  t.y = block_allsum(t.y, scratch);
  if (fixed) t = make_double2(t.x * unit.a * unit.b, t.y * unit.a * unit.b);
  return t;
}

// Application of the whole circuit to one tile (DIR kRotFwd: from the left; kRotTrans: to the
// rows, from the right); optionally writes the tile back and/or the traced diagonal partial.
// Without write-back (cost only) the sweep runs in fixed point.
template <bool WRITE_BACK, bool TRACE, int DIR>
__device__ __forceinline__ void tile_forward_body(const TileArgs& a, int b, int tile, double2* smem) {
  double2* s = smem;
  double* red = reinterpret_cast<double*>(smem + (size_t)a.TC * a.N);
  StagedOp* st = reinterpret_cast<StagedOp*>(red + 2 * kTileMaxWarps);  // [kRotChunk]
  __shared__ int ends[16 * kEndGroups];
  const int v0 = tile * a.TC;
  const int tc = min(a.TC, a.cols - v0);
  bool finite;
  const double2 phase = tile_phase(a, b, finite);
  fill_end_table(ends, a.ends, a.n);
  if (DIR == kRotTrans) __syncthreads();
  load_tile(s, a, b, v0, tc, ends);
  bool fixed = false;
  FxUnit unit;
  if (!WRITE_BACK && a.fixed && finite)
    fixed = fx_from_tile(s, a.N, tc, red, unit);
  const RotRec* recs = a.recs + (long long)b * a.nrecs;
  const int nchunks = (a.nops + kRotChunk - 1) / kRotChunk;
  for (int q = 0; q < nchunks; q++) {
    const int k0 = (DIR == kRotFwd ? q : nchunks - 1 - q) * kRotChunk;
    const int kn = min(kRotChunk, a.nops - k0);
    __syncthreads();  // the previous chunk's operations are no longer read
    if (!WRITE_BACK && fixed)
      fx_stage_ops<true>(st, a.ops, recs, k0, kn, 1.0);
    else
      stage_ops<DIR == kRotFwd, false>(st, a.ops, recs, k0, kn);
    __syncthreads();
    for (int j = 0; j < kn; j++) {
      if (!WRITE_BACK && fixed)
        fx_tile(reinterpret_cast<Fx2*>(s), a.N, a.n, tc, st[j]);
      else
        rot_tile<DIR>(s, a.N, a.n, tc, st[DIR == kRotFwd ? j : kn - 1 - j]);
      __syncthreads();
    }
  }
  __syncthreads();
  if (TRACE) {
    const double2 t = tile_trace_at(s, a.N, tc, v0 + a.trace_offset, ends, red, fixed, unit);
    if (threadIdx.x == 0) a.ws_tr[(long long)b * a.tiles + tile] = phase_mul(phase, t);
  }
  if (WRITE_BACK) store_tile(s, a, b, v0, tc, phase, ends);
}

// Adds the overlaps `mask` of one pair of psi (x, y) and lambda (lx, ly) to acc.  CPLX = false
// (FROBENIUS_NORM needs only the real part of a derivative): acc = Im <X>, Im <Y>, Im of the
// upper rows' <lambda|psi>; 4 + 4 + 2 instructions.  CPLX: acc = the complex overlaps
// <lambda_0|psi_0>, <lambda_0|psi_1>, <lambda_1|psi_0>.
template <bool CPLX, int mask>
__device__ __forceinline__ void measure_pair(double2 x, double2 y, double2 lx, double2 ly,
                                             double (&acc)[CPLX ? 6 : 3]) {
  if (!CPLX) {
    if (mask & 1) {  // Im(conj(lx) y + conj(ly) x)
      acc[0] = fma(lx.x, y.y, fma(-lx.y, y.x, acc[0]));
      acc[0] = fma(ly.x, x.y, fma(-ly.y, x.x, acc[0]));
    }
    if (mask & 2) {  // Im(i (conj(ly) x - conj(lx) y)) = Re(conj(ly) x - conj(lx) y)
      acc[1] = fma(ly.x, x.x, fma(ly.y, x.y, acc[1]));
      acc[1] = fma(-lx.x, y.x, fma(-lx.y, y.y, acc[1]));
    }
    if (mask & 4) acc[2] = fma(lx.x, x.y, fma(-lx.y, x.x, acc[2]));
  } else {
    if (mask & 4) {
      acc[0] = fma(lx.x, x.x, fma(lx.y, x.y, acc[0]));
      acc[1] = fma(lx.x, x.y, fma(-lx.y, x.x, acc[1]));
    }
    if (mask & 3) {
      acc[2] = fma(lx.x, y.x, fma(lx.y, y.y, acc[2]));
      acc[3] = fma(lx.x, y.y, fma(-lx.y, y.x, acc[3]));
      acc[4] = fma(ly.x, x.x, fma(ly.y, x.y, acc[4]));
      acc[5] = fma(ly.x, x.y, fma(-ly.y, x.x, acc[5]));
    }
  }
}

// One measured operation of the reverse sweep on a tile: the overlaps behind it, then its
// adjoint on psi and lambda.
template <bool CPLX, int KIND, int MASK, bool RS>
__device__ __forceinline__ void adjoint_tile_kind(double2* psi, double2* lam, int N, int logN, int tc,
                                                  const StagedOp& staged, double (&acc)[CPLX ? 6 : 3]) {
  const DirOp op = directed<kRotAdj, KIND>(staged);
  const OpPlaces pl = op_places(staged);
  const int lognp = KIND == kOpCry ? logN - 2 : logN - 1;
  const int npairs = 1 << lognp;
  const int items = tc << lognp;
  for (int it = threadIdx.x; it < items; it += blockDim.x) {
    const int col = it >> lognp;
    double2* ps = psi + col * N;
    double2* ls = lam + col * N;
    int ix, iy;
    pair_places<KIND>(pl, it & (npairs - 1), ix, iy);
    double2 x = ps[ix], y = ps[iy], lx = ls[ix], ly = ls[iy];
    measure_pair<CPLX, MASK>(x, y, lx, ly, acc);
    if (KIND == kOpPhase) {
      rot_phase(y, op.zix, op.ziy, op.nzi);
      rot_phase(ly, op.zix, op.ziy, op.nzi);
    } else {
      if (KIND == kOpCry) {
        cry_pair(op, x, y);
        cry_pair(op, lx, ly);
      } else {
        rot_pair<kRotAdj, KIND, RS>(op, x, y);
        rot_pair<kRotAdj, KIND, RS>(op, lx, ly);
      }
      pair_signs(pl, ix, iy, x, y);
      pair_signs(pl, ix, iy, lx, ly);
      ps[ix] = x;
      ls[ix] = lx;
    }
    ps[iy] = y;
    ls[iy] = ly;
  }
}

// The forms that build_rot_plan makes: each kind with the overlaps it is measured with.
template <bool CPLX>
__device__ __forceinline__ void adjoint_tile(double2* psi, double2* lam, int N, int logN, int tc, const StagedOp& st,
                                             double (&acc)[CPLX ? 6 : 3]) {
#define SQG_ROT_CASE(KIND, MASK) \
  case (KIND) | (MASK) << 8: \
    if (st.kind & kStRescale) \
      adjoint_tile_kind<CPLX, (KIND), (MASK), true>(psi, lam, N, logN, tc, st, acc); \
    else \
      adjoint_tile_kind<CPLX, (KIND), (MASK), false>(psi, lam, N, logN, tc, st, acc); \
    break;
  switch (st.kind & 0xffff) {
    case kOpCry | 2 << 8: adjoint_tile_kind<CPLX, kOpCry, 2, false>(psi, lam, N, logN, tc, st, acc); break;
    case kOpPhase | 4 << 8: adjoint_tile_kind<CPLX, kOpPhase, 4, false>(psi, lam, N, logN, tc, st, acc); break;
    SQG_ROT_CASE(kOpRot, 2)
    SQG_ROT_CASE(kOpRot | kOpX, 1)
    SQG_ROT_CASE(kOpRot | kOpZi, 3)
    SQG_ROT_CASE(kOpRot | kOpZi, 6)
    SQG_ROT_CASE(kOpRot | kOpX | kOpZi, 5)
    SQG_ROT_CASE(kOpRot | kOpZi | kOpZo, 7)
  }
#undef SQG_ROT_CASE
}

// Warp totals of the overlaps: lane l ends with value (l >> 3) & 3 (real) or (l >> 2) & 7.
__device__ __forceinline__ double warp_reduce_scatter4(double r0, double r1, double r2) {
  const int lane = threadIdx.x & 31;
  const bool hi = lane & 16;
  double a = (hi ? r2 : r0) + __shfl_xor_sync(0xffffffffu, hi ? r0 : r2, 16);
  double b = hi ? 0.0 : r1;
  const double br = __shfl_xor_sync(0xffffffffu, r1, 16);  // the upper half's r1 goes to the lower half
  if (!hi) b += br;
  const bool odd = lane & 8;
  const double send = odd ? a : b;
  double v = (odd ? b : a) + __shfl_xor_sync(0xffffffffu, send, 8);
  v += __shfl_xor_sync(0xffffffffu, v, 4);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v;
}

// Cost trace and overlaps of one (instance, tile): forward sweep, then the adjoint sweep
// psi <- G^dagger psi, lambda <- G^dagger lambda with lambda starting at e_{j + offset}.
// A U3 run of a CNOT circuit takes 8 products per pair forward and 16 + 6 or 8 on the way back (a
// U3 by itself: 14, 28 and 16 with the gates as given); in fixed point (fx.cuh) unless the tile
// holds infinities or NaN or checkpoints are kept.
template <bool CPLX>
__device__ __forceinline__ void tile_adjoint_body(const TileArgs& a, int b, int tile, double2* smem) {
  constexpr int NV = CPLX ? 8 : 4;  // reduced values per operation (the last ones unused)
  constexpr int NA = CPLX ? 6 : 3;
  const int N = a.N, logN = a.n;
  double2* psi = smem;
  double2* lam = smem + (size_t)a.TC * N;
  double* redd = reinterpret_cast<double*>(lam + (size_t)a.TC * N);  // [2][kTileMaxWarps][4 or 8]
  StagedOp* st = reinterpret_cast<StagedOp*>(redd + kTileMaxWarps * 16);  // [kRotChunk]
  const int v0 = tile * a.TC;
  const int tc = min(a.TC, a.cols - v0);
  const size_t tile_elems = (size_t)a.TC * N;
  double2* ck = a.ckpt ? a.ckpt + ((long long)b * a.tiles + tile) * a.nck * tile_elems : nullptr;
  const RotRec* recs = a.recs + (long long)b * a.nrecs;
  bool finite;
  const double2 phase = tile_phase(a, b, finite);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;

  __shared__ int ends[16 * kEndGroups];
  fill_end_table(ends, a.ends, logN);
  load_tile(psi, a, b, v0, tc, ends);
  for (int e = threadIdx.x; e < tc * N; e += blockDim.x) lam[e] = make_double2(0.0, 0.0);
  bool fixed = false;
  FxUnit unit = {1.0, 1.0};
  if (!ck && a.fixed && finite && (tc <= kFxItems || tc * (N / 2) <= kFxItems * (int)blockDim.x))
    fixed = fx_from_tile(psi, N, tc, redd, unit);
  __syncthreads();
  // <lambda| carries the common phase: lambda_j = conj(phase) e_{j + offset}
  for (int c = threadIdx.x; c < tc; c += blockDim.x) {
    double2 v = cconj(phase);
    if (fixed)
      v = make_double2(__longlong_as_double(__double2ll_rn(v.x * 0x1p62)),
                       __longlong_as_double(__double2ll_rn(v.y * 0x1p62)));
    lam[c * N + end_place(ends, v0 + c + a.trace_offset)] = v;
  }
  // forward sweep, storing psi after every ckpt_interval-th operation
  const int nchunks = (a.nops + kRotChunk - 1) / kRotChunk;
  for (int q = 0; q < nchunks; q++) {
    const int k0 = q * kRotChunk, kn = min(kRotChunk, a.nops - k0);
    __syncthreads();
    if (fixed)
      fx_stage_ops<true>(st, a.ops, recs, k0, kn, 1.0);
    else
      stage_ops<true, false>(st, a.ops, recs, k0, kn);
    __syncthreads();
    for (int j = 0; j < kn; j++) {
      if (fixed)
        fx_tile(reinterpret_cast<Fx2*>(psi), N, logN, tc, st[j]);
      else
        rot_tile<kRotFwd>(psi, N, logN, tc, st[j]);
      __syncthreads();
      if (ck && (k0 + j + 1) % a.ckpt_interval == 0 && (k0 + j + 1) / a.ckpt_interval <= a.nck) {
        double2* dst = ck + (size_t)((k0 + j + 1) / a.ckpt_interval - 1) * tile_elems;
        for (int e = threadIdx.x; e < tc * N; e += blockDim.x) dst[e] = psi[e];
        __syncthreads();  // the next operation changes psi
      }
    }
  }
  __syncthreads();
  double2 t = tile_trace_at(psi, N, tc, v0 + a.trace_offset, ends, redd, fixed, unit);
  if (threadIdx.x == 0) a.ws_tr[(long long)b * a.tiles + tile] = phase_mul(phase, t);
  __syncthreads();

  // reverse sweep.  The warps' totals of an operation are summed and written by the last warp
  // while the next operation runs: redd alternates between two halves, one barrier per operation.
  double* wgr = a.ws_gr + ((long long)b * a.tiles + tile) * a.noverlaps * (CPLX ? 2 : 1);
  int pend_coff = 0, pend_mask = 0, pend_aw = 0, buf = 0;
  double pend_fac = 0.0;
  const int shift = fx_sum_shift(tc);
  // the 2^-60 of a sum goes into the unit where that could exceed the range of a double without it
  const double sum_unit = unit.b >= 1.0 ? 1.0 : 0x1p-60;
  const double fx_unit = fixed ? (double)(1 << shift) * (unit.b >= 1.0 ? 0x1p-60 : 1.0) * unit.a * unit.b : 1.0;
  auto flush = [&]() {  // one thread per measured overlap
    if (!pend_mask || warp != nw - 1 || lane >= 3) return;
    const int axis = lane;  // 0 X, 1 Y, 2 Z
    if (!((pend_mask >> axis) & 1)) return;
    const double* rd = redd + (buf ^ 1) * kTileMaxWarps * 8;
    const int pos = pend_coff + __popc(pend_mask & ((1 << axis) - 1));
    auto total = [&](int k) {
      if (fixed) {
        long long v = 0;
        for (int w = 0; w < pend_aw; w++) v += __double_as_longlong(rd[w * NV + k]);
        return (double)v * sum_unit * pend_fac;
      }
      double v = 0.0;
      for (int w = 0; w < pend_aw; w++) v += rd[w * NV + k];
      return v * pend_fac;
    };
    if (!CPLX) {
      wgr[pos] = total(axis);
    } else {
      double2 v;
      if (axis == 2) v = make_double2(total(0), total(1));                           // <lambda_0|psi_0>
      else if (axis == 0) v = make_double2(total(2) + total(4), total(3) + total(5));  // <X>
      else v = make_double2(total(3) - total(5), total(4) - total(2));                 // <Y> = i (m10 - m01)
      reinterpret_cast<double2*>(wgr)[pos] = v;
    }
  };
  for (int q = nchunks - 1; q >= 0; q--) {
    const int k0 = q * kRotChunk, kn = min(kRotChunk, a.nops - k0);
    __syncthreads();
    if (fixed)
      fx_stage_ops<false>(st, a.ops, recs, k0, kn, fx_unit);
    else
      stage_ops<false, false>(st, a.ops, recs, k0, kn);
    __syncthreads();
    for (int j = kn - 1; j >= 0; j--) {
      const int k = k0 + j;
      // before step k, psi holds the state behind operation k; the stored copy replaces it at
      // checkpoints, so that the error of undoing never spans more than ckpt_interval
      // operations.  Between a group's first and last rotation the copy's scale is all / pre (pre:
      // its cosines up to here, all: of the group) and the one on the way back pre.
      if (ck && (k + 1) % a.ckpt_interval == 0 && (k + 1) / a.ckpt_interval <= a.nck && k + 1 < a.nops) {
        const double2* src = ck + (size_t)((k + 1) / a.ckpt_interval - 1) * tile_elems;
        const double f = st[j].kind & kStInside ? 1.0 / (st[j].mfac * st[j].scale) : 1.0;
        for (int e = threadIdx.x; e < tc * N; e += blockDim.x) psi[e] = cscale(src[e], f);
        __syncthreads();
      }
      const int kind = st[j].kind & 255, mask = (st[j].kind >> 8) & 255;
      if (mask == 0) {  // a CZ by itself
        if (fixed) {
          fx_tile(reinterpret_cast<Fx2*>(psi), N, logN, tc, st[j]);
          fx_tile(reinterpret_cast<Fx2*>(lam), N, logN, tc, st[j]);
        } else {
          rot_tile<kRotAdj>(psi, N, logN, tc, st[j]);
          rot_tile<kRotAdj>(lam, N, logN, tc, st[j]);
        }
        __syncthreads();
        continue;
      }
      const int items = tc << (kind == kOpCry ? logN - 2 : logN - 1);
      const int aw = min(nw, (items + 31) >> 5);  // warps holding pairs
      double* rd = redd + buf * kTileMaxWarps * 8 + warp * NV;
      if (fixed) {
        long long acc[NA];
#pragma unroll
        for (int r = 0; r < NA; r++) acc[r] = 0;
        fx_adjoint<CPLX>(reinterpret_cast<Fx2*>(psi), reinterpret_cast<Fx2*>(lam), N, logN, tc, st[j], acc);
        if (warp < aw) {
          long long r[8] = {};
#pragma unroll
          for (int i = 0; i < NA; i++) r[i] = fx_scaled(acc[i], shift);
          const long long v = fx_reduce_scatter8(r);
          if ((lane & 3) == 0 && (lane >> 2) < NV) rd[lane >> 2] = __longlong_as_double(v);
        }
      } else {
        double acc[NA];
#pragma unroll
        for (int r = 0; r < NA; r++) acc[r] = 0.0;
        adjoint_tile<CPLX>(psi, lam, N, logN, tc, st[j], acc);
        if (warp < aw) {
          if constexpr (CPLX) {
            double r[8] = {acc[0], acc[1], acc[2], acc[3], acc[4], acc[5], 0.0, 0.0};
            const double v = warp_reduce_scatter8(r);
            if ((lane & 3) == 0) rd[lane >> 2] = v;
          } else {
            const double v = warp_reduce_scatter4(acc[0], acc[1], acc[2]);
            if ((lane & 7) == 0) rd[((lane >> 4) & 1) * 2 + ((lane >> 3) & 1)] = v;
          }
        }
      }
      flush();  // the operation before this one
      __syncthreads();
      pend_coff = st[j].coff;
      pend_mask = mask;
      pend_aw = aw;
      pend_fac = st[j].mfac;
      buf ^= 1;
    }
  }
  flush();
}

// Shared memory bytes of one work item: tiles plus reduction scratch.
__host__ __device__ inline size_t tile_smem_bytes(int TC, int N, bool grad) {
  size_t per = (size_t)N * sizeof(double2) * (grad ? 2 : 1);
  size_t extra = grad ? kTileMaxWarps * 16 * sizeof(double) + kStageBytes
                      : kTileMaxWarps * sizeof(double2) + kStageBytes;
  return per * TC + extra;
}

}  // namespace sqg
