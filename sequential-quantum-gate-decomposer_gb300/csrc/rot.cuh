// Rotation plan of a circuit: the form in which the tile and state kernels apply it.
//
// What bounds these kernels is the number of FP64 instructions per amplitude pair (the FP64
// pipe takes two lanes per clock and SM; every other pipe is nearly idle), so the plan rewrites
// the gate list into operations with as few of them as the circuit allows:
//  * A run of single-qubit gates on one qubit, with no two-qubit gate on that qubit between
//    them, is one 2x2 unitary M.
//  * M = scalar * diag(1, zo) * R * diag(1, zi) with R a rotation.  R is applied without its
//    cosine ([[1, -t], [t, 1]], |t| <= 1 after an exchange of the two rows where needed):
//    4 multiply-adds per pair instead of 8.  The cosines of up to kRotChunk consecutive
//    operations are multiplied back in one of them, so the scale never leaves [1, 2^16].
//    A phase diag(1, z) touches one row of the pair: 4 instructions.
//  * The rotation that M ends with is moved through the next two-qubit gate into the next run
//    on the qubit where it commutes with that gate: Z through a control or a CZ, X through a
//    CNOT target, Y through a CRY target.  What is left of M is R * diag(1, zi): 8
//    instructions per pair, against 14 of a U3 as given.
//  * Phases common to all amplitudes are collected per instance and multiplied in once.
//  * The gradient needs only <lambda| P |psi> for the Paulis P at the end of each run; the one
//    along the axis that the run pushes equals that of the next run and is not measured, and
//    the derivatives of the run's gates follow from these three numbers, once per run (rot_grad_body), not per amplitude.
// Measured on GB300 against the gates as given (U3 14 instructions, merged runs 16): gradient at
// 8 qubits, 360 blocks, 128 vectors 333 -> 182 ms; cost alone, 120 blocks, 200 vectors 41.5 ->
// 25.3 ms; 2000 random gates on a 4096 x 4096 matrix 143 -> 99 ms; 829 gates on 24 qubits 128 ->
// 86 ms.  The FP64 pipe is 91 % busy either way.
// The numbers behind each operation depend on the parameters and are made per instance by
// rot_plan_body; which operations there are depends on the gate list alone (build_rot_plan).
#pragma once
#include "gates.cuh"

namespace sqg {

// Kinds of operations.  kOpRot carries flags: rotation about X instead of Y, phase before
// (zi), phase after (zo).
enum : int { kOpCnot = 0, kOpCz = 1, kOpCry = 2, kOpPhase = 3, kOpRot = 4, kOpX = 8, kOpZi = 16, kOpZo = 32 };
enum : int { kAxisNone = 0, kAxisX = 1, kAxisY = 2, kAxisZ = 3 };

// One operation of the plan.  coff: first of its overlaps in the instance's overlap list;
// mask: which are measured (1 X, 2 Y, 4 Z; kOpCry: 2, on the controlled half).
struct RotOp {
  int kind;
  int qubits;  // target | control << 8
  int coff;
  int mask;
};

// One run (or CRY gate): its operation, its gates members[first .. first + count), the axis it
// pushes (kAxisNone: nothing) into the run right behind it in the chain order, whether the run
// before it pushes into it, a copy of its operation's kind, coff and mask, and whether it is a
// single U3.
struct RotRun {
  int op, first, count, push, pulled, kind, coff, mask, lone_u3;
};

// Numbers of one operation.  t, c: tangent and cosine of the rotation (kOpCry: sine and
// cosine, lo: what c lacks to the exact cosine of t); turn: the two rows are exchanged between
// zi and the rotation (a quarter turn about Y with its sign in zi, about X up to a phase).  zo of
// a run that pushes holds (cos, sin) of the pushed rotation's full angle.
struct RotRec {
  double t, c;
  double2 zi, zo;
  double lo;
  long long turn;
};
static_assert(sizeof(RotRec) == sizeof(GateMat), "the workspace counts both as 64 bytes");

// Device view of a circuit's plan.
struct RotPlan {
  const Gate* gates;
  const RotOp* ops;
  const RotRun* runs;
  const int* members;
  const int* cta;  // runs [cta[i], cta[i + 1]) are handled by one CTA of kRotThreads threads
  int nops, ncta, noverlaps;
};

constexpr int kRotThreads = 128;  // runs per CTA of the per-instance kernels; no chain straddles two
constexpr int kRotChain = 16;     // runs linked by pushed rotations (their numbers are made one after another)
constexpr int kRotChunk = 32;     // operations staged in shared memory together

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cmulc(double2 a, double2 b) {  // a * conj(b)
  return make_double2(fma(a.x, b.x, a.y * b.y), fma(a.y, b.x, -a.x * b.y));
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cscale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double cnorm2(double2 a) { return fma(a.x, a.x, a.y * a.y); }
// One Newton step towards |z| = 1 for z that is a few roundings away from it.
__device__ __forceinline__ double2 cunit(double2 z) { return cscale(z, fma(-0.5, cnorm2(z), 1.5)); }

// M <- G M
__device__ __forceinline__ void matmul2(const double2 G[4], double2 M[4]) {
  const double2 a = M[0], b = M[1];
  M[0] = cadd(cmul(G[0], a), cmul(G[1], M[2]));
  M[1] = cadd(cmul(G[0], b), cmul(G[1], M[3]));
  M[2] = cadd(cmul(G[2], a), cmul(G[3], M[2]));
  M[3] = cadd(cmul(G[2], b), cmul(G[3], M[3]));
}

// Full 2x2 matrix of a single-qubit gate from its stored parameters.
__device__ __forceinline__ void gate_matrix(int type, const double* th, double2 u[4]) {
  double s, c;
  sincos(th[0], &s, &c);
  if (type == G_U3) {
    double sp, cp, sl, cl;
    sincos(th[1], &sp, &cp);
    sincos(th[2], &sl, &cl);
    u[0] = make_double2(c, 0.0);
    u[1] = make_double2(-s * cl, -s * sl);
    u[2] = make_double2(s * cp, s * sp);
    u[3] = make_double2(c * (cp * cl - sp * sl), c * (sp * cl + cp * sl));
  } else if (type == G_RX) {
    u[0] = u[3] = make_double2(c, 0.0);
    u[1] = u[2] = make_double2(0.0, -s);
  } else if (type == G_RZ) {
    u[0] = make_double2(c, -s);
    u[1] = u[2] = make_double2(0.0, 0.0);
    u[3] = make_double2(c, s);
  } else {  // RY, CRY
    u[0] = u[3] = make_double2(c, 0.0);
    u[1] = make_double2(-s, 0.0);
    u[2] = make_double2(s, 0.0);
  }
}

// The cosine 1 / sqrt(1 + t^2) of a rotation by its tangent, as c + lo: tens of them are
// multiplied into one scale, and c alone would put a rounding of each on every amplitude.
__device__ __forceinline__ void set_cosine(RotRec& r) {
  const double t2 = r.t * r.t, t2e = fma(r.t, r.t, -t2);
  const double s = 1.0 + t2, se = (1.0 - s) + t2 + t2e;
  r.c = 1.0 / sqrt(s);
  const double c2 = r.c * r.c, c2e = fma(r.c, r.c, -c2);
  const double p = c2 * s, pe = fma(c2, s, -p) + fma(c2e, s, c2 * se);
  r.lo = 0.5 * r.c * ((1.0 - p) - pe);
}

// M (unitary) as scalar * diag(1, zo) * R * [exchange] * diag(1, zi); returns the scalar's
// phase.  The larger entry of the first column is the pivot, so |t| <= 1.
__device__ __forceinline__ double2 split_zyz(const double2 M[4], RotRec& r) {
  const double na = cnorm2(M[0]), nc = cnorm2(M[2]);
  const bool turn = nc > na;
  const double2 piv = turn ? M[2] : M[0], oth = turn ? M[0] : M[2];
  const double np = turn ? nc : na;
  const double2 q = cscale(cmulc(oth, piv), 1.0 / np);  // f = 0: t zo, f = 1: -t / zo
  const double t2 = cnorm2(q), t = sqrt(t2);
  double2 zo = make_double2(1.0, 0.0);
  if (t2 > 1e-280) zo = cscale(turn ? make_double2(-q.x, q.y) : q, 1.0 / t);
  zo = cunit(zo);
  // turn = 0: zi = (d / a) / zo;  turn = 1: zi = -(b / c) zo
  const double2 w = cscale(cmulc(turn ? M[1] : M[3], piv), 1.0 / np);
  double2 zi = turn ? cmul(make_double2(-w.x, -w.y), zo) : cmulc(w, zo);
  zi = cunit(cunit(zi));
  r.turn = turn;
  r.t = t;
  set_cosine(r);
  // the quarter turn (x, y) -> (-y, x) as an exchange: its sign goes into zi
  r.zi = turn ? make_double2(-zi.x, -zi.y) : zi;
  r.zo = zo;
  const double2 u = cscale(piv, 1.0 / sqrt(np));
  return turn ? cmulc(u, zo) : u;
}

// M (unitary) as W * Ry(atan t) * diag(1, zi) with W = phase * Rx: W is returned in w00, w01
// (its diagonal and off-diagonal entry).  |t| <= 1 always.
__device__ __forceinline__ void split_x(const double2 M[4], RotRec& r, double2& w00, double2& w01) {
  // (M00^2 - M10^2) / det M = e^{-2 i gamma} cos 2 beta, with zi = e^{2 i gamma}
  const double2 det = csub(cmul(M[0], M[3]), cmul(M[1], M[2]));
  const double2 d = cmulc(csub(cmul(M[0], M[0]), cmul(M[2], M[2])), det);
  const double nd2 = cnorm2(d), nd = sqrt(nd2);
  const double s = cnorm2(M[0]) + cnorm2(M[2]);
  double2 zi = make_double2(1.0, 0.0);
  if (nd2 > 1e-280) zi = cunit(make_double2(d.x / nd, -d.y / nd));
  const double sb = 2.0 * fma(M[0].x, M[2].x, M[0].y * M[2].y);
  r.t = sb / (s + nd);
  set_cosine(r);
  const double c = r.c, sn = r.t * c;
  // W = M diag(1, conj zi) Ry(-beta)
  const double2 b = cmulc(M[1], zi);
  w00 = csub(cscale(M[0], c), cscale(b, sn));
  w01 = cadd(cscale(M[0], sn), cscale(b, c));
  const double k = fma(-0.5, cnorm2(w00) + cnorm2(w01), 1.5);
  w00 = cscale(w00, k);
  w01 = cscale(w01, k);
  r.turn = 0;
  r.zi = zi;
}

// U3 = diag(1, phi) Ry(s, c) diag(1, lam), all three given as (cos, sin), times a phase: the
// numbers of its operation read off without forming the matrix (fewer roundings than split_zyz).
// Returns the sign that the rotation's scale leaves.
__device__ __forceinline__ double split_u3(double2 cs, double2 phi, double2 lam, RotRec& r) {
  const bool turn = fabs(cs.y) > fabs(cs.x);
  // Ry(theta) = Ry(theta - pi/2) after the quarter turn
  const double c = turn ? cs.y : cs.x, s = turn ? -cs.x : cs.y;
  r.turn = turn;
  r.t = s / c;
  set_cosine(r);
  r.zi = turn ? make_double2(-lam.x, -lam.y) : lam;
  r.zo = phi;
  return c < 0.0 ? -1.0 : 1.0;
}

// The numbers of all operations of the runs of one CTA, for one parameter vector: thread i
// makes the matrix of run i (the factors of a lone U3); the first thread of each chain of pushed
// rotations then walks it.  phase_out receives the product of the runs' phases.
__device__ __forceinline__ void rot_plan_body(const RotPlan& pl, int cta, const double* theta, RotRec* recs,
                                              double2* phase_out) {
  __shared__ double2 Ms[kRotThreads][4];
  __shared__ double2 ph[kRotThreads];
  const int base = pl.cta[cta], n = pl.cta[cta + 1] - base, i = threadIdx.x;
  const double2 one = make_double2(1.0, 0.0), zero = make_double2(0.0, 0.0);
  RotRun run;
  double2 phase = one;
  if (i < n) {
    run = pl.runs[base + i];
    double2 M[4];
    Gate g = pl.gates[pl.members[run.first]];
    if (run.lone_u3) {
      double s, c;
      for (int k = 0; k < 3; k++) {
        sincos(theta[g.pstart + k], &s, &c);
        M[k] = make_double2(c, s);
      }
      M[3] = zero;
    } else {
      gate_matrix(g.type, theta + g.pstart, M);
      for (int k = 1; k < run.count; k++) {
        double2 G[4];
        g = pl.gates[pl.members[run.first + k]];
        gate_matrix(g.type, theta + g.pstart, G);
        matmul2(G, M);
      }
    }
    for (int k = 0; k < 4; k++) Ms[i][k] = M[k];
  }
  __syncthreads();
  if (i < n && !run.pulled) {
    // the rotation pushed into the next run: diag(1, pz) times a phase (zpend), or a matrix
    bool zpend = true;
    double2 pz = one, pphase = one, pend[4];
    int j = i;
    for (int step = 0; step < kRotChain; step++, j++) {
      if (step) run = pl.runs[base + j];
      RotRec r = {0.0, 1.0, one, one, 0.0, 0};
      double2 M[4];
      for (int k = 0; k < 4; k++) M[k] = Ms[j][k];
      if (run.kind == kOpCry) {
        r.t = M[2].x;
        r.c = M[0].x;
      } else if (run.kind == kOpPhase) {  // diagonal
        r.zi = cunit(cmulc(M[3], M[0]));
        phase = M[0];
      } else if (!(run.kind & kOpZi)) {  // Ry or Rx by itself: M[0] = cos, M[2] = sin or -i sin
        const double2 cs = make_double2(M[0].x, (run.kind & kOpX) ? -M[2].y : M[2].x);
        const double sign = split_u3(cs, one, one, r);
        r.zi = one;
        // about X the quarter turn is -i times the exchange
        phase = r.turn && (run.kind & kOpX) ? make_double2(0.0, -sign) : make_double2(sign, 0.0);
      } else if (run.lone_u3 && zpend && (run.push == kAxisNone || run.push == kAxisZ)) {
        const double2 lam = step ? cunit(cmul(M[2], pz)) : M[2];
        pphase = cscale(pphase, split_u3(M[0], M[1], lam, r));
        if (run.push == kAxisNone)
          phase = pphase;
        else
          pz = M[1];
      } else {
        double2 A[4];
        if (run.lone_u3) {
          const double2 cs = M[0], pl2 = cmul(M[1], M[2]);
          A[0] = make_double2(cs.x, 0.0);
          A[1] = cscale(M[2], -cs.y);
          A[2] = cscale(M[1], cs.y);
          A[3] = cscale(pl2, cs.x);
        } else {
          for (int k = 0; k < 4; k++) A[k] = M[k];
        }
        if (zpend) {
          A[1] = cmul(A[1], pz);
          A[3] = cmul(A[3], pz);
          for (int k = 0; k < 4; k++) A[k] = cmul(A[k], pphase);
        } else {
          for (int k = 0; k < 4; k++) M[k] = A[k];
          for (int k = 0; k < 4; k++) A[k] = pend[k];
          matmul2(M, A);
        }
        if (run.push == kAxisNone) {
          phase = split_zyz(A, r);
        } else if (run.push == kAxisZ) {
          pphase = cunit(split_zyz(A, r));
          pz = r.zo;
          zpend = true;
        } else {
          // Y: with S = diag(1, i), S A S^dagger = Rx(-alpha) Ry(beta) diag(1, zi)
          if (run.push == kAxisY) {
            A[1] = make_double2(A[1].y, -A[1].x);
            A[2] = make_double2(-A[2].y, A[2].x);
          }
          double2 w0, w1;
          split_x(A, r, w0, w1);
          zpend = false;
          pend[0] = pend[3] = w0;
          pend[1] = pend[2] = w1;
          const double c2 = cnorm2(w0) - cnorm2(w1);
          double s2 = -2.0 * fma(w0.x, w1.y, -w0.y * w1.x);  // sin of the full angle: -2 Im(conj(w0) w1)
          if (run.push == kAxisY) {
            pend[1] = make_double2(-w1.y, w1.x);
            pend[2] = make_double2(w1.y, -w1.x);
            s2 = -s2;
          }
          r.zo = make_double2(c2, s2);
        }
      }
      recs[run.op] = r;
      if (run.push == kAxisNone) break;
    }
  }
  ph[i] = phase;
  __syncthreads();
  for (int o = kRotThreads / 2; o > 0; o >>= 1) {
    if (i < o) ph[i] = cmul(ph[i], ph[i + o]);
    __syncthreads();
  }
  if (i == 0) *phase_out = ph[0];
}

// ---- application ---------------------------------------------------------------------------
// Operation staged for the sweeps.  Negated copies of its numbers (nt, nzi, nzo) are staged with
// them: the sweeps would otherwise negate them once per thread, on the FP64 pipe.  scale: of the
// operation that multiplies the chunk's cosines back in (kStRescale; t and nt include it), the
// cosine of a kOpCry.  mfac: what the overlaps measured behind the operation, with both vectors
// on the way back, are multiplied by.
struct StagedOp {
  int kind, qubits, coff, mask;  // qubits: target | control << 8 | flags << 16
  double t, nt, scale, mfac;
  double2 zi, zo;
  double nzi, nzo;
};
enum : int { kStTurn = 1 << 16, kStRescale = 1 << 17 };

// Loads operations [k0, k0 + kn) (at most kRotChunk) into st with the first warp of the CTA.
// The cosines that the chunk's rotations leave out are multiplied back in its last rotation.
// The caller synchronises before and after.
__device__ __forceinline__ void stage_ops(StagedOp* st, const RotOp* ops, const RotRec* recs, int k0, int kn) {
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  const bool on = lane < kn;
  RotOp op = {kOpCnot, 0, 0, 0};
  RotRec r = {0.0, 1.0, make_double2(1.0, 0.0), make_double2(1.0, 0.0), 0.0, 0};
  if (on) {
    op = ops[k0 + lane];
    if (op.kind >= kOpCry) r = recs[k0 + lane];
  }
  const bool rot = (op.kind & kOpRot) != 0;
  // product of the cosines up to and including this operation, as pre + plo
  double pre = rot ? r.c : 1.0, plo = rot ? r.lo : 0.0;
  for (int o = 1; o < 32; o <<= 1) {
    const double v = __shfl_up_sync(0xffffffffu, pre, o), vlo = __shfl_up_sync(0xffffffffu, plo, o);
    if (lane >= o) {
      const double p = pre * v;
      plo = fma(pre, v, -p) + fma(pre, vlo, plo * v);
      pre = p;
    }
  }
  const double all = __shfl_sync(0xffffffffu, pre + plo, 31);
  const unsigned rots = __ballot_sync(0xffffffffu, rot);
  const int last = rots ? 31 - __clz(rots) : -1;
  if (on) {
    StagedOp s;
    s.kind = op.kind;
    s.qubits = op.qubits | (r.turn ? kStTurn : 0) | (lane == last ? kStRescale : 0);
    s.coff = op.coff;
    s.mask = op.mask;
    s.scale = lane == last ? all : op.kind == kOpCry ? r.c : 1.0;
    s.t = lane == last ? r.t * all : r.t;
    s.nt = dneg(s.t);
    const double inv = 1.0 / pre;
    s.mfac = lane < last ? inv * inv : 1.0;
    s.zi = r.zi;
    s.zo = r.zo;
    s.nzi = dneg(r.zi.y);
    s.nzo = dneg(r.zo.y);
    st[lane] = s;
  }
}

enum { kRotFwd = 0, kRotAdj = 1, kRotTrans = 2 };  // G, G^dagger, G^T (right multiplication)

// The numbers of a staged operation in a direction: G^dagger takes -t and the conjugate phases,
// G^T takes -t about Y (Rx^T = Rx).
struct DirOp {
  double t, nt, scale;
  double zix, ziy, nzi, zox, zoy, nzo;
  unsigned flip;  // sign bit for a turned Ry without a zi that could hold its sign
  bool turn;
};

template <int DIR, int KIND>
__device__ __forceinline__ DirOp directed(const StagedOp& s) {
  DirOp o;
  const bool neg = DIR == kRotAdj || (DIR == kRotTrans && !(KIND & kOpX));
  o.t = neg ? s.nt : s.t;
  o.nt = neg ? s.t : s.nt;
  o.scale = s.scale;
  o.zix = s.zi.x;
  o.ziy = DIR == kRotAdj ? s.nzi : s.zi.y;
  o.nzi = DIR == kRotAdj ? s.zi.y : s.nzi;
  o.zox = s.zo.x;
  o.zoy = DIR == kRotAdj ? s.nzo : s.zo.y;
  o.nzo = DIR == kRotAdj ? s.zo.y : s.nzo;
  o.turn = (s.qubits & kStTurn) != 0;
  o.flip = o.turn ? 0x80000000u : 0u;
  return o;
}

// v with the sign bit `flip` changed (an integer operation).
__device__ __forceinline__ double flip_sign(double v, unsigned flip) {
  return __hiloint2double(__double2hiint(v) ^ (int)flip, __double2loint(v));
}

// y <- z y, nzy = -z.y
__device__ __forceinline__ void rot_phase(double2& y, double zx, double zy, double nzy) {
  const double re = fma(zx, y.x, nzy * y.y);
  y.y = fma(zx, y.y, zy * y.x);
  y.x = re;
}

// (x, y) <- [[1, nt], [t, 1]] (x, y), about Y, or (AX) the same about X: [[1, -i t], [-i t, 1]].
// RS: the ones are `scale`.
template <bool AX, bool RS>
__device__ __forceinline__ void rot_turnless(double2& x, double2& y, double t, double nt, double scale) {
  double2 nx, ny;
  if (!RS) {
    if (!AX) {
      nx.x = fma(nt, y.x, x.x);
      nx.y = fma(nt, y.y, x.y);
      ny.x = fma(t, x.x, y.x);
      ny.y = fma(t, x.y, y.y);
    } else {
      nx.x = fma(t, y.y, x.x);
      nx.y = fma(nt, y.x, x.y);
      ny.x = fma(t, x.y, y.x);
      ny.y = fma(nt, x.x, y.y);
    }
  } else {
    if (!AX) {
      nx.x = fma(scale, x.x, nt * y.x);
      nx.y = fma(scale, x.y, nt * y.y);
      ny.x = fma(t, x.x, scale * y.x);
      ny.y = fma(t, x.y, scale * y.y);
    } else {
      nx.x = fma(scale, x.x, t * y.y);
      nx.y = fma(scale, x.y, nt * y.x);
      ny.x = fma(scale, y.x, t * x.y);
      ny.y = fma(scale, y.y, nt * x.x);
    }
  }
  x = nx;
  y = ny;
}

// One kOpRot operation on a pair.  kRotAdj / kRotTrans walk its factors backwards.  The form of
// the operation is a template parameter, chosen once per operation and not per pair: a
// predicated FP64 instruction takes the pipe as long as an executed one.
template <int DIR, int KIND, bool RS>
__device__ __forceinline__ void rot_pair(const DirOp& op, double2& x, double2& y) {
  constexpr bool AX = KIND & kOpX, ZI = KIND & kOpZi, ZO = KIND & kOpZo;
  if (DIR == kRotFwd) {
    if (ZI) rot_phase(y, op.zix, op.ziy, op.nzi);
    if (!ZI && !AX) y = make_double2(flip_sign(y.x, op.flip), flip_sign(y.y, op.flip));
    const double2 a = op.turn ? y : x, b = op.turn ? x : y;
    x = a;
    y = b;
    rot_turnless<AX, RS>(x, y, op.t, op.nt, op.scale);
    if (ZO) rot_phase(y, op.zox, op.zoy, op.nzo);
  } else {
    if (ZO) rot_phase(y, op.zox, op.zoy, op.nzo);
    rot_turnless<AX, RS>(x, y, op.t, op.nt, op.scale);
    const double2 a = op.turn ? y : x, b = op.turn ? x : y;
    x = a;
    y = b;
    if (!ZI && !AX) y = make_double2(flip_sign(y.x, op.flip), flip_sign(y.y, op.flip));
    if (ZI) rot_phase(y, op.zix, op.ziy, op.nzi);
  }
}

// Controlled Ry on a pair with its control bit set: [[c, ns], [s, c]].
__device__ __forceinline__ void cry_pair(const DirOp& op, double2& x, double2& y) {
  double2 nx, ny;
  nx.x = fma(op.scale, x.x, op.nt * y.x);
  nx.y = fma(op.scale, x.y, op.nt * y.y);
  ny.x = fma(op.t, x.x, op.scale * y.x);
  ny.y = fma(op.t, x.y, op.scale * y.y);
  x = nx;
  y = ny;
}

// Applies one staged operation to every vector of a tile: tc vectors of length N = 2^logN, one
// after another in s.  All threads of the CTA.
template <int DIR, int KIND, bool RS>
__device__ __forceinline__ void rot_tile_kind(double2* s, int N, int logN, int tc, const StagedOp& staged) {
  const DirOp op = directed<DIR, KIND>(staged);
  const int target = staged.qubits & 255, control = (staged.qubits >> 8) & 255;
  constexpr bool ctrl = KIND <= kOpCry;
  const int lognp = ctrl ? logN - 2 : logN - 1;
  const int npairs = 1 << lognp;
  const int items = tc << lognp;
  const int step = 1 << target;
  for (int it = threadIdx.x; it < items; it += blockDim.x) {
    const int col = it >> lognp;
    const int p = it & (npairs - 1);
    const int i = ctrl ? pair_index2(p, target, control) : pair_index1(p, target);
    double2* v = s + col * N;
    if (KIND == kOpPhase || KIND == kOpCz) {  // the target = 0 row is not touched
      double2 y = v[i + step];
      if (KIND == kOpCz)
        y = make_double2(dneg(y.x), dneg(y.y));
      else
        rot_phase(y, op.zix, op.ziy, op.nzi);
      v[i + step] = y;
      continue;
    }
    double2 x = v[i], y = v[i + step];
    if (KIND == kOpCnot) {
      const double2 o = x;
      x = y;
      y = o;
    } else if (KIND == kOpCry) {
      cry_pair(op, x, y);
    } else {
      rot_pair<DIR, KIND, RS>(op, x, y);
    }
    v[i] = x;
    v[i + step] = y;
  }
}

template <int DIR>
__device__ __forceinline__ void rot_tile(double2* s, int N, int logN, int tc, const StagedOp& st) {
#define SQG_ROT_CASE(KIND) \
  case (KIND): \
    if (st.qubits & kStRescale) \
      rot_tile_kind<DIR, (KIND), true>(s, N, logN, tc, st); \
    else \
      rot_tile_kind<DIR, (KIND), false>(s, N, logN, tc, st); \
    break;
  switch (st.kind) {
    case kOpCnot: rot_tile_kind<DIR, kOpCnot, false>(s, N, logN, tc, st); break;
    case kOpCz: rot_tile_kind<DIR, kOpCz, false>(s, N, logN, tc, st); break;
    case kOpCry: rot_tile_kind<DIR, kOpCry, false>(s, N, logN, tc, st); break;
    case kOpPhase: rot_tile_kind<DIR, kOpPhase, false>(s, N, logN, tc, st); break;
    SQG_ROT_CASE(kOpRot)
    SQG_ROT_CASE(kOpRot | kOpX)
    SQG_ROT_CASE(kOpRot | kOpZi)
    SQG_ROT_CASE(kOpRot | kOpX | kOpZi)
    SQG_ROT_CASE(kOpRot | kOpZi | kOpZo)
  }
#undef SQG_ROT_CASE
}

}  // namespace sqg
