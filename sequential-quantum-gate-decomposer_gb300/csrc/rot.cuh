// Rotation plan of a circuit: the form in which the tile and state kernels apply it.
//
// What bounds these kernels is the number of products per amplitude pair: FP64 instructions where
// amplitudes go back to the caller (the FP64 pipe takes two lanes per clock and SM; every other pipe is
// nearly idle), fixed-point products (fx.cuh) for cost and gradient.  The plan rewrites the gate list into
// operations with as few of them as the circuit allows:
//  * A run of single-qubit gates on one qubit, with no two-qubit gate on that qubit between
//    them, is one 2x2 unitary M.
//  * M = scalar * diag(1, zo) * R * diag(1, zi) with R a rotation.  R is applied without its
//    cosine ([[1, -t], [t, 1]], |t| <= 1 after an exchange of the two rows where needed):
//    4 multiply-adds per pair instead of 8.  The cosines of a group of consecutive operations are
//    multiplied in with the first of them, so the scale never exceeds 1.
//    A phase diag(1, z) touches one row of the pair: 4 instructions.
//  * The rotation that M ends with is moved through the next two-qubit gate into the next run
//    on the qubit where it commutes with that gate: Z through a control or a CZ, X through a
//    CNOT target, Y through a CRY target.  What is left of M is R * diag(1, zi): 8
//    instructions per pair, against 14 of a U3 as given.
//  * Phases common to all amplitudes are collected per instance and multiplied in once.
//  * The gradient needs only <lambda| P |psi> for the Paulis P at the end of each run; the one
//    along the axis that the run pushes equals that of the next run and is not measured, and
//    the derivatives of the run's gates follow from these three numbers, once per run
//    (rot_grad_body) and not per amplitude.
// Measured on GB300 in FP64 against the gates as given (U3 14 instructions, merged runs 16): 2000 random gates
// on a 4096 x 4096 matrix 143 -> 98 ms; 829 gates on 24 qubits 128 -> 87 ms, the FP64 pipe 92 % busy either way;
// gradient at 8 qubits, 360 blocks, 128 vectors 333 -> 182 ms, and 77 ms with the sweeps in fixed point.
// Error against long double, random circuits of 6 to 16 qubits and 200 to 2000 gates, as a multiple of that of
// the gates as given: 0.94 in the mean at uniform angles (0.6 to 1.5), 0.6 and 0.7 at multiples of pi/4.
// The numbers behind each operation depend on the parameters and are made per instance by
// rot_plan_body; which operations there are depends on the gate list alone (build_rot_plan).
#pragma once
#include "gates.cuh"

namespace sqg {

// Kinds of operations.  kOpRot carries flags: rotation about X instead of Y, phase before
// (zi), phase after (zo).
enum : int { kOpCnot = 0, kOpCz = 1, kOpCry = 2, kOpPhase = 3, kOpRot = 4, kOpX = 8, kOpZi = 16, kOpZo = 32 };
enum : int { kAxisNone = 0, kAxisX = 1, kAxisY = 2, kAxisZ = 3 };

// One operation of the plan as the sweeps apply it to 2^n amplitudes.  A CNOT moves no data: it
// only changes which amplitude a place holds.  Place p holds the amplitude whose bit q is the
// parity of p & row_q, and its partner under qubit q is p ^ pair_q; the plan follows these masks
// through the CNOTs.  A CZ flips signs where two parities are odd; it rides on the next
// operation that does not commute with it (cz0, cz1; none: 0) or is one of its own (kOpCz).
// coff: first of the operation's overlaps in the instance's overlap list; mask: which are
// measured (1 X, 2 Y, 4 Z; kOpCry: 2, on the controlled half).
struct RotOp {
  int kind;
  int rec;  // of its numbers
  int coff;
  int mask;
  unsigned short pair, row, crow;  // the target's pair and row, a CRY control's row
  unsigned short cz0, cz1;
  unsigned short b0, b1;  // bits that number the pairs: set in pair; kOpCry: in crow, not b0
  unsigned short pad;
};

// One run (or CRY gate): its record, its gates members[first .. first + count), the axis it
// pushes (kAxisNone: nothing) into the run right behind it in the chain order, whether the run
// before it pushes into it, a copy of its operation's kind, coff and mask, and whether it is a
// single U3 with no other than Z rotations pushed into it and by it.  soff: place of its first parameter in its CTA's parameter list, the parameters of its
// gates behind one another (-1: not listed).
struct RotRun {
  int rec, first, count, push, pulled, kind, coff, mask, lone_u3, soff;
};

// Numbers of one operation.  t, c: tangent and cosine of the rotation (kOpCry: sine and
// cosine, lo: what c lacks to the exact cosine of t); turn: the two rows are exchanged between
// zi and the rotation (a quarter turn about Y with its sign in zi, about X up to a phase).  zo of
// a run that pushes holds (cos, sin) of the pushed rotation's full angle.
struct RotRec {
  double t, c;
  double2 zi, zo;
  double lo;
  double turn;  // 0 or 1 (all members are doubles: batch_matrices_body keeps matrices here)
};
static_assert(sizeof(RotRec) == sizeof(GateMat), "the workspace counts both as 64 bytes");

// Device view of a circuit's plan.
struct RotPlan {
  const Gate* gates;
  const RotOp* ops;
  const RotRun* runs;
  const int* members;
  const int* cta;  // runs [cta[i], cta[i + 1]) are handled by one CTA of kRotThreads threads
  const int* params;  // parameters of CTA i's runs: params[cta_params[i] .. cta_params[i + 1])
  const int* cta_params;
  const int* heads;  // first runs of the chains, those of two and more runs first
  const int* ends;  // place of the amplitude 2^q behind the last operation (a sum of them: their XOR)
  int nops, nrecs, ncta, noverlaps, nheads;
};

constexpr int kRotThreads = 128;  // runs per CTA of the per-instance kernels; no chain straddles two
constexpr int kRotParams = 512;  // parameters listed per CTA
// Runs linked by pushed rotations.  Their numbers are made one after another, half a microsecond a run, and
// the run that ends a chain costs 4 products more per pair and vector: 3 % at 16, 12 % at 4.  A launch
// that does not fill the device waits for the chains: 46 U3 of one vector 36 us at 16, 30 us at 4.
constexpr int kRotChain = 16, kRotShortChain = 4;
constexpr int kRotChunk = 32;     // operations staged in shared memory together (a warp)
// The cosines of a group of consecutive operations are multiplied in together.  In FP64 the scale costs no
// precision: the whole chunk is a group.  In fixed point it costs amplitudes its size and overlaps its
// square, so a group ends before the cosines of all but its last rotation pass 2^-1.5: after three
// operations at angles of pi/4, ten at uniform ones.  Error of gradients against long double over 6 to 12
// qubits, 1 to 256 columns, angles uniform and at or near multiples of pi/4, as a multiple of that of the gates
// as given in FP64: 0.7 to 1.1 in the mean, 3 at worst; groups of 16 operations whatever their cosines
// 1.0 to 6.4, 2800 at worst.  Bounds of 2^-1, 2^-2: gradients at four qubits, 1024 vectors 5 % slower, 3 % faster;
// single columns of 4096 rows at uniform angles 1.4, 3.7 times the error of FP64 at worst (2^-1.5: 1.7).
constexpr int kFxGroupBits = (3 << 20) / 2;  // 1.5, in units of 2^-20

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cmulc(double2 a, double2 b) {  // a * conj(b)
  return make_double2(fma(a.x, b.x, a.y * b.y), fma(a.y, b.x, -a.x * b.y));
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 cscale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double cnorm2(double2 a) { return fma(a.x, a.x, a.y * a.y); }
// 1 / sqrt(x) and 1 / x for x in [2^-120, 2^120], to 1.5 and 1 times 2^-53 (relative): from the
// device's approximation of some 20 bits by two Newton steps.  The chains of rot_plan_body wait for every one of their
// instructions, and the general functions take several times as many.
__device__ __forceinline__ double fast_rsqrt(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double h = -0.5 * x;
  y = fma(y, fma(h * y, y, 0.5), y);
  return fma(y, fma(h * y, y, 0.5), y);
}
__device__ __forceinline__ double fast_rcp(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}
// One Newton step towards |z| = 1 for z that is a few roundings away from it, as z + e z: a factor
// 1 + e would be rounded, more coarsely above 1 than below, and hundreds of runs would shrink.
__device__ __forceinline__ double2 cgrow(double2 z, double e) { return make_double2(fma(z.x, e, z.x), fma(z.y, e, z.y)); }
__device__ __forceinline__ double2 cunit(double2 z) { return cgrow(z, -0.5 * fma(z.x, z.x, fma(z.y, z.y, -1.0))); }

// ---- numbers of the chains: 64-bit fixed point --------------------------------------------------
// The entries of unitaries, in units of 2^-62.  What a chain hands from run to run passes some
// twenty products, whose roundings in FP64 would be as large as those of all amplitudes: with the chains
// in FP64 the error of circuits of U3 and CNOT was 1.1 to 1.6 times that of the gates as given.  Here a product
// is good to 2^-60 and answers in a tenth of the time.
struct Q2 {
  long long x, y;
};
constexpr long long kQOne = 1LL << 62;
__device__ __forceinline__ long long q_of(double v) { return __double2ll_rn(v * 0x1p62); }
__device__ __forceinline__ Q2 q_of(double2 v) { return {q_of(v.x), q_of(v.y)}; }
__device__ __forceinline__ double q_to(long long v) { return (double)v * 0x1p-62; }
__device__ __forceinline__ double2 q_to(Q2 v) { return make_double2(q_to(v.x), q_to(v.y)); }
// Four units of the sum are those of the upper words; half of what their floors drop is put back.
__device__ __forceinline__ long long q_mul(long long a, long long b) { return __mul64hi(a, b) * 4 + 2; }
__device__ __forceinline__ long long q_sum(long long a, long long b, long long c, long long d) {  // a b + c d
  return (__mul64hi(a, b) + __mul64hi(c, d)) * 4 + 4;
}
__device__ __forceinline__ long long q_diff(long long a, long long b, long long c, long long d) {  // a b - c d
  return (__mul64hi(a, b) - __mul64hi(c, d)) * 4;
}
__device__ __forceinline__ Q2 q_mul(Q2 a, Q2 b) { return {q_diff(a.x, b.x, a.y, b.y), q_sum(a.x, b.y, a.y, b.x)}; }
__device__ __forceinline__ Q2 q_mulc(Q2 a, Q2 b) {  // a * conj(b)
  return {q_sum(a.x, b.x, a.y, b.y), q_diff(a.y, b.x, a.x, b.y)};
}
__device__ __forceinline__ Q2 q_scale(Q2 a, long long s) { return {q_mul(a.x, s), q_mul(a.y, s)}; }
__device__ __forceinline__ Q2 q_add(Q2 a, Q2 b) { return {a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ Q2 q_sub(Q2 a, Q2 b) { return {a.x - b.x, a.y - b.y}; }

// (cos, sin) of every listed parameter of a CTA's runs, one per thread: a warp's FP64 instruction
// costs the same for one lane as for 32.  sc: kRotParams entries of shared memory; the caller
// synchronises.
__device__ __forceinline__ void cta_sincos(const RotPlan& pl, int cta, const double* theta, double2* sc) {
  const int first = pl.cta_params[cta], n = pl.cta_params[cta + 1] - first;
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    double s, c;
    sincos(theta[pl.params[first + k]], &s, &c);
    sc[k] = make_double2(c, s);
  }
}
// (cos, sin) of parameter k of a gate whose listed ones start at soff.
__device__ __forceinline__ double2 param_sincos(const double2* sc, int soff, const double* th, int k) {
  if (soff >= 0) return sc[soff + k];
  double s, c;
  sincos(th[k], &s, &c);
  return make_double2(c, s);
}

// Full 2x2 matrix of a gate of one parameter, given as (cos, sin).
__device__ __forceinline__ void gate_matrix(int type, double2 a, double2 u[4]) {
  const double c = a.x, s = a.y;
  if (type == G_RX) {
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
  r.c = fast_rsqrt(s);
  const double c2 = r.c * r.c, c2e = fma(r.c, r.c, -c2);
  const double p = c2 * s, pe = fma(c2, s, -p) + fma(c2e, s, c2 * se);
  r.lo = 0.5 * r.c * ((1.0 - p) - pe);
}

// A unitary with first column (p, q) and determinant det as scalar * diag(1, zo) * R * [exchange] * diag(1,
// zi); returns the scalar's phase.  The larger entry of the first column is the pivot, so |t| <= 1.
__device__ __forceinline__ double2 split_zyz(Q2 p, Q2 q, Q2 det, RotRec& r) {
  const double2 pd = q_to(p), qd = q_to(q);
  const double na = cnorm2(pd), nc = cnorm2(qd);
  const bool turn = nc > na;
  const Q2 piv = turn ? q : p;
  const double np = turn ? nc : na;
  // other entry / pivot: f = 0: t zo, f = 1: -t / zo
  const double2 x = q_to(q_mulc(turn ? p : q, piv));
  const double x2 = cnorm2(x);
  // t below 1e-17 is an entry lost in the rounding of the others: any phase does
  const double rx = x2 > 1e-34 ? fast_rsqrt(x2) : 0.0;
  const double inv = fast_rcp(np), t = x2 * rx;
  r.t = fma(fma(-t * inv, np, t), inv, t * inv);
  double2 zo = make_double2(1.0, 0.0);
  if (x2 > 1e-34) zo = cscale(turn ? make_double2(-x.x, x.y) : x, rx);
  zo = cunit(zo);
  // the second column is (-conj q, conj p) det: its entry beside the pivot, over the pivot (f = 0: d / a, f
  // = 1: b / c), is det conj(piv)^2 / np, negated for f = 1, where zi has another minus: zi = it / zo, or times zo
  const Q2 w = q_mulc(q_mulc(det, piv), piv), zq = q_of(zo);
  const double2 z = q_to(turn ? q_mul(w, zq) : q_mulc(w, zq));
  const double2 zi = cunit(cscale(z, inv));  // |z| = |piv|^2
  r.turn = turn;
  // the quarter turn (x, y) -> (-y, x) as an exchange: its sign goes into zi
  r.zi = turn ? make_double2(-zi.x, -zi.y) : zi;
  r.zo = zo;
  const Q2 u = turn ? q_mulc(piv, zq) : piv;
  return cunit(cscale(q_to(u), fast_rsqrt(np)));
}

// A unitary with first column (p, q) and determinant det as W * Ry(atan t) * diag(1, zi) with W =
// phase * Rx = [[w0, w1], [w1, w0]].  |t| <= 1 always.  The cosine is left to set_cosine.  On
// return p, q, det are those of W, made with t and zi as the record holds them: their roundings go no
// further.
__device__ __forceinline__ void split_x(Q2& p, Q2& q, Q2& det, RotRec& r) {
  // (p^2 - q^2) / det = e^{-2 i gamma} cos 2 beta, with zi = e^{2 i gamma}
  const double2 d = q_to(q_mulc(q_mul(q_add(p, q), q_sub(p, q)), det));
  const double nd2 = cnorm2(d), rnd = nd2 > 1e-34 ? fast_rsqrt(nd2) : 0.0;
  r.zi = nd2 > 1e-34 ? cunit(make_double2(d.x * rnd, -d.y * rnd)) : make_double2(1.0, 0.0);
  // tan beta = sin 2 beta / (1 + cos 2 beta), cos^2 beta = (1 + cos 2 beta) / 2
  const double sb2 = 2.0 * q_to(q_sum(p.x, q.x, p.y, q.y)), den = fma(nd2, rnd, 1.0), root = fast_rsqrt(2.0 * den);
  const double inv = 2.0 * root * root, t0 = sb2 * inv;
  r.t = fma(fma(-t0, den, sb2), inv, t0);
  r.turn = 0;
  // the cosine of t as rounded: one Newton step in units from the double
  const long long t = q_of(r.t), c0 = q_of(den * root);
  const long long c2 = q_mul(c0, c0), e = kQOne - c2 - q_mul(c2, q_mul(t, t));
  const long long c = c0 + q_mul(c0, e) / 2, sn = q_mul(t, c);
  // W = A diag(1, conj zi) Ry(-beta); the second column of A is (-conj q, conj p) det
  det = q_mulc(det, q_of(r.zi));
  det = q_add(det, q_scale(det, (kQOne - q_sum(det.x, det.x, det.y, det.y)) / 2));  // zi is a unit to 2^-53
  const Q2 b = q_mulc(det, q);  // minus the upper entry of A diag(1, conj zi)
  const Q2 w0 = {q_sum(c, p.x, sn, b.x), q_sum(c, p.y, sn, b.y)};
  q = {q_diff(sn, p.x, c, b.x), q_diff(sn, p.y, c, b.y)};
  p = w0;
}

// U3 = diag(1, phi) Ry(s, c) diag(1, lam), all three given as (cos, sin), times a phase: the
// numbers of its operation read off without forming the matrix (fewer roundings than split_zyz).
// Returns the sign that the rotation's scale leaves.
__device__ __forceinline__ double split_u3(double2 cs, double2 phi, double2 lam, RotRec& r) {
  const bool turn = fabs(cs.y) > fabs(cs.x);
  // Ry(theta) = Ry(theta - pi/2) after the quarter turn
  const double c = turn ? cs.y : cs.x, s = turn ? -cs.x : cs.y;
  r.turn = turn;
  const double rc = fast_rcp(c), t = s * rc;
  r.t = fma(fma(-t, c, s), rc, t);
  r.zi = turn ? make_double2(-lam.x, -lam.y) : lam;
  r.zo = phi;
  return c < 0.0 ? -1.0 : 1.0;
}

// M <- G M in units with G = diag(f0, f1) Ry diag(1, l), a form that every gate has: U3 by its angles, RX =
// diag(1, -i) Ry diag(1, i), RZ = diag(c - i s, c + i s).  One form for all, so that the threads of a warp, each
// with its own gates, stay together.
__device__ __forceinline__ void q_gate(int type, double2 a, double2 phi, double2 lambda, Q2 M[4]) {
  const Q2 one = {kQOne, 0}, cs = q_of(a);
  const bool u3 = type == G_U3, rx = type == G_RX, rz = type == G_RZ;
  const long long c = rz ? kQOne : cs.x, s = rz ? 0 : cs.y;
  const Q2 l = u3 ? q_of(lambda) : rx ? Q2{0, kQOne} : one;
  const Q2 f0 = rz ? Q2{cs.x, -cs.y} : one, f1 = u3 ? q_of(phi) : rx ? Q2{0, -kQOne} : rz ? cs : one;
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const Q2 x = M[j], y = q_mul(l, M[2 + j]);
    M[j] = q_mul(f0, Q2{q_diff(c, x.x, s, y.x), q_diff(c, x.y, s, y.y)});
    M[2 + j] = q_mul(f1, Q2{q_sum(s, x.x, c, y.x), q_sum(s, x.y, c, y.y)});
  }
}

// Matrix of a run from its CTA's parameters: of a lone U3 (cos, sin) of its three angles; of a rotation by
// itself its entries; else entries in units (Q2), kQBad for the first where an angle is not finite.
constexpr long long kQBad = (long long)0x8000000000000000ULL;
__device__ __forceinline__ bool run_in_units(const RotRun& run) {
  return run.count > 1 || ((run.kind & kOpRot) && (run.kind & kOpZi) && !run.lone_u3);
}
__device__ __forceinline__ double2 q_bits(Q2 v) { return make_double2(__longlong_as_double(v.x), __longlong_as_double(v.y)); }
__device__ __forceinline__ Q2 q_of_bits(double2 v) { return {__double_as_longlong(v.x), __double_as_longlong(v.y)}; }

__device__ __forceinline__ void run_matrix(const RotPlan& pl, const RotRun& run, const double2* sc,
                                           const double* theta, double2 M[4]) {
  const double2 one = make_double2(1.0, 0.0);
  Gate g = pl.gates[pl.members[run.first]];
  int soff = run.soff;
  if (run.lone_u3) {
    for (int k = 0; k < 3; k++) M[k] = param_sincos(sc, soff, theta + g.pstart, k);
    M[3] = one;
    return;
  }
  if (!run_in_units(run)) {
    gate_matrix(g.type, param_sincos(sc, soff, theta + g.pstart, 0), M);
    return;
  }
  Q2 P[4] = {{kQOne, 0}, {0, 0}, {0, 0}, {kQOne, 0}};
  bool finite = true;
  for (int k = 0; k < run.count; k++) {
    if (k > 0) {
      if (soff >= 0) soff += gate_param_num(g.type);
      g = pl.gates[pl.members[run.first + k]];
    }
    const double* th = theta + g.pstart;
    const double2 a = param_sincos(sc, soff, th, 0);
    double2 ph = one, la = one;
    if (g.type == G_U3) {
      ph = param_sincos(sc, soff, th, 1);
      la = param_sincos(sc, soff, th, 2);
    }
    finite = finite && isfinite(a.x) && isfinite(ph.x) && isfinite(la.x);
    q_gate(g.type, a, ph, la, P);
  }
  if (!finite) P[0].x = kQBad;
  for (int j = 0; j < 4; j++) M[j] = q_bits(P[j]);
}

// Walks the chain that starts with run `first` (a run by itself: a chain of one), mat(j, M)
// giving the matrix of run j: writes their records, but for the cosines of rotations.  Returns
// the phase that the chain leaves.
template <class Mat>
__device__ __forceinline__ double2 walk_chain(const RotPlan& pl, int first, RotRec* recs, Mat mat) {
  const double2 one = make_double2(1.0, 0.0);
  const double nan = __longlong_as_double(0x7ff8000000000000LL);
  // the rotation pushed into the next run: diag(1, pz) times pphase (zpend), or a unitary given
  // by its first column (wp, wq) and its determinant wdet
  bool zpend = true;
  double2 pz = one, pphase = one, own = one;
  Q2 wp = {kQOne, 0}, wq = {0, 0}, wdet = {kQOne, 0};
  bool finite = true;  // units hold no NaN: every record from the first that meets one on is marked
  for (int step = 0; step < kRotChain; step++) {
    const RotRun run = pl.runs[first + step];
    RotRec r = {0.0, 1.0, one, one, 0.0, 0.0};
    double2 M[4];
    mat(first + step, run, M);
    Q2 Q[4];
    const bool units = run_in_units(run);
    if (units) {
      for (int k = 0; k < 4; k++) Q[k] = q_of_bits(M[k]);
      finite = finite && Q[0].x != kQBad;
    }
    if (run.kind == kOpCry) {
      r.t = M[2].x;
      r.c = M[0].x;
    } else if (!(run.kind & kOpRot) || !(run.kind & kOpZi)) {  // gates about one axis
      if (units) M[0] = q_to(Q[0]), M[2] = q_to(Q[2]), M[3] = q_to(Q[3]);
      if (run.kind == kOpPhase) {  // diagonal
        r.zi = cunit(cmulc(M[3], M[0]));
        own = M[0];
      } else {  // Ry or Rx: M[0] = cos, M[2] = sin or -i sin
        const double2 cs = make_double2(M[0].x, (run.kind & kOpX) ? -M[2].y : M[2].x);
        const double sign = split_u3(cs, one, one, r);
        r.zi = one;
        // about X the quarter turn is -i times the exchange
        own = r.turn && (run.kind & kOpX) ? make_double2(0.0, -sign) : make_double2(sign, 0.0);
      }
    } else if (run.lone_u3) {  // nothing but a phase pulled, nothing but a phase pushed
      const double2 lam = step ? cunit(cmul(M[2], pz)) : M[2];
      pphase = cscale(pphase, split_u3(M[0], M[1], lam, r));
      if (run.push == kAxisNone)
        own = pphase;
      else
        pz = M[1];
    } else {
      // A = M * pushed, by its first column (p, q) and its determinant
      if (zpend) {
        finite = finite && isfinite(pphase.x) && isfinite(pz.x);
        wp = q_of(pphase);
        wq = {0, 0};
        wdet = q_mul(q_mul(wp, wp), q_of(pz));
      }
      Q2 p = q_add(q_mul(Q[0], wp), q_mul(Q[1], wq)), q = q_add(q_mul(Q[2], wp), q_mul(Q[3], wq));
      Q2 d = q_mul(q_sub(q_mul(Q[0], Q[3]), q_mul(Q[1], Q[2])), wdet);
      if (run.push == kAxisNone || run.push == kAxisZ) {
        const double2 ph = split_zyz(p, q, d, r);
        zpend = true;
        pphase = own = ph;
        pz = r.zo;
      } else {
        // Y: with S = diag(1, i), S A S^dagger = Rx(-alpha) Ry(beta) diag(1, zi)
        if (run.push == kAxisY) q = {-q.y, q.x};
        split_x(p, q, d, r);
        const double c2 = q_to(q_sum(p.x, p.x, p.y, p.y) - q_sum(q.x, q.x, q.y, q.y));
        const double s2 = -2.0 * q_to(q_diff(p.x, q.y, p.y, q.x));  // sin of the full angle: -2 Im(conj(w0) w1)
        zpend = false;
        wp = p;
        wq = run.push == kAxisY ? Q2{q.y, -q.x} : q;
        wdet = d;
        r.zo = make_double2(c2, run.push == kAxisY ? -s2 : s2);
      }
    }
    if (!finite) r.t = nan, r.zi = r.zo = make_double2(nan, nan);
    recs[run.rec] = r;
    if (run.push == kAxisNone) break;
  }
  return own;
}

// The cosines of a run's record.  Returns whether its numbers are all finite (an infinite angle, say, makes
// NaN of some).
__device__ __forceinline__ bool finish_record(const RotRun& run, RotRec& r) {
  RotRec v = r;
  if (run.kind & kOpRot) set_cosine(v);
  r.c = v.c;
  r.lo = v.lo;
  return isfinite(v.t + v.c + v.zi.x + v.zi.y + v.zo.x + v.zo.y);
}

// Product of the threads' phases (kRotThreads of them), written by thread 0; twice that if a record of the
// CTA's runs is not finite, which sweeps in fixed point need to know and amplitudes that do not meet
// that record must not notice (phase_factor).
__device__ __forceinline__ void phase_product(double2 phase, bool finite, double2* out) {
  __shared__ double2 ph[kRotThreads / 32];
  const int warp = threadIdx.x >> 5;
  for (int o = 16; o > 0; o >>= 1)
    phase = cmul(phase, make_double2(__shfl_xor_sync(0xffffffffu, phase.x, o), __shfl_xor_sync(0xffffffffu, phase.y, o)));
  if ((threadIdx.x & 31) == 0) ph[warp] = phase;
  finite = __syncthreads_and(finite);
  if (threadIdx.x > 0) return;
  phase = cmul(cmul(ph[0], ph[1]), cmul(ph[2], ph[3]));
  *out = finite ? phase : cadd(phase, phase);
}
static_assert(kRotThreads == 128, "phase_product multiplies four warps' products");

// A phase as phase_product left it, and whether the records behind it are finite.  The larger component of
// a phase is at most 1 and a few roundings, that of a doubled one at least 1.41.
__device__ __forceinline__ double2 phase_factor(double2 p, bool& finite) {
  const int top = max(__double2hiint(p.x) & 0x7fffffff, __double2hiint(p.y) & 0x7fffffff);
  if (top < 0x3ff40000) return p;  // 1.25
  finite = false;
  return cscale(p, 0.5);
}

// The common phase of all amplitudes, times one of them.  Phases of 1, -1, i and -i (none at all; rotations
// about X and Y, CRY) move components as they are: an infinite one must not make NaN of the other.  put(mul)
// is called with the form that the phase has, so that the choice is not made per amplitude (a predicated
// FP64 instruction takes the pipe as long as an executed one: 10 us for 1.2 million amplitudes).
struct PhaseTurn {
  bool swap;
  unsigned fx, fy;  // sign bits of the components
  __device__ __forceinline__ double2 operator()(double2 v) const {
    return make_double2(flip_sign(swap ? v.y : v.x, fx), flip_sign(swap ? v.x : v.y, fy));
  }
};
struct PhaseFactor {
  double2 p;
  __device__ __forceinline__ double2 operator()(double2 v) const { return cmul(p, v); }
};
template <class Put>
__device__ __forceinline__ void with_phase(double2 p, Put put) {
  if ((p.y == 0.0 && fabs(p.x) == 1.0) || (p.x == 0.0 && fabs(p.y) == 1.0)) {
    const bool swap = p.x == 0.0;
    const unsigned neg = (swap ? p.y : p.x) < 0.0 ? 0x80000000u : 0u;
    put(PhaseTurn{swap, swap ? neg ^ 0x80000000u : neg, neg});
  } else {
    put(PhaseFactor{p});
  }
}
__device__ __forceinline__ double2 phase_mul(double2 p, double2 v) {
  with_phase(p, [&](auto mul) { v = mul(v); });
  return v;
}

// The numbers of all operations of the runs of one CTA, for one parameter vector, in one go:
// thread i makes the matrix of run i, the first thread of each chain walks it.  phase_out receives
// the product of the runs' phases.
__device__ __forceinline__ void rot_plan_body(const RotPlan& pl, int cta, const double* theta, RotRec* recs,
                                              double2* phase_out, int deal) {
  __shared__ double2 Ms[kRotThreads][4];
  __shared__ int chain_of[kRotThreads], warp_heads[kRotThreads / 32];
  __shared__ double2 sc[kRotParams];
  const int base = pl.cta[cta], n = pl.cta[cta + 1] - base, i = threadIdx.x;
  cta_sincos(pl, cta, theta, sc);
  __syncthreads();
  RotRun run;
  if (i < n) {
    run = pl.runs[base + i];
    run_matrix(pl, run, sc, theta, Ms[i]);
  }
  // Chains of two and more runs are few and take longest: they are dealt out over `deal` warps.  All
  // four where the launch waits for one CTA (as few as possible wait for one another's branches); or, where runs
  // by themselves take as long as a step of a chain, the warps that have no runs of their own, so that the few
  // chains do not wait for those (60 gates of all kinds on five qubits applied to a matrix 83 -> 76 us).  Two, which hold
  // the most there can be, where the FP64 pipe is shared by many CTAs and takes as long for a warp of two
  // chains as for one of 32.
  const int warp = i >> 5, lane = i & 31;
  const bool head = i < n && !run.pulled && run.push != kAxisNone;
  const unsigned heads = __ballot_sync(0xffffffffu, head);
  if (lane == 0) warp_heads[warp] = __popc(heads);
  const bool general = i < n && !run.pulled && !head && (run.kind & kOpRot) && (run.kind & kOpZi) && !run.lone_u3;
  const bool long_runs = __syncthreads_or(general);
  int rank = __popc(heads & ((1u << lane) - 1)), nheads = 0;
  for (int w = 0; w < kRotThreads / 32; w++) {
    if (w < warp) rank += warp_heads[w];
    nheads += warp_heads[w];
  }
  int dealer = 0;  // the first warp
  const int used = (n + 31) >> 5, idle = kRotThreads / 32 - used;
  if (deal == kRotThreads / 32 && long_runs && nheads <= 2 * idle) dealer = used, deal = max(idle, 1);
  if (head) chain_of[(dealer + rank % deal) * 32 + rank / deal] = i;
  __syncthreads();
  const bool walks = warp >= dealer && warp < dealer + deal && lane * deal + (warp - dealer) < nheads;
  double2 phase = make_double2(1.0, 0.0);
  auto mat = [&](int j, const RotRun&, double2 M[4]) {
    for (int k = 0; k < 4; k++) M[k] = Ms[j - base][k];
  };
  for (int pass = 0; pass < 2; pass++) {
    // first the runs by themselves, each by its own thread, then the chains
    if (pass == 0 ? !(i < n && !run.pulled && run.push == kAxisNone) : !walks) continue;
    phase = cmul(phase, walk_chain(pl, base + (pass == 0 ? i : chain_of[i]), recs, mat));
  }
  __syncthreads();
  // the cosines of all runs at once: the chains need not wait for them
  const bool finite = i >= n || finish_record(run, recs[run.rec]);
  phase_product(phase, finite, phase_out);
}

// The same in three launches for many parameter vectors, the matrices kept in the records: a
// thread walks one chain of one vector, and the 32 of a warp the same chain of 32 vectors, so no
// lane idles or takes another's branch.
__device__ __forceinline__ void batch_matrices_body(const RotPlan& pl, int cta, const double* theta, RotRec* recs) {
  __shared__ double2 sc[kRotParams];
  const int base = pl.cta[cta], n = pl.cta[cta + 1] - base;
  cta_sincos(pl, cta, theta, sc);
  __syncthreads();
  if ((int)threadIdx.x >= n) return;
  const RotRun run = pl.runs[base + threadIdx.x];
  double2 M[4];
  run_matrix(pl, run, sc, theta, M);
  double2* out = reinterpret_cast<double2*>(recs + run.rec);
  for (int k = 0; k < 4; k++) out[k] = M[k];
}
// The phase of a chain is left in the place of its last run's cosine.
__device__ __forceinline__ void batch_chain_body(const RotPlan& pl, int head, RotRec* recs) {
  int last = 0;
  auto mat = [&](int, const RotRun& run, double2 M[4]) {
    const double2* in = reinterpret_cast<const double2*>(recs + run.rec);
    for (int k = 0; k < 4; k++) M[k] = in[k];
    last = run.rec;
  };
  const int first = pl.heads[head];
  const double2 phase = walk_chain(pl, first, recs, mat);
  if (pl.runs[first].kind == kOpCry) return;  // its cosine is in use, its phase 1
  recs[last].c = phase.x;
  recs[last].lo = phase.y;
}
__device__ __forceinline__ void batch_finish_body(const RotPlan& pl, int cta, RotRec* recs, double2* phase_out) {
  const int base = pl.cta[cta], n = pl.cta[cta + 1] - base;
  double2 phase = make_double2(1.0, 0.0);
  bool finite = true;
  if ((int)threadIdx.x < n) {
    const RotRun run = pl.runs[base + threadIdx.x];
    RotRec r = recs[run.rec];
    if (run.kind != kOpCry) {
      if (run.push == kAxisNone) phase = make_double2(r.c, r.lo);
      r.c = 1.0;
      r.lo = 0.0;
    }
    finite = finish_record(run, r);
    recs[run.rec].c = r.c;
    recs[run.rec].lo = r.lo;
  }
  phase_product(phase, finite, phase_out);
}

// ---- application ---------------------------------------------------------------------------
// Operation staged for the sweeps.  scale: the product of its group's cosines, multiplied in by the
// operation with kStRescale (whose t includes it; fixed point on the way back: fx_rescale).  zi.x of a kOpCry: its cosine.  mfac: what the
// overlaps measured behind the operation, with both vectors on the way back, are multiplied by.
struct StagedOp {
  int kind, coff;  // kind | mask << 8 | flags
  unsigned pair_row, crow_bits, cz;  // pair | row << 16, crow | b0 << 16 | b1 << 24, cz0 | cz1 << 16
  int pad;
  double t, scale, mfac;
  double2 zi, zo;
};
// kStInside: from the group's first rotation to before its last.
enum : int { kStTurn = 1 << 16, kStRescale = 1 << 17, kStInside = 1 << 18 };

// Loads operations [k0, k0 + kn) (at most kRotChunk) into st with the first warp of the CTA.
// The cosines that a group's rotations leave out are multiplied in by the first rotation in the
// direction of travel (FWD: the group's first, else its last): from there the scale rises back to
// 1, and amplitudes never exceed what they were.  FX: groups as kFxGroupBits ends them; both directions
// make the same ones.  The caller synchronises before and after.
template <bool FWD, bool FX>
__device__ __forceinline__ void stage_ops(StagedOp* st, const RotOp* ops, const RotRec* recs, int k0, int kn) {
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  const bool on = lane < kn;
  RotOp op = {kOpCnot, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
  RotRec r = {0.0, 1.0, make_double2(1.0, 0.0), make_double2(1.0, 0.0), 0.0, 0.0};
  if (on) {
    op = ops[k0 + lane];
    if (op.kind >= kOpCry) r = recs[op.rec];
  }
  const bool rot = (op.kind & kOpRot) != 0;
  int base = 0, end = 31;  // this lane's group
  if (FX) {
    // bits in front of this operation, in units of 2^-20: a group starts where they pass a multiple of
    // kFxGroupBits, so those of all but its last rotation stay below
    const int bits = rot ? (int)(-0x1p20f * __log2f((float)r.c)) : 0;
    int upto = bits;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const int before = (upto - bits) / kFxGroupBits, last = __shfl_up_sync(0xffffffffu, before, 1);
    const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || before != last);
    base = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
    const unsigned later = heads & ~(0xffffffffu >> (31 - lane));
    if (later) end = __ffs(later) - 2;
  }
  // product of the cosines of the group up to and including this operation, as pre + plo
  double pre = rot ? r.c : 1.0, plo = rot ? r.lo : 0.0;
  for (int o = 1; o < 32; o <<= 1) {
    if (FX && !__any_sync(0xffffffffu, lane - base >= o)) break;
    const double v = __shfl_up_sync(0xffffffffu, pre, o), vlo = __shfl_up_sync(0xffffffffu, plo, o);
    if (lane - base >= o) {
      const double p = pre * v;
      plo = fma(pre, v, -p) + fma(pre, vlo, plo * v);
      pre = p;
    }
  }
  const double all = __shfl_sync(0xffffffffu, pre + plo, end);
  const unsigned rots = __ballot_sync(0xffffffffu, rot) & (0xffffffffu >> (31 - end)) & (0xffffffffu << base);
  const int first = rots ? __ffs(rots) - 1 : 32, last = rots ? 31 - __clz(rots) : 32;
  const bool rescale = lane == (FWD ? first : last);
  if (on) {
    StagedOp s;
    s.kind = op.kind | op.mask << 8 | (r.turn ? kStTurn : 0) | (rescale ? kStRescale : 0) |
             (lane >= first && lane < last ? kStInside : 0);
    s.coff = op.coff;
    s.pair_row = op.pair | (unsigned)op.row << 16;
    s.crow_bits = op.crow | (unsigned)op.b0 << 16 | (unsigned)op.b1 << 24;
    s.cz = op.cz0 | (unsigned)op.cz1 << 16;
    s.pad = 0;
    s.scale = all;
    s.t = rescale && (FWD || !FX) ? r.t * all : r.t;
    s.mfac = 1.0;
    if (!FWD && lane < last) {
      const double inv = fast_rcp(pre + plo);
      s.mfac = inv * inv;
    }
    s.zi = op.kind == kOpCry ? make_double2(r.c, 0.0) : r.zi;
    s.zo = r.zo;
    st[lane] = s;
  }
}

enum { kRotFwd = 0, kRotAdj = 1, kRotTrans = 2 };  // G, G^dagger, G^T (right multiplication)

// The numbers of a staged operation in a direction: G^dagger takes -t and the conjugate phases,
// G^T takes -t about Y (Rx^T = Rx).  The negated copies are made here with integer operations
// (opaque_sign): the compiler's own took 18 % of a sweep's FP64 instructions.
struct DirOp {
  double t, nt, scale;
  double zix, ziy, nzi, zox, zoy, nzo;
  unsigned flip;  // sign bit for a turned Ry without a zi that could hold its sign
  bool turn;
};

template <int DIR, int KIND>
__device__ __forceinline__ DirOp directed(const StagedOp& s) {
  DirOp o;
  const unsigned sign = opaque_sign();
  const bool neg = DIR == kRotAdj || (DIR == kRotTrans && !(KIND & kOpX));
  const double t = s.t, nt = flip_sign(t, sign);
  o.t = neg ? nt : t;
  o.nt = neg ? t : nt;
  o.scale = s.scale;
  o.zix = s.zi.x;
  const double zi = s.zi.y, nzi = flip_sign(zi, sign);
  o.ziy = DIR == kRotAdj ? nzi : zi;
  o.nzi = DIR == kRotAdj ? zi : nzi;
  o.zox = s.zo.x;
  const double zo = s.zo.y, nzo = flip_sign(zo, sign);
  o.zoy = DIR == kRotAdj ? nzo : zo;
  o.nzo = DIR == kRotAdj ? zo : nzo;
  o.turn = (s.kind & kStTurn) != 0;
  o.flip = o.turn ? sign : 0u;
  return o;
}

// Where a staged operation finds its pairs, as in RotOp.
struct OpPlaces {
  unsigned pair, row, crow, cz0, cz1;
  int b0, b1;
};
__device__ __forceinline__ OpPlaces op_places(const StagedOp& s) {
  OpPlaces o;
  o.pair = s.pair_row & 0xffffu;
  o.row = s.pair_row >> 16;
  o.crow = s.crow_bits & 0xffffu;
  o.b0 = (s.crow_bits >> 16) & 255;
  o.b1 = s.crow_bits >> 24;
  o.cz0 = s.cz & 0xffffu;
  o.cz1 = s.cz >> 16;
  return o;
}

__device__ __forceinline__ unsigned parity(unsigned v) { return __popc(v) & 1u; }

// Places of pair q of an operation: x with its target bit 0, y with 1 (kOpCry: control bit 1).
template <int KIND>
__device__ __forceinline__ void pair_places(const OpPlaces& op, int q, int& ix, int& iy) {
  unsigned p;
  if (KIND == kOpCry) {
    const int lo = min(op.b0, op.b1), hi = max(op.b0, op.b1);
    p = ((q >> lo) << (lo + 1)) | (q & ((1 << lo) - 1));
    p = ((p >> hi) << (hi + 1)) | (p & ((1u << hi) - 1));
    p |= (parity(p & op.crow) ^ 1u) << op.b1;
  } else {
    p = ((q >> op.b0) << (op.b0 + 1)) | (q & ((1 << op.b0) - 1));
  }
  const unsigned par = parity(p & op.row) ? op.pair : 0u;
  ix = (int)(p ^ par);
  iy = (int)(p ^ par ^ op.pair);
}

// Signs of the CZ that rides on an operation.
__device__ __forceinline__ void pair_signs(const OpPlaces& op, int ix, int iy, double2& x, double2& y) {
  if (op.cz0) {
    const unsigned fx = (parity(ix & op.cz0) & parity(ix & op.cz1)) << 31;
    const unsigned fy = (parity(iy & op.cz0) & parity(iy & op.cz1)) << 31;
    x = make_double2(flip_sign(x.x, fx), flip_sign(x.y, fx));
    y = make_double2(flip_sign(y.x, fy), flip_sign(y.y, fy));
  }
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

// Controlled Ry on a pair with its control bit set: [[c, nt], [t, c]], t its sine.
__device__ __forceinline__ void cry_pair(const DirOp& op, double2& x, double2& y) {
  rot_turnless<false, true>(x, y, op.t, op.nt, op.zix);
}

// Applies one staged operation to every vector of a tile: tc vectors of length N = 2^logN, one
// after another in s.  All threads of the CTA.
template <int DIR, int KIND, bool RS>
__device__ __forceinline__ void rot_tile_kind(double2* s, int N, int logN, int tc, const StagedOp& staged) {
  const DirOp op = directed<DIR, KIND>(staged);
  const OpPlaces pl = op_places(staged);
  const int lognp = KIND == kOpCry ? logN - 2 : logN - 1;
  const int npairs = 1 << lognp;
  const int items = tc << lognp;
  for (int it = threadIdx.x; it < items; it += blockDim.x) {
    double2* v = s + (it >> lognp) * N;
    int ix, iy;
    pair_places<KIND>(pl, it & (npairs - 1), ix, iy);
    if (KIND == kOpPhase) {  // the target = 0 row is not touched
      double2 y = v[iy];
      rot_phase(y, op.zix, op.ziy, op.nzi);
      v[iy] = y;
      continue;
    }
    double2 x = v[ix], y = v[iy];
    if (DIR == kRotFwd) pair_signs(pl, ix, iy, x, y);
    if (KIND == kOpCry)
      cry_pair(op, x, y);
    else
      rot_pair<DIR, KIND, RS>(op, x, y);
    if (DIR != kRotFwd) pair_signs(pl, ix, iy, x, y);
    v[ix] = x;
    v[iy] = y;
  }
}

// A CZ by itself.
__device__ __forceinline__ void cz_tile(double2* s, int N, int tc, unsigned cz0, unsigned cz1) {
  for (int e = threadIdx.x; e < tc * N; e += blockDim.x) {
    const unsigned p = e & (N - 1);
    if (!(parity(p & cz0) & parity(p & cz1))) continue;
    const double2 v = s[e];
    s[e] = make_double2(dneg(v.x), dneg(v.y));
  }
}

template <int DIR>
__device__ __forceinline__ void rot_tile(double2* s, int N, int logN, int tc, const StagedOp& st) {
#define SQG_ROT_CASE(KIND) \
  case (KIND): \
    if (st.kind & kStRescale) \
      rot_tile_kind<DIR, (KIND), true>(s, N, logN, tc, st); \
    else \
      rot_tile_kind<DIR, (KIND), false>(s, N, logN, tc, st); \
    break;
  switch (st.kind & 255) {
    case kOpCz: cz_tile(s, N, tc, st.cz & 0xffffu, st.cz >> 16); break;
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

// Table of places behind the last operation, kEndGroups groups of 16 entries: the amplitude with
// index r is at the XOR over its hexadecimal digits d of table[16 g + d].  ends: RotPlan::ends or a
// state block's.  All threads of the CTA; the caller synchronises.
constexpr int kEndGroups = 4;
__device__ __forceinline__ void fill_end_table(int* table, const int* ends, int logN) {
  for (int e = threadIdx.x; e < 16 * kEndGroups; e += blockDim.x) {
    int p = 0;
    for (int q = 0; q < 4; q++)
      if (((e >> q) & 1) && (e >> 4) * 4 + q < logN) p ^= ends[(e >> 4) * 4 + q];
    table[e] = p;
  }
}
__device__ __forceinline__ int end_place(const int* table, int r) {
  return table[r & 15] ^ table[16 + ((r >> 4) & 15)] ^ table[32 + ((r >> 8) & 15)] ^ table[48 + ((r >> 12) & 15)];
}

}  // namespace sqg
