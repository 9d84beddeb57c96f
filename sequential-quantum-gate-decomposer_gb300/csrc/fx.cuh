// Fixed-point sweeps of the rotation plan, for the cost and its gradient.
//
// The FP64 pipe takes one warp instruction per 16 clocks and SM and answers after about 64; the
// integer multiplier takes a 32 x 32 -> 64 bit multiply-add per clock.  The amplitudes of a tile
// are bounded by its norm, so they fit 64-bit fixed point under one power of two, and a product
// with a coefficient of 62 bits costs three such multiplies and six adds and exclusive-ors
// instead of one FP64 instruction: about 6 clocks against 16, with a tenth of the latency.  The
// resolution is 2^-62 of the largest vector's norm, 2^-60 where a group of rotations has made the vectors
// shorter (kFxGroupBits); FP64 amplitudes round to 2^-53 of each, 2^-57 of the norm at 8 qubits.
// Cost and gradient are sums over all amplitudes, so an absolute resolution is what they need;
// matrices and state vectors that go back to the caller stay in FP64.  Tiles with infinities or
// NaN, and sweeps with checkpoints, stay in FP64 too.
// GB300, FP64 sweeps -> these: gradient at 8 qubits, 360 blocks, 128 vectors 179 -> 76 ms; at 10
// qubits, 300 blocks, 6 vectors 116 -> 50 ms; cost alone at 8 qubits, 120 blocks, 200 vectors 24.7
// -> 10.5 ms.  Error of the gradient against 64-bit reference values: 2.3e-14 at 8 and 8.8e-14 at
// 10 qubits, as with the gates as given in FP64.
#pragma once
#include "rot.cuh"

namespace sqg {

constexpr int kFxBits = 62;  // an amplitude of 1 (the largest norm of a tile's vectors, lambda's) is 2^62

struct Fx2 {
  long long x, y;
};
static_assert(sizeof(Fx2) == sizeof(double2), "tiles are converted in place");

// Coefficient c of |c| <= 1: upper 63 bits of 2^64 |c|, its sign in the lowest.  By shifts of its
// significand (no FP64 instruction); 1 itself becomes 1 - 2^-63.
__device__ __forceinline__ unsigned long long fx_encode(double c) {
  const unsigned long long v = (unsigned long long)__double_as_longlong(c);
  const int s = (int)((v >> 52) & 0x7ff) - 1012;  // 2^63 |c| = significand * 2^s
  const unsigned long long sig = (v & 0xfffffffffffffULL) | 0x10000000000000ULL;
  const unsigned long long m = s > 10 ? 0x7fffffffffffffffULL : s >= 0 ? sig << s : s > -64 ? sig >> -s : 0ULL;
  return m << 1 | v >> 63;
}

// The same, split for fx_mul.  xl, xh: what the halves of the amplitude w are exclusive-or'd with: to
// w + 2^63, or to its complement (2^63 - w - 1) for a negative coefficient.  k: what is added to
// fx_mul: less the offset's share 2^63 2^64|c| / 2^64, and the mean of what fx_mul drops (1.25, and
// |c| for the complement's one) to a whole unit.
struct FxCoef {
  unsigned h, l, xl, xh;
  unsigned long long k;
};
__device__ __forceinline__ FxCoef fx_coef(unsigned long long enc, bool flip) {
  FxCoef c;
  const unsigned neg = 0u - (((unsigned)enc & 1u) ^ (flip ? 1u : 0u));
  c.h = (unsigned)(enc >> 32);
  c.l = (unsigned)enc & ~1u;
  c.xl = neg;
  c.xh = 0x80000000u ^ neg;
  c.k = (neg && c.h >= 0x40000000u ? 2ULL : 1ULL) - (enc >> 1);
  return c;
}

// c * w - c.k for |w| <= 2^62: three of the four half products of (w + 2^63) * 2^64 |c| / 2^64.  With c.k
// the error is -2.25 to 1.75 units; in the mean -0.25 for positive c and -0.4 or 0.15 for negative c of
// less or more than 1/4.  An amplitude of zero becomes a unit under a positive c and stays or becomes minus one under a
// negative one.  Rounding both upper halves instead (multiply-adds for the upper multiplies) keeps a zero
// under a positive c, does not change the error of gradients (structured and deep circuits among them) and
// costs 13 % of a gradient.  In PTX: with the sum written in C++ the compiler (CUDA 13.0) lost a carry.
__device__ __forceinline__ unsigned long long fx_mul(long long w, const FxCoef& c) {
  const unsigned wh = (unsigned)((unsigned long long)w >> 32) ^ c.xh, wl = (unsigned)w ^ c.xl;
  unsigned long long p;
  asm("{\n\t"
      ".reg .u64 q;\n\t"
      ".reg .u32 a, b, n;\n\t"
      "mul.hi.u32 a, %1, %4;\n\t"
      "mul.hi.u32 b, %2, %3;\n\t"
      "add.cc.u32 a, a, b;\n\t"
      "addc.u32 n, 0, 0;\n\t"
      "mov.b64 q, {a, n};\n\t"
      "mad.wide.u32 %0, %1, %3, q;\n\t"
      "}"
      : "=l"(p)
      : "r"(wh), "r"(wl), "r"(c.h), "r"(c.l));
  return p;
}

// Numbers of a staged operation (its doubles replaced by fx_encode) in a direction.
struct FxOp {
  FxCoef t, nt, scale;       // t towards y, -t towards x (about X the signs alternate: use both)
  FxCoef zix, ziy, nzi, zox, zoy, nzo;
  bool turn;
};

__device__ __forceinline__ unsigned long long fx_bits(double v) { return (unsigned long long)__double_as_longlong(v); }

template <int DIR, int KIND, bool RS>
__device__ __forceinline__ FxOp fx_directed(const StagedOp& s) {
  FxOp o;
  constexpr bool ADJ = DIR == kRotAdj;
  if (KIND != kOpPhase) {
    o.t = fx_coef(fx_bits(s.t), ADJ);
    o.nt = fx_coef(fx_bits(s.t), !ADJ);
  }
  if (RS) o.scale = fx_coef(fx_bits(s.scale), false);
  if (KIND == kOpCry) o.scale = fx_coef(fx_bits(s.zi.x), false);
  if ((KIND & kOpZi) || KIND == kOpPhase) {
    o.zix = fx_coef(fx_bits(s.zi.x), false);
    o.ziy = fx_coef(fx_bits(s.zi.y), ADJ);
    o.nzi = fx_coef(fx_bits(s.zi.y), !ADJ);
  }
  if (KIND & kOpZo) {
    o.zox = fx_coef(fx_bits(s.zo.x), false);
    o.zoy = fx_coef(fx_bits(s.zo.y), ADJ);
    o.nzo = fx_coef(fx_bits(s.zo.y), !ADJ);
  }
  o.turn = (s.kind & kStTurn) != 0;
  return o;
}

__device__ __forceinline__ long long fx_neg_if(long long v, unsigned neg) {
  const long long m = -(long long)neg;
  return (v ^ m) - m;
}

// y <- z y
__device__ __forceinline__ void fx_phase(Fx2& y, const FxCoef& zx, const FxCoef& zy, const FxCoef& nzy) {
  const long long re = (long long)(fx_mul(y.x, zx) + fx_mul(y.y, nzy) + (zx.k + nzy.k));
  y.y = (long long)(fx_mul(y.y, zx) + fx_mul(y.x, zy) + (zx.k + zy.k));
  y.x = re;
}

// As rot_turnless.
template <bool AX, bool RS>
__device__ __forceinline__ void fx_turnless(Fx2& x, Fx2& y, const FxCoef& t, const FxCoef& nt, const FxCoef& scale) {
  Fx2 nx, ny;
  const unsigned long long xx = AX ? fx_mul(y.y, t) : fx_mul(y.x, nt), xy = AX ? fx_mul(y.x, nt) : fx_mul(y.y, nt);
  const unsigned long long yx = AX ? fx_mul(x.y, t) : fx_mul(x.x, t), yy = AX ? fx_mul(x.x, nt) : fx_mul(x.y, t);
  const unsigned long long kxx = AX ? t.k : nt.k, kxy = nt.k, kyx = t.k, kyy = AX ? nt.k : t.k;
  if (!RS) {
    nx.x = x.x + (long long)(xx + kxx);
    nx.y = x.y + (long long)(xy + kxy);
    ny.x = y.x + (long long)(yx + kyx);
    ny.y = y.y + (long long)(yy + kyy);
  } else {
    nx.x = (long long)(fx_mul(x.x, scale) + xx + (scale.k + kxx));
    nx.y = (long long)(fx_mul(x.y, scale) + xy + (scale.k + kxy));
    ny.x = (long long)(fx_mul(y.x, scale) + yx + (scale.k + kyx));
    ny.y = (long long)(fx_mul(y.y, scale) + yy + (scale.k + kyy));
  }
  x = nx;
  y = ny;
}

// As rot_pair, or cry_pair for kOpCry.
template <int DIR, int KIND, bool RS>
__device__ __forceinline__ void fx_pair(const FxOp& op, Fx2& x, Fx2& y) {
  constexpr bool AX = KIND & kOpX, ZI = KIND & kOpZi, ZO = KIND & kOpZo;
  if (KIND == kOpCry) {
    fx_turnless<false, true>(x, y, op.t, op.nt, op.scale);
    return;
  }
  if (DIR == kRotFwd) {
    if (ZI) fx_phase(y, op.zix, op.ziy, op.nzi);
    if (!ZI && !AX) y = {fx_neg_if(y.x, op.turn), fx_neg_if(y.y, op.turn)};
    const Fx2 a = op.turn ? y : x, b = op.turn ? x : y;
    x = a;
    y = b;
    fx_turnless<AX, RS>(x, y, op.t, op.nt, op.scale);
    if (ZO) fx_phase(y, op.zox, op.zoy, op.nzo);
  } else {
    if (ZO) fx_phase(y, op.zox, op.zoy, op.nzo);
    fx_turnless<AX, RS>(x, y, op.t, op.nt, op.scale);
    const Fx2 a = op.turn ? y : x, b = op.turn ? x : y;
    x = a;
    y = b;
    if (!ZI && !AX) y = {fx_neg_if(y.x, op.turn), fx_neg_if(y.y, op.turn)};
    if (ZI) fx_phase(y, op.zix, op.ziy, op.nzi);
  }
}

// As pair_signs.
__device__ __forceinline__ void fx_signs(const OpPlaces& pl, int ix, int iy, Fx2& x, Fx2& y) {
  if (pl.cz0) {
    const unsigned fx = parity(ix & pl.cz0) & parity(ix & pl.cz1);
    const unsigned fy = parity(iy & pl.cz0) & parity(iy & pl.cz1);
    x = {fx_neg_if(x.x, fx), fx_neg_if(x.y, fx)};
    y = {fx_neg_if(y.x, fy), fx_neg_if(y.y, fy)};
  }
}

// stage_ops with the numbers encoded; mfac times `unit`, the power of two that a sum of overlaps
// is multiplied by: done here once per chunk, not in the serial end of each operation.
template <bool FWD>
__device__ __forceinline__ void fx_stage_ops(StagedOp* st, const RotOp* ops, const RotRec* recs, int k0, int kn,
                                             double unit) {
  stage_ops<FWD, true>(st, ops, recs, k0, kn);
  if ((int)threadIdx.x >= kn) return;  // each thread the operation that it staged
  StagedOp& s = st[threadIdx.x];
  auto enc = [](double c) { return __longlong_as_double((long long)fx_encode(c)); };
  if (!FWD) s.mfac *= unit;
  s.t = enc(s.t);
  s.scale = enc(s.scale);
  s.zi = make_double2(enc(s.zi.x), enc(s.zi.y));
  s.zo = make_double2(enc(s.zo.x), enc(s.zo.y));
}

// One forward operation on a tile, as rot_tile.
template <int KIND, bool RS>
__device__ __forceinline__ void fx_tile_kind(Fx2* s, int N, int logN, int tc, const StagedOp& staged) {
  const FxOp op = fx_directed<kRotFwd, KIND, RS>(staged);
  const OpPlaces pl = op_places(staged);
  const int lognp = KIND == kOpCry ? logN - 2 : logN - 1;
  const int npairs = 1 << lognp;
  const int items = tc << lognp;
  for (int it = threadIdx.x; it < items; it += blockDim.x) {
    Fx2* v = s + (it >> lognp) * N;
    int ix, iy;
    pair_places<KIND>(pl, it & (npairs - 1), ix, iy);
    if (KIND == kOpPhase) {
      Fx2 y = v[iy];
      fx_phase(y, op.zix, op.ziy, op.nzi);
      v[iy] = y;
      continue;
    }
    Fx2 x = v[ix], y = v[iy];
    fx_signs(pl, ix, iy, x, y);
    fx_pair<kRotFwd, KIND, RS>(op, x, y);
    v[ix] = x;
    v[iy] = y;
  }
}

// Multiplies a group's scale into a tile behind the rotation that it belongs to, each thread on the pairs
// that it has rotated (no barrier between); until then amplitudes may reach 2^62.5.  The way back takes
// this pass of its own: with the scale in the rotation, as on the way up, every kind has a second form of
// 20 KB of code, which small tiles wait for.  GB300, gradients, in the rotation against here: four qubits, 1024
// vectors 744, 685 us; eight qubits, 128 vectors 75.4, 75.9 ms; 60 instances of 3 to 8 qubits 2.76, 2.78 ms.
__device__ __forceinline__ void fx_rescale(Fx2* s, int N, int logN, int tc, const StagedOp& staged) {
  const OpPlaces pl = op_places(staged);
  const FxCoef c = fx_coef(fx_bits(staged.scale), false);
  auto scaled = [&](Fx2 v) {
    return Fx2{(long long)(fx_mul(v.x, c) + c.k), (long long)(fx_mul(v.y, c) + c.k)};
  };
  const int npairs = 1 << (logN - 1);
  for (int it = threadIdx.x; it < tc << (logN - 1); it += blockDim.x) {
    Fx2* v = s + (it >> (logN - 1)) * N;
    int ix, iy;
    pair_places<kOpRot>(pl, it & (npairs - 1), ix, iy);
    v[ix] = scaled(v[ix]);
    v[iy] = scaled(v[iy]);
  }
}

__device__ __forceinline__ void fx_cz_tile(Fx2* s, int N, int tc, unsigned cz0, unsigned cz1) {
  for (int e = threadIdx.x; e < tc * N; e += blockDim.x) {
    const unsigned p = e & (N - 1);
    if (!(parity(p & cz0) & parity(p & cz1))) continue;
    const Fx2 v = s[e];
    s[e] = {-v.x, -v.y};
  }
}

__device__ __forceinline__ void fx_tile(Fx2* s, int N, int logN, int tc, const StagedOp& st) {
#define SQG_ROT_CASE(KIND) \
  case (KIND): \
    if (st.kind & kStRescale) \
      fx_tile_kind<(KIND), true>(s, N, logN, tc, st); \
    else \
      fx_tile_kind<(KIND), false>(s, N, logN, tc, st); \
    break;
  switch (st.kind & 255) {
    case kOpCz: fx_cz_tile(s, N, tc, st.cz & 0xffffu, st.cz >> 16); break;
    case kOpCry: fx_tile_kind<kOpCry, false>(s, N, logN, tc, st); break;
    case kOpPhase: fx_tile_kind<kOpPhase, false>(s, N, logN, tc, st); break;
    SQG_ROT_CASE(kOpRot)
    SQG_ROT_CASE(kOpRot | kOpX)
    SQG_ROT_CASE(kOpRot | kOpZi)
    SQG_ROT_CASE(kOpRot | kOpX | kOpZi)
    SQG_ROT_CASE(kOpRot | kOpZi | kOpZo)
  }
#undef SQG_ROT_CASE
}

// ---- overlaps ----------------------------------------------------------------------------------
// Amplitude h 2^32 + l with the nearest h: the product of two l that is left out has no bias, and
// none at all where an amplitude is a few units (a floor would leave l close to 2^32 for a small
// negative one, half a unit for every pair of a lambda that is still sparse).
struct FxHalf {
  int h, l;
};
__device__ __forceinline__ FxHalf fx_half(long long v) {
  const int l = (int)v;
  return {(int)(v >> 32) - (l >> 31), l};
}
// Sum of at most four products of amplitudes of two pairs / 2^64, its low part kept to 64 bits until
// fx_less: rounding each product would leave a bias that depends on which components are zero, and
// sum it over the amplitudes.
struct FxSum {
  long long hi, mid;
};
__device__ __forceinline__ void fx_add(FxSum& s, FxHalf a, FxHalf b) {
  s.hi += (long long)a.h * b.h;
  s.mid += (long long)a.h * b.l;
  s.mid += (long long)a.l * b.h;
}
__device__ __forceinline__ long long fx_less(const FxSum& s, const FxSum& u) {
  return (s.hi - u.hi) + ((s.mid - u.mid + 0x80000000LL) >> 32);
}

// A thread's sum (|sum| <= 2^60 per vector, at most kFxItems vectors) / 2^shift, so that those of a
// whole tile can be added; halves to the even side: a bias of half a unit's last place would add
// up over the threads.
constexpr int kFxItems = 7;
__device__ __forceinline__ int fx_sum_shift(int tc) { return tc > 4 ? 30 - __clz(tc - 1) : 0; }  // 2^(62 - 60) vectors fit
__device__ __forceinline__ long long fx_scaled(long long v, int shift) {
  return shift ? (v + ((1LL << (shift - 1)) - 1) + ((v >> shift) & 1)) >> shift : v;
}

// As measure_pair.
template <bool CPLX, int MASK>
__device__ __forceinline__ void fx_measure(const Fx2& x, const Fx2& y, const Fx2& lx, const Fx2& ly,
                                           long long (&acc)[CPLX ? 6 : 3]) {
  const FxHalf xx = fx_half(x.x), xy = fx_half(x.y), yx = fx_half(y.x), yy = fx_half(y.y);
  const FxHalf lxx = fx_half(lx.x), lxy = fx_half(lx.y), lyx = fx_half(ly.x), lyy = fx_half(ly.y);
  // (a b + c d) - (e f + g h)
  auto folded = [](FxHalf a, FxHalf b, FxHalf c, FxHalf d, FxHalf e, FxHalf f, FxHalf g, FxHalf h) {
    FxSum s = {0, 0}, u = {0, 0};
    fx_add(s, a, b);
    fx_add(s, c, d);
    fx_add(u, e, f);
    fx_add(u, g, h);
    return fx_less(s, u);
  };
  auto plus = [](FxHalf a, FxHalf b, FxHalf c, FxHalf d) {
    FxSum s = {0, 0};
    fx_add(s, a, b);
    fx_add(s, c, d);
    return fx_less(s, {0, 0});
  };
  auto minus = [](FxHalf a, FxHalf b, FxHalf c, FxHalf d) {  // a b - c d
    FxSum s = {0, 0}, u = {0, 0};
    fx_add(s, a, b);
    fx_add(u, c, d);
    return fx_less(s, u);
  };
  if (!CPLX) {
    if (MASK & 1) acc[0] += folded(lxx, yy, lyx, xy, lxy, yx, lyy, xx);
    if (MASK & 2) acc[1] += folded(lyx, xx, lyy, xy, lxx, yx, lxy, yy);
    if (MASK & 4) acc[2] += minus(lxx, xy, lxy, xx);
  } else {
    if (MASK & 4) {
      acc[0] += plus(lxx, xx, lxy, xy);
      acc[1] += minus(lxx, xy, lxy, xx);
    }
    if (MASK & 3) {
      acc[2] += plus(lxx, yx, lxy, yy);
      acc[3] += minus(lxx, yy, lxy, yx);
      acc[4] += plus(lyx, xx, lyy, xy);
      acc[5] += minus(lyx, xy, lyy, xx);
    }
  }
}

template <bool CPLX, int KIND, int MASK>
__device__ __forceinline__ void fx_adjoint_kind(Fx2* psi, Fx2* lam, int N, int logN, int tc, const StagedOp& staged,
                                                long long (&acc)[CPLX ? 6 : 3]) {
  const FxOp op = fx_directed<kRotAdj, KIND, false>(staged);
  const OpPlaces pl = op_places(staged);
  const int lognp = KIND == kOpCry ? logN - 2 : logN - 1;
  const int npairs = 1 << lognp;
  const int items = tc << lognp;
  for (int it = threadIdx.x; it < items; it += blockDim.x) {
    const int col = it >> lognp;
    Fx2* ps = psi + col * N;
    Fx2* ls = lam + col * N;
    int ix, iy;
    pair_places<KIND>(pl, it & (npairs - 1), ix, iy);
    Fx2 x = ps[ix], y = ps[iy], lx = ls[ix], ly = ls[iy];
    fx_measure<CPLX, MASK>(x, y, lx, ly, acc);
    if (KIND == kOpPhase) {
      fx_phase(y, op.zix, op.ziy, op.nzi);
      fx_phase(ly, op.zix, op.ziy, op.nzi);
    } else {
      fx_pair<kRotAdj, KIND, false>(op, x, y);
      fx_signs(pl, ix, iy, x, y);
      fx_pair<kRotAdj, KIND, false>(op, lx, ly);
      fx_signs(pl, ix, iy, lx, ly);
      ps[ix] = x;
      ls[ix] = lx;
    }
    ps[iy] = y;
    ls[iy] = ly;
  }
}

template <bool CPLX>
__device__ __forceinline__ void fx_adjoint(Fx2* psi, Fx2* lam, int N, int logN, int tc, const StagedOp& st,
                                           long long (&acc)[CPLX ? 6 : 3]) {
#define SQG_ROT_CASE(KIND, MASK) \
  case (KIND) | (MASK) << 8: fx_adjoint_kind<CPLX, (KIND), (MASK)>(psi, lam, N, logN, tc, st, acc); break;
  switch (st.kind & 0xffff) {
    case kOpCry | 2 << 8: fx_adjoint_kind<CPLX, kOpCry, 2>(psi, lam, N, logN, tc, st, acc); break;
    case kOpPhase | 4 << 8: fx_adjoint_kind<CPLX, kOpPhase, 4>(psi, lam, N, logN, tc, st, acc); break;
    SQG_ROT_CASE(kOpRot, 2)
    SQG_ROT_CASE(kOpRot | kOpX, 1)
    SQG_ROT_CASE(kOpRot | kOpZi, 3)
    SQG_ROT_CASE(kOpRot | kOpZi, 6)
    SQG_ROT_CASE(kOpRot | kOpX | kOpZi, 5)
    SQG_ROT_CASE(kOpRot | kOpZi | kOpZo, 7)
  }
#undef SQG_ROT_CASE
  if (st.kind & kStRescale) {
    fx_rescale(psi, N, logN, tc, st);
    fx_rescale(lam, N, logN, tc, st);
  }
}

// Warp totals of up to eight sums: lane l ends with value (l >> 2) & 7.
__device__ __forceinline__ long long fx_reduce_scatter8(long long r[8]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 16, half = 4; half >= 1; o >>= 1, half >>= 1) {
    const bool hi = lane & o;
#pragma unroll
    for (int k = 0; k < half; k++) {
      const long long send = hi ? r[k] : r[k + half], keep = hi ? r[k + half] : r[k];
      r[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  long long v = r[0];
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v;
}

}  // namespace sqg
