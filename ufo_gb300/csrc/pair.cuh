// pair.cuh -- one particle on two lanes: the horizontal plane (x, px) on the
// even lane, the vertical one (y, py) on the odd lane.
//
// Why.  A sub-partition of this GPU starts one FP64 warp instruction every
// 64.6 cycles, whatever the active mask and however many independent chains
// the warp holds (ufo_fp64_probe), so a warp's time is its number of FP64
// instructions.  With a particle per lane every drift, kick and thick map
// spends one instruction per plane; with a plane per lane one instruction does
// both.  A warp then carries 16 particles and half the instructions: a launch
// with fewer warps than sub-partitions (608) finishes in about half the time,
// and at full occupancy the work is the same but comes in twice as many,
// shorter warps, which spread more evenly.  What couples the planes (z = x+iy
// of a kick, an aperture) goes through a warp shuffle.
//
// Results are those of the one-lane interpreter (one_turn) bit for bit (up to
// the sign of an exact zero): every quantity is formed by the same IEEE
// operations; a - b*c is evaluated as a + (-b)*c and the like, which only moves
// signs, and a term that one plane lacks is added there as a zero.  The trimmed
// expressions of the fast paths hold for finite coordinates, and a coordinate
// that left the finite range never returns (x += px L keeps inf and NaN).  So
// the list is cut into segments of 16 ops: a segment in which some particle
// ends non-finite is run again from its entry state by the one-lane code on the
// gathered state (`wide`).
//
// Latency.  FP64 results reach the next FP64 instruction of a chain in 64.6
// cycles but any other instruction only after about 115 (measured: one integer
// operation, shuffle, vote or select per step of a dependent DFMA chain takes
// the step from 64.7 to 114-115 cycles).  The code therefore keeps selects and
// sign changes on constants and off the chain, and tests once per segment.
#pragma once
#include "pair_list.h"

namespace ufo {

struct Half {
  double u, pu;  // (x, px) on even lanes, (y, py) on odd lanes
};

// a lane's state besides its coordinates
struct PairCtx {
  double o;       // 1 / (1 + dp)
  const double *tab;
  int neg;        // sign bit on even lanes: a - b as a + (b ^ neg)
  int group;      // the warp's lanes of the coefficient cache
  bool even;
  bool dead;      // no particle, or all four coordinates are NaN (they stay NaN)
  bool bad_o;     // o is not finite
};

// what only some ops read, kept out of the registers
struct PairShared {
  // particle; PAIR_NONE: none (the lane runs along on zeros); PAIR_ORBIT: a
  // closed-orbit trial (z = dp = 0)
  int64_t p[32];
  double *obs[32];       // this turn's first observation slot, or null
  int64_t obs_left[32];  // observation slots left from there
  int turn[32], target[32];
  // the lane's state across the out-of-line calls
  double u[32], pu[32], o[32];
  const double *tab[32];
  bool dead[32];
};

constexpr unsigned PAIR_ALL = 0xffffffffu;
constexpr int64_t PAIR_NONE = -1, PAIR_ORBIT = -2;

UFO_DEV double pair_other(double v) { return __shfl_xor_sync(PAIR_ALL, v, 1); }
UFO_DEV double flip(double v, int bit) {
  return __hiloint2double(__double2hiint(v) ^ bit, __double2loint(v));
}
UFO_DEV double pick(bool first, double a, double b) { return first ? a : b; }

// Correctly rounded a / d for a small integer d with one FMA: q = RN(a r + u),
// r = RN(1/d), u = +-a 2^-s (the exponent field moved, no FP64 instruction).
// With r = 1/d - eps ulp(r) the exact quotient is a r + a eps ulp(r).  N/d for
// an integer N is at least 1/(2 d') ulp away from every rounding boundary (d'
// the odd part of d: 2N - (2i+1) d' is odd), so any u closer to a eps ulp(r)
// than that gives the correctly rounded quotient; the host admits the form
// when a power of two is (d' = 3: eps = 1/3, 1/4 serves; d' = 7: eps = 2/7,
// 1/4 serves; d' = 5 has none and keeps the general form).  A zero takes u = 0;
// `bad` collects operands whose exponent the shift would take out of range, and
// the subnormal ones, whose quotient by an even d may be a tie (9 2^-1074 / 6).
UFO_DEV double div_shift(double a, double r, int shift_hi, int sign, bool &bad) {
  const int hi = __double2hiint(a), lo = __double2loint(a);
  const unsigned mag = static_cast<unsigned>(hi) & 0x7fffffffu;
  const bool zero = (mag | static_cast<unsigned>(lo)) == 0;
  bad = bad || (!zero && mag < 0x07100000u);
  const double u = __hiloint2double(zero ? 0 : (hi - shift_hi) ^ sign, lo);
  return fma_(a, r, u);
}

// divc without its branch: operands outside its range set `bad`
UFO_DEV double div_markstein(double a, double d, double r, bool &bad) {
  const int hi = __double2hiint(a);
  const unsigned e = static_cast<unsigned>(hi) & 0x7ff00000u;
  const bool zero = ((hi & 0x7fffffff) | __double2loint(a)) == 0;
  bad = bad || (!zero && e - 0x07700000u > 0x77f00000u - 0x07700000u);
  const double q0 = mul(a, r);
  return fma_(fma_(-q0, d, a), r, q0);
}

// a / order of the strict Horner scheme
UFO_DEV double div_order_pair(double a, int order, bool &bad) {
  if (order == 1) return a;
  if (order == 2) return mul(a, 0.5);
  if (order == 4) return mul(a, 0.25);
  const double r = c_rcp_order[order];
  if (order == 3) return div_shift(a, r, 56 << 20, 0, bad);
  return div_markstein(a, static_cast<double>(order), r, bad);
}

// Correctly rounded a / d with r = RN(1/d) and z = RN((1 - d r)/d) prepared:
// q1 = RN(a r + RN(a z)) is within an ulp of a/d, and Markstein's correction
// with the exact remainder rounds it correctly.  The caller keeps a and d in
// the range where nothing under- or overflows.
UFO_DEV double div_prepared(double a, double d, double r, double z) {
  const double q1 = fma_(a, r, mul(a, z));
  return fma_(fma_(-q1, d, a), r, q1);
}

// ---------------------------------------------------------------- wide ops
template <bool FMA>
__device__ __noinline__ P4 wide_op(double x, double px, double y, double py, double z, double dp,
                                   double o, int turn, const Op *raw, const double *c) {
  State s{};
  s.x = x; s.px = px; s.y = y; s.py = py; s.z = z; s.dp = dp; s.o = o;
  s.opdp = add(1., dp);
  s.turn = turn;
  s.bad_o = nf(o);
  const int4 w0 = __ldg(reinterpret_cast<const int4 *>(raw));
  const int4 w1 = __ldg(reinterpret_cast<const int4 *>(raw) + 1);
  apply_op<FMA, true>(s, Op{w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w}, c, [](int) {});
  return {s.x, s.px, s.y, s.py};
}

// ---------------------------------------------------------------- kicks
// One Horner pass of the strict mode (methods.kick, ufo/methods.py:45-76) over
// a trimmed coefficient list, the pair form of horner_trim: the even lane
// holds dpx, the odd lane dpy.  Normal: dpx = a, dpy = b; skew: dpx = b,
// dpy = a.  Returns this lane's kick.
template <bool SKEW>
UFO_DEV double pair_horner(double u, double v, const PairCtx &x, uint32_t mask, const double *c,
                           double o1, bool &bad) {
  const int m = 31 - __clz(mask);
  int k = __popc(mask) - 1;
  const double top = mul(ld(c + k), o1);
  --k;
  // lane that carries `a` (the accumulator the coefficients enter)
  const bool lane_a = SKEW ? !x.even : x.even;
  if (m == 0) return lane_a ? top : 0.0;
  double own;
  for (int order = m; order > 0; --order) {
    if (order == m) {  // b is an exact zero: na = a x, nb = +-a y
      own = mul(top, SKEW ? flip(v, x.neg) : u);
    } else {
      const double oth = pair_other(own);
      const double A = pick(lane_a, own, oth), B = pick(lane_a, oth, own);
      own = add(mul(SKEW ? B : A, u), mul(flip(SKEW ? A : B, x.neg), v));
    }
    own = div_order_pair(own, order, bad);
    if ((mask >> (order - 1)) & 1u) {
      own = add(lane_a ? mul(ld(c + k), o1) : 0.0, own);
      --k;
    }
  }
  return own;
}

// General kick on finite coordinates: the new momentum.  Strict mode: the
// normal, then the skew list.
UFO_DEV double pair_kick_strict(const Half &h, const PairCtx &x, double o1, uint32_t masks,
                                const double *c, bool &bad) {
  const double v = pair_other(h.u);
  const uint32_t mn = masks & 0xffffu, ms = masks >> 16;
  double pu = h.pu;
  if (mn) pu = add(pu, flip(pair_horner<false>(h.u, v, x, mn, c, o1, bad), x.neg));
  if (ms) pu = add(pu, flip(pair_horner<true>(h.u, v, x, ms, c + __popc(mn), o1, bad), x.neg));
  return pu;
}

// With FMA: one complex Horner pass over the dense series of M terms
// (kick_pser_ool)
UFO_DEV double pair_kick_series(const Half &h, const PairCtx &x, double o1, int M,
                                const double *ps) {
  const double v = pair_other(h.u);
  const double *q = ps + (x.even ? 0 : M);
  double own = ld(q + M - 1);
  const double vs = flip(v, x.neg);
#pragma unroll 1
  for (int n = M - 2; n >= 0; --n) {
    const double oth = pair_other(own);
    own = fma_(pick(x.even, own, oth), h.u, fma_(pick(x.even, oth, own), vs, ld(q + n)));
  }
  return fma_(flip(o1, x.neg), own, h.pu);
}

// ---------------------------------------------------------------- teapot
// one kick; t: the strength (with the plane's sign, pair_strength), or the
// factor o of a general kick
template <bool FMA, int PAT>
UFO_DEV void pair_kick(Half &h, const PairCtx &x, uint32_t masks, const double *ck, double t,
                       const double *ps, bool &bad) {
  if (PAT == 0) {
    h.pu = FMA ? pair_kick_series(h, x, t, pser_len(masks & 0xffffu, masks >> 16), ps)
               : pair_kick_strict(h, x, t, masks, ck, bad);
  } else if (PAT == 1) {
    h.pu = FMA ? fma_(t, h.u, h.pu) : add(h.pu, mul(t, h.u));
  } else if (PAT == 2) {
    const double v = pair_other(h.u);
    if (FMA) {  // px -= t (x^2 - y^2), py += 2t xy
      const double m = mul(v, pick(x.even, flip(v, x.neg), h.u));  // -y^2 | xy
      h.pu = fma_(t, fma_(pick(x.even, h.u, 0.0), h.u, m), h.pu);
    } else {  // a = t x, b = t y; px -= a x - b y; py += a y + b x
      const double own = mul(t, h.u);  // -a | b
      const double oth = pair_other(own);
      const double A = pick(x.even, own, flip(oth, static_cast<int>(0x80000000u)));
      const double B = pick(x.even, oth, own);
      h.pu = add(h.pu, add(mul(A, h.u), mul(B, v)));
    }
  }
}

template <bool FMA, int PAT>
UFO_DEV double pair_strength(const PairCtx &x, double K, double o1) {
  if (PAT == 0 || PAT == 3) return o1;
  // constants carry the signs and the factor 1/2 (exact unless K is subnormal,
  // which the host keeps from this path)
  if (PAT == 1 || (FMA && !x.even)) return mul(flip(K, x.neg), o1);
  return mul(mul(flip(K, x.neg), o1), 0.5);
}

template <bool FMA>
UFO_DEV void pair_drift(Half &h, double L) {
  h.u = FMA ? fma_(h.pu, L, h.u) : add(h.u, mul(h.pu, L));
}

// DIV = DIV_ANY, WEAK = 2: decided at run time (the general kicks, whose code
// is long and is instantiated once)
template <bool FMA, int PAT, int DIV, int WEAK>
UFO_DEV void pair_teapot(Half &h, const PairCtx &x, const PairOp &op, double Lo, const double *c,
                         bool &bad) {
  const int N = op.a;
  const uint32_t masks = static_cast<uint32_t>(op.b);  // general kicks only
  const double o1 = (op.head & PF_ACHRO) ? 1.0 : x.o;
  const bool table_div = op.head & PF_DIV;
  const int variant = (op.head & 0xff) - PV_TEAPOT;
  const int form = DIV == DIV_ANY ? variant / 4 % 3 : DIV;
  const bool weak = WEAK == 2 ? variant >= 12 : WEAK != 0;
  const double *ck = c + 1 + (N > 1 ? (table_div ? 4 : 1) : 0);
  double Li = 0.0, A = 0.0, d = 0.0, r = 0.0;
  if (N <= 1) {
    // a single slice has no inner drift
  } else if (FMA || form == DIV_NONE) {
    Li = ld(c + (table_div ? 4 : 1));
  } else {
    A = ld(c + 1);
    d = ld(c + 2);
    r = ld(c + 3);
  }
  const int nk = PAT == 0 ? __popc(masks) : PAT == 3 ? 0 : 1;
  const double W = weak && x.even ? ld(ck + nk) : 0.0;
  const double Lx = (op.head & PF_SPLITO) ? ld(ck + nk + (weak ? 1 : 0)) : Lo;
  const double t = pair_strength<FMA, PAT>(x, PAT == 1 || PAT == 2 ? ld(ck) : 0.0, o1);
  const double *ps =
      FMA && PAT == 0 ? ck + nk + (weak ? 1 : 0) + ((op.head & PF_SPLITO) ? 1 : 0) : nullptr;
  const int shift_hi = ((op.head >> 8) & 0xff) << 20;
  const int sign = static_cast<int>(static_cast<unsigned>(op.head & PF_NEG) << 15);
  const bool then = !FMA && PAT != 0 && (op.head & PF_THEN);
  const double Lt = then ? ld(x.tab + op.b) : 0.0;
  const bool shifts = PAT == 0 && (op.head & (x.even ? PF_X : PF_Y));
  double post = 0.0;
  if (PAT == 0 && (op.head & PF_POST)) {
    const double *end = ck + nk + (weak ? 1 : 0) + ((op.head & PF_SPLITO) ? 1 : 0) +
                        ((op.head & PF_PSER) ? 2 * pser_len(masks & 0xffffu, masks >> 16) : 0) +
                        ((op.head & PF_POST_EDGE) ? 3 : 0);
    if (shifts) post = ld(end + (x.even ? 0 : 1));
  }
  if (PAT == 0 && (op.head & PF_PRE))
    h.u = sub(h.u, shifts ? ld(c - ((op.head & PF_PRE_EDGE) ? 5 : 2) + (x.even ? 0 : 1)) : 0.0);
  pair_drift<FMA>(h, Lo);
  for (int sl = 1;; ++sl) {
    pair_kick<FMA, PAT>(h, x, masks, ck, t, ps, bad);
    if (weak) h.pu = FMA ? fma_(-h.u, W, h.pu) : sub(h.pu, mul(h.u, W));
    if (sl >= N) break;
    if (FMA || form == DIV_NONE)
      pair_drift<FMA>(h, Li);
    else if (form == DIV_SHIFT)
      h.u = add(h.u, div_shift(mul(h.pu, A), r, shift_hi, sign, bad));
    else
      h.u = add(h.u, div_markstein(mul(h.pu, A), d, r, bad));
  }
  pair_drift<FMA>(h, Lx);
  if (PAT == 0 && (op.head & PF_POST)) h.u = sub(h.u, post);
  if (then) pair_drift<FMA>(h, Lt);
}

// ---------------------------------------------------------------- thick
// A thick map is linear in the plane's coordinates with coefficients that
// depend on the particle's momentum alone (ufo/methods.py:99-196):
//   u' = C u + S pu / k2 + D,   pu' = -+S u k2 + C pu + DP.
// The coefficients are formed in a particle's first turn, by the operations of
// thick_quad / thick_bend, and kept for the launch in a per-lane cache; the
// later turns issue 11 to 13 FP64 instructions instead of a square root, a
// sine, a cosine, two hyperbolic functions and the divisions.  k2 = 0 marks a
// plane that is a drift (C = 1, S = length, pu unchanged); r = 0 one that
// takes the one-lane code (k2 out of range, undefined strength).
struct ThickHalf { double C, S, k, r, z, D, DP; };

UFO_DEV void thick_put(const ThickHalf &t, double *out, int64_t n, bool bend) {
  out[TC_C * n] = t.C;
  out[TC_S * n] = t.S;
  out[TC_K * n] = t.k;
  out[TC_R * n] = t.r;
  out[TC_Z * n] = t.z;
  if (bend) {
    out[TC_D * n] = t.D;
    out[TC_DP * n] = t.DP;
  }
}

UFO_DEV void thick_recip(ThickHalf &t, double k2) {
  const unsigned e = static_cast<unsigned>(__double2hiint(k2)) & 0x7ff00000u;
  if (e - 0x30000000u > 0x20000000u) {  // outside [2^-255, 2^257]: not prepared
    t.r = 0.0;
    t.z = 0.0;
    return;
  }
  t.r = dvd(1.0, k2);
  t.z = mul(fma_(-k2, t.r, 1.0), t.r);
}

__device__ __noinline__ void thick_quad_half(double o, int flags, const double *c, double *out,
                                             int64_t n) {
  const bool even = (threadIdx.x & 1) == 0;
  const double k = ld(c), Lf = ld(c + 1);
  const bool foc = even ? k > 0. : !(k > 0.);
  ThickHalf t;
  double k2;
  if (flags & PF_CONST) {
    k2 = ld(c + 2);
    t.C = ld(c + (foc ? 3 : 5));
    t.S = ld(c + (foc ? 4 : 6));
  } else {
    k2 = __dsqrt_rn(fabs((flags & PF_ACHRO) ? k : mul(k, o)));
    const double k2l = mul(Lf, k2);
    if (foc) {
      sincos(k2l, &t.S, &t.C);
    } else {
      t.C = cosh(k2l);
      t.S = sinh(k2l);
    }
  }
  t.k = foc ? -k2 : k2;
  thick_recip(t, k2);
  thick_put(t, out, n, false);
}

__device__ __noinline__ void thick_bend_half(double o, double dp, int flags, const double *c,
                                             double *out, int64_t n) {
  const bool even = (threadIdx.x & 1) == 0;
  const bool achro = flags & PF_ACHRO;
  const double Lf = ld(c + 2);
  const double curv = achro ? ld(c) : mul(ld(c), o);
  const double *q = c + (even ? 9 : 3);  // folded constants of this plane
  double k = (flags & PF_CONST) ? ld(q) : achro ? ld(c + 1) : mul(ld(c + 1), o);
  if (even && !(flags & PF_CONST))
    k = add(k, achro ? mul(curv, curv) : dvd(mul(curv, curv), o));
  ThickHalf t;
  t.D = t.DP = -0.0;
  if (k == 0.) {  // a drift: u += Lf pu
    t.C = 1.0;
    t.S = Lf;
    t.k = 0.0;
    t.r = 1.0;
    t.z = 0.0;
    thick_put(t, out, n, true);
    return;
  }
  const bool foc = even ? k > 0. : k < 0.;
  const double k2 = (flags & PF_CONST) ? ld(q + 1) : __dsqrt_rn(fabs(k));
  if (flags & PF_CONST) {
    t.C = ld(q + (foc ? 2 : 4));
    t.S = ld(q + (foc ? 3 : 5));
  } else {
    const double k2l = mul(Lf, k2);
    if (foc) {
      sincos(k2l, &t.S, &t.C);
    } else {
      t.C = cosh(k2l);
      t.S = sinh(k2l);
    }
  }
  t.k = foc ? -k2 : k2;
  thick_recip(t, k2);
  if (isnan(k)) t.r = 0.0;
  if (even) {
    const double ak = (flags & PF_CONST) ? ld(c + 15) : fabs(k);
    const double dc = mul(dp, curv);
    t.D = dvd(mul(dc, foc ? sub(1., t.C) : sub(t.C, 1.)), ak);
    t.DP = dvd(mul(dc, t.S), k2);
  }
  thick_put(t, out, n, true);
}

// this lane's entry of a cache field; `group`: the warp's 32 lanes of the cache
UFO_DEV double *pair_cache(const TrackArgs &a, int field, int group) {
  return a.cache + field * a.cache_lanes + static_cast<int64_t>(group) * 32 + threadIdx.x;
}

// tan(psi) of a fringe-field edge (edge in ops.cuh)
__device__ __noinline__ double edge_psi_tan(double curv, const double *c) {
  return tan(sub(ld(c + 2), mul(dvd(mul(mul(2.0, curv), ld(c + 3)), ld(c + 4)), ld(c + 5))));
}

// sets `bad` when the plane needs the one-lane code
UFO_DEV void thick_apply(Half &h, const double *t, int64_t n, bool bend, bool &bad) {
  const double C = t[TC_C * n], S = t[TC_S * n], k = t[TC_K * n], r = t[TC_R * n],
               z = t[TC_Z * n];
  const double a = mul(S, h.pu);
  const int hi = __double2hiint(a);
  const unsigned e = static_cast<unsigned>(hi) & 0x7ff00000u;
  const bool zero = ((hi & 0x7fffffff) | __double2loint(a)) == 0;
  const bool drift = (__double2hiint(k) & 0x7fffffff) == 0;
  bad = bad || __double2hiint(r) == 0 || (!zero && e - 0x1f000000u > 0x60f00000u - 0x1f000000u);
  // |k| by its sign bit (an FP64 instruction otherwise)
  const double d = __hiloint2double(drift ? 0x3ff00000 : __double2hiint(k) & 0x7fffffff,
                                    __double2loint(k));
  const double q = div_prepared(a, d, r, z);
  double u = add(mul(C, h.u), q);
  double pu = add(mul(mul(S, h.u), k), mul(C, h.pu));
  if (bend) {
    u = add(u, t[TC_D * n]);
    pu = add(pu, t[TC_DP * n]);
  }
  h.pu = pu;  // a drift's k = 0 leaves it unchanged
  h.u = u;
}

// ---------------------------------------------------------------- one turn
UFO_DEV void pair_observe(const Half &h, bool even, const TrackArgs &a, const PairShared &sh,
                          int k) {
  const int lane = threadIdx.x;
  if (k >= sh.obs_left[lane]) return;
  double *t = sh.obs[lane] + 6 * static_cast<int64_t>(k);
  t[even ? 0 : 2] = h.u;
  t[even ? 1 : 3] = h.pu;
  if (!(a.flags & UFO_TRACK_FIVED)) t[even ? 4 : 5] = a.coords[sh.p[lane] * 6 + (even ? 4 : 5)];
}

// Out-of-line work takes the lane's state from shared memory and leaves it
// there: a call with the interpreter's state in registers would have it spilled
// on the hot path as well (490 bytes at the 128 registers of 16 warps per SM).

// The public ops [first, last) by the one-lane code on the gathered particle
// state; both lanes of a pair compute it and keep their half.  Called by whole
// warps.
template <bool FMA>
__device__ __noinline__ void pair_wide(const TrackArgs &a, PairShared &sh, int first, int last) {
  const int lane = threadIdx.x;
  const bool even = (lane & 1) == 0;
  const int64_t p = sh.p[lane];
  Half h{sh.u[lane], sh.pu[lane]};
  double z = 0.0, dp = 0.0;
  if (p >= 0) {
    z = a.coords[p * 6 + 4];
    dp = a.coords[p * 6 + 5];
  }
  for (int i = first; i < last; ++i) {
    const Op *raw = a.ops + i;
    if (raw->kind == OP_OBSERVE) {
      pair_observe(h, even, a, sh, raw->i0);
      continue;
    }
    const double ou = pair_other(h.u), opu = pair_other(h.pu);
    const P4 r = wide_op<FMA>(even ? h.u : ou, even ? h.pu : opu, even ? ou : h.u,
                              even ? opu : h.pu, z, dp, sh.o[lane], sh.turn[lane], raw,
                              sh.tab[lane] + raw->toff);
    __syncwarp();
    h = {even ? r.x : r.y, even ? r.px : r.py};
  }
  const unsigned nans = __ballot_sync(PAIR_ALL, isnan(h.u) && isnan(h.pu));
  sh.dead[lane] = p == PAIR_NONE || ((nans >> (lane & 30)) & 3u) == 3u;
  sh.u[lane] = h.u;
  sh.pu[lane] = h.pu;
}

UFO_DEV PairOp pair_fetch(const int4 *w) {
  const int4 v = __ldg(w);
  return {v.x, v.y, v.z, v.w};
}

// A particle's first turn in a launch: its coefficient-cache fields.
__device__ __noinline__ void pair_fill(const TrackArgs &a, const PairShared &sh, int group) {
  const int lane = threadIdx.x;
  const bool even = (lane & 1) == 0;
  const int64_t p = sh.p[lane];
  const double dp = p >= 0 ? a.coords[p * 6 + 5] : 0.0, o = sh.o[lane];
  for (const int4 *w = reinterpret_cast<const int4 *>(a.pair_fills);; ++w) {
    const PairOp op = pair_fetch(w);
    const int variant = op.head & 0xff;
    if (variant == PV_SEGMENT) return;  // the end
    const double *c = sh.tab[lane] + op.toff;
    double *t = pair_cache(a, op.a, group);
    if (variant == PV_THICKQ) {
      thick_quad_half(o, op.head, c, t, a.cache_lanes);
    } else if (variant == PV_THICKB) {
      thick_bend_half(o, dp, op.head, c, t, a.cache_lanes);
    } else {  // an edge's factor: tan(e1), or -tan(psi) of the vertical plane
      const double curv = (op.head & PF_ACHRO) ? ld(c) : mul(ld(c), o);
      *t = even ? ((op.head & PF_X) ? ld(c + 1) : 0.0) : -edge_psi_tan(curv, c);
    }
  }
}

// What ends a run of the inner loop, which holds no call: the end of the list;
// a segment to run again; an op without a two-lane form (a segment of its own).
enum : int { PE_END = 0, PE_REDO = 1, PE_WIDE = 2 };

// Run the list from op `pos`, where a segment's header or its WIDE op stands.
// PE_REDO leaves the segment's entry state in h and its public ops in [first,
// last).
// The drift that goes with an op, in the ops' own code: common code after the
// dispatch costs every op some 100 cycles.  Only the strict list has it (FODO
// ring 1,024 particles 67 -> 60 us per turn, thick ring 350 -> 318): FMA programs
// have their drifts merged into the magnets, and the code alone slowed them by 6 %.
template <bool FMA>
UFO_DEV void pair_then(Half &h, const PairCtx &x, const PairOp &op) {
  if (!FMA && (op.head & PF_THEN)) pair_drift<FMA>(h, ld(x.tab + op.b));
}

template <bool FMA>
UFO_DEV int pair_run(Half &h, const PairCtx &x, int &pos, int &first, int &last,
                     const TrackArgs &a, const PairShared &sh, bool any_bad_o) {
  const bool even = x.even;
  const int4 *w = reinterpret_cast<const int4 *>(a.pair_ops) + pos + 1;
  PairOp op = pair_fetch(w - 1), next = pair_fetch(w);
  double c0 = ld(x.tab + op.toff);
  Half in = h;
  bool bad = false;
  first = last = 0;
  for (;;) {
    // two ops ahead, and the first constant of the next one (the list ends in
    // two padding ops)
    const PairOp after = pair_fetch(w + 1);
    const double next_c0 = ld(x.tab + next.toff);
    const double *c = x.tab + op.toff;
    switch (op.head & 0xff) {
      case PV_SEGMENT: {  // the previous segment's test; the entry state of the next
        const bool redo = !x.dead && (bad || nf(h.u) || any_bad_o);
        if (last > first && __any_sync(PAIR_ALL, redo)) {
          h = in;
          pos = static_cast<int>(w - 1 - reinterpret_cast<const int4 *>(a.pair_ops));
          return PE_REDO;
        }
        if (op.b <= op.a) return PE_END;
        first = op.a;
        last = op.b;
        in = h;
        bad = false;
        break;
      }
      case PV_DRIFT:
        pair_drift<FMA>(h, c0);
        pair_then<FMA>(h, x, op);
        break;
      case PV_DRIFT2: {
        const double t = mul(h.pu, c0);
        h.u = FMA ? fma_(t, ld(c + 1), h.u) : add(h.u, mul(t, ld(c + 1)));
        break;
      }
      case PV_DRIFT_DIV:
        h.u = FMA ? fma_(h.pu, ld(c + 3), h.u)
                  : add(h.u, div_markstein(mul(h.pu, c0), ld(c + 1), ld(c + 2), bad));
        break;
      case PV_ALIGN:
        h.u = sub(h.u, (op.head & (even ? PF_X : PF_Y)) ? ld(c + (even ? 0 : 1)) : 0.0);
        pair_then<FMA>(h, x, op);
        break;
      case PV_EDGE: {
        const double curv = mul(c0, (op.head & PF_ACHRO) ? 1.0 : x.o);
        const double T = (op.head & (even ? PF_X : PF_Y))
                             ? flip(ld(c + (even ? 1 : 2)), x.neg ^ static_cast<int>(0x80000000u))
                             : 0.0;
        const double t = mul(h.u, curv);
        h.pu = FMA ? fma_(t, T, h.pu) : add(h.pu, mul(t, T));
        bad = bad || nf(curv);
        pair_then<FMA>(h, x, op);
        break;
      }
      case PV_EDGE_PSI: {
        const double curv = (op.head & PF_ACHRO) ? c0 : mul(c0, x.o);
        const double T = *pair_cache(a, op.a, x.group);
        h.pu = add(h.pu, mul(mul(h.u, curv), T));
        bad = bad || nf(curv);
        pair_then<FMA>(h, x, op);
        break;
      }
      case PV_THICKQ:
        thick_apply(h, pair_cache(a, op.a, x.group), a.cache_lanes, false, bad);
        pair_then<FMA>(h, x, op);
        break;
      case PV_THICKB:
        thick_apply(h, pair_cache(a, op.a, x.group), a.cache_lanes, true, bad);
        pair_then<FMA>(h, x, op);
        break;
      case PV_CIRCLE: {
        const double s = mul(h.u, h.u);
        const double r2 = add(s, pair_other(s));
        if (even && !(r2 < c0)) h.u = __longlong_as_double(0x7ff8000000000000ll);
        break;
      }
      case PV_OBSERVE:
        pair_observe(h, even, a, sh, op.a);
        break;
      case PV_LINEAR: {
        // (x, px) through a 2x2 matrix, (y, py) through a drift: on odd lanes
        // the matrix [0 ly; 0 1] with y itself as the addend of the first row
        const double m11 = even ? c0 : 0.0, m12 = ld(c + (even ? 1 : 4));
        const double m21 = even ? ld(c + 2) : 0.0, m22 = even ? ld(c + 3) : 1.0;
        const double t2 = mul(m22, h.pu);
        const double t1 = fma_(m12, h.pu, even ? 0.0 : h.u);
        h.pu = fma_(m21, h.u, t2);
        h.u = fma_(m11, h.u, t1);
        break;
      }
      case PV_KICK:
        pair_kick<FMA, 0>(h, x, static_cast<uint32_t>(op.b), c,
                          (op.head & PF_ACHRO) ? 1.0 : x.o,
                          c + __popc(static_cast<uint32_t>(op.b)), bad);
        break;
      case PV_KICK + 1:
        pair_kick<FMA, 1>(h, x, 0, c,
                          pair_strength<FMA, 1>(x, c0, (op.head & PF_ACHRO) ? 1.0 : x.o), nullptr,
                          bad);
        break;
      case PV_KICK + 2:
        pair_kick<FMA, 2>(h, x, 0, c,
                          pair_strength<FMA, 2>(x, c0, (op.head & PF_ACHRO) ? 1.0 : x.o), nullptr,
                          bad);
        break;
      case PV_WIDE:
        pos = static_cast<int>(w - reinterpret_cast<const int4 *>(a.pair_ops));
        return PE_WIDE;
#define UFO_PAIR_TEAPOTS(DIV, WEAK)                                                  \
  case PV_TEAPOT + 1 + 4 * DIV + 12 * WEAK:                                          \
    pair_teapot<FMA, 1, FMA ? 0 : DIV, WEAK>(h, x, op, c0, c, bad);                  \
    break;                                                                           \
  case PV_TEAPOT + 2 + 4 * DIV + 12 * WEAK:                                          \
    pair_teapot<FMA, 2, FMA ? 0 : DIV, WEAK>(h, x, op, c0, c, bad);                  \
    break;                                                                           \
  case PV_TEAPOT + 3 + 4 * DIV + 12 * WEAK:                                          \
    pair_teapot<FMA, 3, FMA ? 0 : DIV, WEAK>(h, x, op, c0, c, bad);                  \
    break;
      UFO_PAIR_TEAPOTS(0, 0)
      UFO_PAIR_TEAPOTS(1, 0)
      UFO_PAIR_TEAPOTS(2, 0)
      UFO_PAIR_TEAPOTS(0, 1)
      UFO_PAIR_TEAPOTS(1, 1)
      UFO_PAIR_TEAPOTS(2, 1)
#undef UFO_PAIR_TEAPOTS
      default:  // the general teapots
        pair_teapot<FMA, 0, FMA ? 0 : DIV_ANY, 2>(h, x, op, c0, c, bad);
        break;
    }
    ++w;
    op = next;
    next = after;
    c0 = next_c0;
  }
}

// the cache fields of the lanes with a new particle
UFO_DEV void pair_prepare(PairCtx &x, const TrackArgs &a, PairShared &sh, bool fresh) {
  if (!a.cache) return;
  const int lane = threadIdx.x;
  sh.o[lane] = x.o;
  sh.tab[lane] = x.tab;
  if (fresh) pair_fill(a, sh, x.group);
  __syncwarp();
  x.o = sh.o[lane];
  x.tab = sh.tab[lane];
}

template <bool FMA>
UFO_DEV void pair_turn(Half &h, PairCtx &x, const TrackArgs &a, PairShared &sh, bool any_bad_o) {
  const int lane = threadIdx.x;
  for (int pos = 0, first, last;;) {
    const int event = pair_run<FMA>(h, x, pos, first, last, a, sh, any_bad_o);
    if (event == PE_END) return;
    sh.u[lane] = h.u;
    sh.pu[lane] = h.pu;
    sh.o[lane] = x.o;
    sh.tab[lane] = x.tab;
    pair_wide<FMA>(a, sh, first, last);
    h.u = sh.u[lane];
    h.pu = sh.pu[lane];
    x.o = sh.o[lane];
    x.tab = sh.tab[lane];
    x.dead = sh.dead[lane];
  }
}

UFO_DEV void pair_store(const Half &h, bool even, int64_t p, int turn, const TrackArgs &a) {
  if (a.lost && even) a.lost[p] = static_cast<uint32_t>(turn);
  if (a.final_state) {
    double *f = a.final_state + p * 6;
    f[even ? 0 : 2] = h.u;
    f[even ? 1 : 3] = h.pu;
    f[even ? 4 : 5] = a.coords[p * 6 + (even ? 4 : 5)];
  }
}

UFO_DEV void pair_idle(PairCtx &x, const TrackArgs &a) {
  x.o = 1.0;
  x.bad_o = false;
  x.dead = true;
  x.tab = a.table;
}

// this turn's observation slots of the lane's particle
UFO_DEV void pair_slots(const TrackArgs &a, PairShared &sh, bool idle) {
  const int lane = threadIdx.x, turn = sh.turn[lane];
  sh.obs_left[lane] = 0;
  if (a.tracks && !idle && (turn + 1) % a.every == 0) {
    const int64_t slot = static_cast<int64_t>((turn + 1) / a.every - 1) * a.n_dumps;
    sh.obs[lane] = a.tracks + (sh.p[lane] * a.slots + slot) * 6;
    sh.obs_left[lane] = a.slots - slot;
  }
}

// the loss test (is_lost) of the lane's particle: isnan(x), or |x| > 1, |y| > 1
UFO_DEV bool pair_lost(const Half &h, bool even, int mode) {
  bool out;
  if (mode == UFO_MODE_TRACK)
    out = even && isnan(h.u);
  else
    out = fabs(h.u) > 1. || (even && isnan(h.u));
  return ((__ballot_sync(PAIR_ALL, out) >> (threadIdx.x & 30)) & 3u) != 0u;
}

// The persistent loop of track_kernel with 16 particles per warp: pairs whose
// particle finished refill from the work counter at turn boundaries.
template <bool FMA>
__global__ void __launch_bounds__(32, 16) track_pair_kernel(const __grid_constant__ TrackArgs a) {
  __shared__ PairShared sh;
  const int lane = threadIdx.x;
  const unsigned below = (1u << (lane & 30)) - 1u;  // lanes of the pairs before this one
  PairCtx x{};
  x.even = (lane & 1) == 0;
  x.neg = x.even ? static_cast<int>(0x80000000u) : 0;
  x.group = blockIdx.x;
  pair_idle(x, a);
  sh.p[lane] = PAIR_NONE;
  Half h{0.0, 0.0};
  bool idle = true, exhausted = false;
  bool fresh = false;  // the particle's first turn in this launch: fill the cache
  while (true) {
    const unsigned need = __ballot_sync(PAIR_ALL, idle && !exhausted);
    if (need) {  // both lanes of a pair are in `need` or neither
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(a.queue, static_cast<unsigned long long>(__popc(need) / 2));
      base = __shfl_sync(PAIR_ALL, base, 0);
      if (idle && !exhausted) {
        const int64_t q = static_cast<int64_t>(base) + __popc(need & below) / 2;
        if (q < a.n) {
          const double *c = a.coords + q * 6;
          h.u = c[x.even ? 0 : 2];
          h.pu = c[x.even ? 1 : 3];
          const int target = a.pturns ? a.pturns[q] : a.turns;
          const int64_t sd = a.seed ? static_cast<int64_t>(a.seed[q]) : 0;
          if (sd < 0 || sd >= a.n_seeds) {  // seed outside the table: not tracked
            if (a.lost && x.even) a.lost[q] = 0xffffffffu;
          } else if (target <= 0) {  // nothing to track
            pair_store(h, x.even, q, 0, a);
          } else {
            idle = false;
            x.o = dvd(1., add(c[5], 1.));  // as load_particle: the same bits
            x.bad_o = nf(x.o);
            fresh = true;
            x.dead = false;
            x.tab = a.table + sd * a.stride;
            sh.p[lane] = q;
            sh.turn[lane] = 0;
            sh.target[lane] = target;
          }
        } else {
          exhausted = true;
        }
      }
      continue;  // a pair that got a zero-turn particle needs another
    }
    if (__all_sync(PAIR_ALL, idle)) break;
    if (idle) h.u = h.pu = 0.0;  // idle lanes run along on a finite state
    pair_slots(a, sh, idle);
    const bool any_bad_o = __any_sync(PAIR_ALL, x.bad_o);
    if (__any_sync(PAIR_ALL, fresh)) pair_prepare(x, a, sh, fresh);
    pair_turn<FMA>(h, x, a, sh, any_bad_o);
    const bool lost = pair_lost(h, x.even, a.mode);
    fresh = false;
    if (!idle) {
      const int t = sh.turn[lane] + (lost ? 0 : 1);
      sh.turn[lane] = t;
      if (lost || t >= sh.target[lane]) {
        pair_store(h, x.even, sh.p[lane], t, a);
        sh.p[lane] = PAIR_NONE;
        idle = true;
        pair_idle(x, a);
      }
    }
  }
}

// ---------------------------------------------------------------- time slices
// A launch of more warps' worth of particles than stay resident, all with the
// same turns, ends unevenly: the work counter hands out whole runs, so after
// the first round of resident warps each SM sub-partition holds anything from
// none to four of the rest, and the fullest sets the time.  The sliced kernels
// hand out (slice of turns, group of particles) instead, slice by slice, so a
// sub-partition that is ahead takes more slices and all finish together.
// A group's state rests in the output arrays between its slices: coordinates in
// `final`, turns so far in `lost` with the top bit set while it runs.  Its word
// in `claims` counts the slices handed out and not yet run (low half) and those
// run (high half).  Whoever raises the low half from 0 runs the group; a warp
// that finds it raised leaves the slice to that runner, which goes on until the
// count is back at 0.  So no warp waits for another, and every slice runs once,
// in order.  The last slice runs to the end whatever its length.  A group whose
// particles are all finished keeps its count raised, so its other slices are
// passed over; the last group to finish moves the work counter past the end.
struct Slices {
  unsigned long long *claims;  // [groups], then the groups finished; zero at launch
  int groups, count, turns;    // slices per group, turns per slice
};

// The group of the next slice that this warp may run, or -1 when all are handed
// out; `done`: the group's slices run so far.
UFO_DEV int slice_take(const Slices &s, unsigned long long *queue, int &done) {
  const unsigned all = 0xffffffffu;
  const unsigned long long total = static_cast<unsigned long long>(s.groups) * s.count;
  while (true) {
    unsigned long long t = 0, old = 0;
    if ((threadIdx.x & 31) == 0) {
      t = atomicAdd(queue, 1ull);
      if (t < total) old = atomicAdd(s.claims + t % s.groups, 1ull);
    }
    t = __shfl_sync(all, t, 0);
    old = __shfl_sync(all, old, 0);
    if (t >= total) return -1;
    if ((old & 0xffffffffull) == 0) {
      __threadfence();  // the state that the last runner left
      done = static_cast<int>(old >> 32);
      return static_cast<int>(t % s.groups);
    }
  }
}

// A slice of `group` has run: true when another was handed out meanwhile.
UFO_DEV bool slice_more(const Slices &s, int group, int &done) {
  __threadfence();
  __syncwarp();
  unsigned long long old = 0;
  if ((threadIdx.x & 31) == 0) old = atomicAdd(s.claims + group, (1ull << 32) - 1ull);
  old = __shfl_sync(0xffffffffu, old, 0);
  ++done;
  return (old & 0xffffffffull) > 1;
}

// Every particle of a group has finished.
UFO_DEV void slice_finish(const Slices &s, unsigned long long *queue) {
  if ((threadIdx.x & 31) != 0) return;
  const unsigned long long total = static_cast<unsigned long long>(s.groups) * s.count;
  if (atomicAdd(s.claims + s.groups, 1ull) + 1 == static_cast<unsigned long long>(s.groups))
    atomicMax(queue, total);
}

constexpr uint32_t SLICE_RUNNING = 0x80000000u;

template <bool FMA>
__global__ void __launch_bounds__(32, 16)
    track_pair_sliced(const __grid_constant__ TrackArgs a, const Slices s) {
  __shared__ PairShared sh;
  const int lane = threadIdx.x;
  PairCtx x{};
  x.even = (lane & 1) == 0;
  x.neg = x.even ? static_cast<int>(0x80000000u) : 0;
  int done, group;
  while ((group = slice_take(s, a.queue, done)) >= 0) {
    x.group = group;
    do {
      const int64_t p = static_cast<int64_t>(group) * 16 + lane / 2;
      pair_idle(x, a);
      sh.p[lane] = PAIR_NONE;
      Half h{0.0, 0.0};
      bool idle = true;
      if (p < a.n) {
        const int64_t sd = a.seed ? static_cast<int64_t>(a.seed[p]) : 0;
        const uint32_t at = done ? __ldcg(a.lost + p) : SLICE_RUNNING;
        if (sd < 0 || sd >= a.n_seeds) {  // seed outside the table: not tracked
          if (!done && x.even) a.lost[p] = 0xffffffffu;
        } else if (at & SLICE_RUNNING) {
          idle = false;
          const double *c = (done ? a.final_state : a.coords) + p * 6 + (x.even ? 0 : 2);
          h.u = __ldcg(c);
          h.pu = __ldcg(c + 1);
          x.o = dvd(1., add(a.coords[p * 6 + 5], 1.));  // as load_particle: the same bits
          x.bad_o = nf(x.o);
          x.dead = false;
          x.tab = a.table + sd * a.stride;
          sh.p[lane] = p;
          sh.turn[lane] = static_cast<int>(at & ~SLICE_RUNNING);
        }
      }
      const bool mine = !idle;
      const bool last = done == s.count - 1;
      if (!done && __any_sync(PAIR_ALL, !idle)) pair_prepare(x, a, sh, !idle);
      for (int k = 0; (last || k < s.turns) && __any_sync(PAIR_ALL, !idle); ++k) {
        if (!mine) h.u = h.pu = 0.0;  // idle lanes run along on a finite state
        if (!idle && sh.turn[lane] >= a.turns) idle = true;  // nothing to track
        if (__all_sync(PAIR_ALL, idle)) break;
        pair_slots(a, sh, idle);
        const Half before = h;
        pair_turn<FMA>(h, x, a, sh, __any_sync(PAIR_ALL, x.bad_o));
        const bool lost = pair_lost(h, x.even, a.mode);
        if (idle) {
          h = before;  // a finished particle keeps its state
        } else {
          const int t = sh.turn[lane] + (lost ? 0 : 1);
          sh.turn[lane] = t;
          if (lost || t >= a.turns) {
            idle = true;
            x.dead = true;
          }
        }
      }
      if (mine) {
        double *f = a.final_state + p * 6;
        f[x.even ? 0 : 2] = h.u;
        f[x.even ? 1 : 3] = h.pu;
        if (!done) f[x.even ? 4 : 5] = a.coords[p * 6 + (x.even ? 4 : 5)];
        if (x.even)
          a.lost[p] = static_cast<uint32_t>(sh.turn[lane]) | (idle ? 0u : SLICE_RUNNING);
      }
      __syncwarp();
      if (__all_sync(PAIR_ALL, idle)) {
        slice_finish(s, a.queue);
        break;
      }
    } while (slice_more(s, group, done));
  }
}

// ---------------------------------------------------------------- closed orbit
// The search of co_amoeba_kernel (one thread per orbit) with four trial points
// of each step tracked at once on four lane pairs: the reflection, and what may
// follow it -- the expansion and the contraction if the reflection is kept, the
// contraction if it is not.  A warp instruction costs the same however many
// lanes use it, so the step takes one turn instead of the one to two dependent
// ones of the sequential search; the trials it would not have made are dropped,
// and the simplex goes through the same values.  A shrink (four more trials)
// and an expansion of an unkept reflection (equal residuals) take a second turn.
// Measured, 200 steps, whole calls: 12 orbits of the thick 768-element ring
// 735 ms -> 67 ms.
struct OrbitShared {
  double sx[4][5][4], y[4][5], psum[4][4];  // per orbit of the warp
};

// Residual of the trial in (t0, t1) of every lane pair, on all its lanes.  Out
// of line: the interpreter's registers are its own.
__device__ __noinline__ double orbit_residual(double t0, double t1, const double *tab,
                                              const TrackArgs &a, PairShared &sh) {
  PairCtx x;
  x.even = (threadIdx.x & 1) == 0;
  x.neg = x.even ? static_cast<int>(0x80000000u) : 0;
  x.o = 1.0;
  x.tab = tab;
  x.group = blockIdx.x;
  x.dead = x.bad_o = false;
  Half h{t0, t1};
  pair_turn<false>(h, x, a, sh, false);
  const double d0 = sub(t0, h.u), d1 = sub(t1, h.pu);
  const double s0 = mul(d0, d0), s1 = mul(d1, d1);
  const double o0 = pair_other(s0), o1 = pair_other(s1);
  return add(add(add(pick(x.even, s0, o0), pick(x.even, s1, o1)), pick(x.even, o0, s0)),
             pick(x.even, o1, s1));
}

__global__ void __launch_bounds__(32, 16)
    co_pair_kernel(const __grid_constant__ TrackArgs a, const double *start, double *orbits,
                   int iterations, int per_warp) {
  __shared__ PairShared sh;
  __shared__ OrbitShared os;
  const int lane = threadIdx.x, g = lane >> 3, j = (lane >> 1) & 3;
  const int c0 = (lane & 1) * 2, c1 = c0 + 1;  // this lane's coordinates
  double(*sx)[4] = os.sx[g], *y = os.y[g], *psum = os.psum[g];
  auto group = [&](double v, int pair) { return __shfl_sync(PAIR_ALL, v, 8 * g + 2 * pair); };
  PairCtx x{};
  x.even = (lane & 1) == 0;
  x.neg = x.even ? static_cast<int>(0x80000000u) : 0;
  x.group = blockIdx.x;
  sh.turn[lane] = 0;
  sh.obs_left[lane] = 0;
  const int64_t groups = (a.n + per_warp - 1) / per_warp;
  for (int64_t w = blockIdx.x; w < groups; w += gridDim.x) {
    const int64_t p = w * per_warp + g;
    const bool have = g < per_warp && p < a.n;
    const int64_t sd = have && a.seed ? static_cast<int64_t>(a.seed[p]) : 0;
    const bool in_table = sd >= 0 && sd < a.n_seeds;
    pair_idle(x, a);
    sh.p[lane] = PAIR_ORBIT;
    if (in_table) x.tab = a.table + sd * a.stride;
    pair_prepare(x, a, sh, true);
    // the simplex {v, v + 1e-4 e_k} and its residuals
    if (j == 0)
      for (int i = 0; i < 5; ++i) {
        for (int c = c0; c <= c1; ++c) sx[i][c] = have ? start[4 * p + c] : 0.0;
        for (int c = c0; c <= c1; ++c)
          if (i == c + 1) sx[i][c] = add(sx[i][c], 1e-4);
      }
    __syncwarp();
    const double r03 = orbit_residual(sx[j][c0], sx[j][c1], x.tab, a, sh);
    const double r4 = orbit_residual(sx[4][c0], sx[4][c1], x.tab, a, sh);
    if ((lane & 1) == 0) y[j] = r03;
    if ((lane & 7) == 0) y[4] = r4;
    __syncwarp();
    if (j == 0)
      for (int c = c0; c <= c1; ++c) {
        double v = 0.0;
        for (int i = 0; i < 5; ++i) v = add(v, sx[i][c]);
        psum[c] = v;
      }
    __syncwarp();
    int iter = 0, ilo = 0;
    bool done = !have || !in_table;
    while (true) {
      int ihi = 1, inhi = 2;
      if (!done) {  // uniform over the orbit's lanes: they read the same residuals
        ilo = 1;
        if (!(y[1] > y[2])) {
          inhi = 1;
          ihi = 2;
        }
        for (int i = 0; i < 5; ++i) {
          if (y[i] < y[ilo]) ilo = i;
          if (y[i] > y[ihi]) {
            inhi = ihi;
            ihi = i;
          } else if (y[i] > y[inhi] && i != ihi) {
            inhi = i;
          }
        }
        done = iter >= iterations;
      }
      if (__all_sync(PAIR_ALL, done)) break;
      // the trials (co_try): t = psum f1 - v_hi f2, f1 = (1 - fac) / 4, f2 = f1 - fac
      auto trial = [](double ps, double v, double fac) {
        const double f1 = dvd(sub(1.0, fac), 4.0);
        return sub(mul(ps, f1), mul(v, sub(f1, fac)));
      };
      const double h0 = sx[ihi][c0], h1 = sx[ihi][c1], p0 = psum[c0], p1 = psum[c1];
      const double q0 = trial(p0, h0, -1.0), q1 = trial(p1, h1, -1.0);  // reflection
      const double k0 = add(p0, sub(q0, h0)), k1 = add(p1, sub(q1, h1));  // psum if kept
      const double fac = j == 1 ? 2.0 : 0.5;
      const bool kept_base = j == 1 || j == 2;
      const double e0 = trial(kept_base ? k0 : p0, kept_base ? q0 : h0, fac);
      const double e1 = trial(kept_base ? k1 : p1, kept_base ? q1 : h1, fac);
      const double t0 = j == 0 ? q0 : e0, t1 = j == 0 ? q1 : e1;
      const double r = orbit_residual(t0, t1, x.tab, a, sh);
      const double yr = group(r, 0), ye = group(r, 1), yck = group(r, 2), ycn = group(r, 3);
      const double yhi = y[ihi], ylo = y[ilo], ynext = y[inhi];
      const bool kept = yr < yhi;
      const double ybase = kept ? yr : yhi;            // y[ihi] after the reflection
      // y[ilo], y[inhi] after it (they may be the same vertex as ihi)
      const double ylo2 = ilo == ihi ? ybase : ylo, ynext2 = inhi == ihi ? ybase : ynext;
      const bool expand = yr <= ylo2, contract = !expand && yr >= ynext2;
      // the second trial's point and residual, where it is among the four
      const double y2 = expand ? ye : kept ? yck : ycn;
      const int src = 8 * g + 2 * (expand ? 1 : kept ? 2 : 3) + (lane & 1);
      double s0 = __shfl_sync(PAIR_ALL, t0, src), s1 = __shfl_sync(PAIR_ALL, t1, src);
      const bool second = expand || contract;
      double y2v = y2;
      const bool odd_expand = expand && !kept;  // not among them
      const bool shrink = contract && y2 >= ybase;
      __syncwarp();
      if (!done && j == 0 && kept) {
        sx[ihi][c0] = q0;
        sx[ihi][c1] = q1;
        psum[c0] = k0;
        psum[c1] = k1;
        if (x.even) y[ihi] = yr;
      }
      __syncwarp();
      const bool more = !done && (odd_expand || shrink);
      if (__any_sync(PAIR_ALL, more)) {
        // vertex of this pair's shrink trial: the j-th that is not ilo
        const int v = j < ilo ? j : j + 1;
        double m0 = mul(add(sx[v][c0], sx[ilo][c0]), 0.5);
        double m1 = mul(add(sx[v][c1], sx[ilo][c1]), 0.5);
        if (odd_expand) {
          m0 = trial(psum[c0], sx[ihi][c0], 2.0);
          m1 = trial(psum[c1], sx[ihi][c1], 2.0);
        }
        const double rm = orbit_residual(m0, m1, x.tab, a, sh);
        const double rm0 = group(rm, 0);
        const double w0 = __shfl_sync(PAIR_ALL, m0, 8 * g + (lane & 1));
        const double w1 = __shfl_sync(PAIR_ALL, m1, 8 * g + (lane & 1));
        if (odd_expand) {
          y2v = rm0;
          s0 = w0;
          s1 = w1;
        }
        __syncwarp();
        if (more && shrink) {
          sx[v][c0] = m0;
          sx[v][c1] = m1;
          if (x.even) y[v] = rm;
        }
        __syncwarp();
        if (more && shrink && j == 0)
          for (int c = c0; c <= c1; ++c) {
            double v2 = 0.0;
            for (int i = 0; i < 5; ++i) v2 = add(v2, sx[i][c]);
            psum[c] = v2;
          }
      }
      ++iter;
      if (!done && shrink) iter += 4;
      if (!done && second && !shrink && y2v < ybase && j == 0) {  // co_try keeps the trial
        psum[c0] = add(psum[c0], sub(s0, sx[ihi][c0]));
        psum[c1] = add(psum[c1], sub(s1, sx[ihi][c1]));
        sx[ihi][c0] = s0;
        sx[ihi][c1] = s1;
        if (x.even) y[ihi] = y2v;
      }
      __syncwarp();
    }
    if (have && j == 0) {
      const double bad = __longlong_as_double(0x7ff8000000000000ll);
      orbits[4 * p + c0] = in_table ? sx[ilo][c0] : bad;
      orbits[4 * p + c1] = in_table ? sx[ilo][c1] : bad;
    }
    __syncwarp();
  }
}

}  // namespace ufo
