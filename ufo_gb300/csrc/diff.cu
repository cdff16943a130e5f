// diff.cu -- tangent map and hand-written adjoint of the one-turn map.
//
// Differentiation runs on its own opcode list (built by ufo_gb300/diff.py from
// the compiled line): drifts, teapot elements, thin kicks, alignments, edges
// (with a fringe angle that may depend on dp) and the exact thick quadrupole
// and sector-bend maps.  Every kick of the reference (ufo/methods.py:45-76, the
// Horner scheme) is the complex polynomial
//     S(z) = o * sum_n (a_n + i b_n) z^n,   z = x + i y,
//     a_n = kn_n / n!,  b_n = ks_n / n!,
//     px -= Re S,   py += Im S,
// so its derivatives follow from S' and S'' (Cauchy-Riemann); one Horner pass
// gives S, S' and S''/2 together.  A teapot slice is kick, weak focusing
// (px -= W x), drift.  Element strengths enter linearly: one parameter per
// element scales coefficient `pm`; the table carries dK/dk / pm! and
// dK/dk / (pm-1)! for the S and S' terms.
//
// diff_forward: z (and optionally the 4x4 tangent T = dz/dz0) through `turns`
//   turns, writing the state (and T) every `ck` turns as checkpoints.
// Reverse pass, given the output cotangents zbar (and Tbar), over the
//   checkpoint segments from the last to the first:
//   * plain (multi-turn) mode: diff_tape re-tracks G segments at once
//     (G x J independent jobs: the segments only need their checkpoints) onto
//     a "rich" tape holding x, y and S'(z) at every kick; diff_reverse_plain
//     then walks those G segments backwards, job by job, with the cheap
//     reverse kick the stored S' allows.  The cotangent state is carried in
//     zbar0 from one group of segments to the next.
//   * tangent mode (optics, one turn): diff_reverse re-tracks each segment
//     onto a tape of x, y and the x/y rows of T and reverses it in one kernel.
//   Both accumulate the cotangent of the start state and of every element
//   parameter.
// Per-job buffers that grow with the work (checkpoints, tape, parameter
// cotangents) are laid out job-fastest, so a warp's 32 jobs touch 32
// consecutive doubles.  Arithmetic is FP64 with fused multiply-adds (gradients
// need FP64 accuracy, not the reference's rounding).  One thread per job.
#include <cuda_runtime.h>

#include <cstdint>

namespace ufo_diff {

enum : int { D_NOP = 0, D_DRIFT, D_TEAPOT, D_KICK, D_ALIGN, D_EDGE, D_THICK };
constexpr int KHDR = 6;   // kick constants: Lo, Li, W, g0, g1, Lx (exit), then a[M], b[M]
constexpr int DT_BEND = 1;      // D_THICK flag: sector bend (h^2 focusing, dispersion term)
constexpr int DE_RTPSI = 1;     // D_EDGE flag: fringe angle psi depends on the job's dp
constexpr int THICK_SLOTS = 2;  // tape slots of a thick element per turn

struct DOp {
  int kind, flags, toff, N, M, pslot, pm, achro;
};

struct DiffArgs {
  const DOp *ops;
  int n_ops;
  const double *tab;      // constants, [n_seeds][tab_stride]
  const int32_t *seed;    // [job] constant-table row, or null (row 0)
  int64_t tab_stride;
  int n_params;
  int kicks_per_turn;
  int n_jobs;
  const double *z0;       // [job][4]
  const double *o;        // [job] 1/(1+dp)
  int turns, ck;          // turns, checkpoint interval
  int tangent;            // propagate T
  double *ckpt;           // [turns/ck + 1][20][job]
  double *zT;             // [job][20] final state (+T)
  const double *zbar;     // [job][4] output cotangents
  const double *Tbar;     // [job][16] (tangent only)
  double *tape;           // [G*ck][warp][kicks_per_turn][nf][lane], nf = 10 (tangent) or 4
  double *zbar0;          // [job][4] cotangent of the start state
  double *pbar;           // [n_params][job]
};

struct St {
  double x, px, y, py;
  double T[16];  // rows x, px, y, py; columns = start coordinates
};

// S(z)/o, S'(z)/o and S''(z)/(2o) by one Horner pass over the power series
// (ND = highest derivative wanted)
template <int ND>
__device__ __forceinline__ void series(const double *__restrict__ a, int M, double x, double y,
                                       double &s0r, double &s0i, double &s1r, double &s1i,
                                       double &s2r, double &s2i) {
  const double *b = a + M;
  s0r = __ldg(a + M - 1);
  s0i = __ldg(b + M - 1);
  s1r = s1i = s2r = s2i = 0.0;
  for (int n = M - 2; n >= 0; --n) {  // x's product first, in both components
    if (ND >= 2) {
      const double tr = fma(-s2i, y, fma(s2r, x, s1r));
      s2i = fma(s2r, y, fma(s2i, x, s1i));
      s2r = tr;
    }
    if (ND >= 1) {
      const double tr = fma(-s1i, y, fma(s1r, x, s0r));
      s1i = fma(s1r, y, fma(s1i, x, s0i));
      s1r = tr;
    }
    const double tr = fma(-s0i, y, fma(s0r, x, __ldg(a + n)));
    s0i = fma(s0r, y, fma(s0i, x, __ldg(b + n)));
    s0r = tr;
  }
}

__device__ __forceinline__ void fwd_drift(St &s, double L, bool tangent) {
  s.x = fma(s.px, L, s.x);
  s.y = fma(s.py, L, s.y);
  if (tangent)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      s.T[j] = fma(s.T[4 + j], L, s.T[j]);
      s.T[8 + j] = fma(s.T[12 + j], L, s.T[8 + j]);
    }
}

__device__ __forceinline__ void fwd_weak(St &s, double W, bool tangent) {
  s.px = fma(-W, s.x, s.px);
  if (tangent)
#pragma unroll
    for (int j = 0; j < 4; ++j) s.T[4 + j] = fma(-W, s.T[j], s.T[4 + j]);
}

__device__ __forceinline__ void fwd_kick(St &s, const double *a, int M, double o, bool tangent) {
  double sr, si, ar, ai, br, bi;
  if (tangent) {
    series<1>(a, M, s.x, s.y, sr, si, ar, ai, br, bi);
    ar *= o;
    ai *= o;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const double dx = s.T[j], dy = s.T[8 + j];
      s.T[4 + j] = fma(ai, dy, fma(-ar, dx, s.T[4 + j]));
      s.T[12 + j] = fma(ai, dx, fma(ar, dy, s.T[12 + j]));
    }
  } else {
    series<0>(a, M, s.x, s.y, sr, si, ar, ai, br, bi);
  }
  s.px = fma(-o, sr, s.px);
  s.py = fma(o, si, s.py);
}

// The exact thick maps (ufo/methods.py:99-134 quadrupole, :136-196 sector
// bend) per plane: q' = C q + Sw pq + disp D1, pq' = -K Sw q + C pq + disp Sw,
// with the plane's focusing strength K (q'' = -K q; K_x = o (k1 + h^2),
// K_y = -o k1, o = 1 when achromatic), C = cos(sqrt(K) L) (cosh for K < 0),
// Sw = sin(sqrt(K) L) / sqrt(K) (sinh), D1 = (1 - C) / K, and the bend's
// horizontal dispersion disp = dp h o.  Power series in u = K L^2 for
// |u| < 1 (no cancellation near K = 0), closed forms above; the derivatives
// in K are dC = -L Sw / 2, dSw = (L C - Sw) / (2K), dD1 = (L Sw / 2 - D1) / K.
// Same arithmetic as ufo_gb300/diff.py: thick_functions.
template <bool DERIV>
__device__ __forceinline__ void thick_fns(double K, double L, double &C, double &Sw, double &D1,
                                          double &dC, double &dSw, double &dD1) {
  const double u = K * L * L;
  if (fabs(u) < 1.0) {
    // Horner over n = 13..0 of (-u)^n / (2n)!, / (2n+1)!, / (2n+2)! (and
    // n (-1)^n u^(n-1) / (2n+1)!, / (2n+2)! for the derivatives)
    double c = 0.0, sw = 0.0, d1 = 0.0, ds = 0.0, dd = 0.0;
    double f2n = 1.0;  // (2n)! for n = 13, built downwards from the top
#pragma unroll
    for (int k = 1; k <= 26; ++k) f2n *= k;
#pragma unroll
    for (int n = 13; n >= 0; --n) {
      const double sg = (n & 1) ? -1.0 : 1.0;
      const double i0 = sg / f2n;                              // 1/(2n)!
      const double i1 = i0 / (2 * n + 1);                      // 1/(2n+1)!
      const double i2 = i1 / (2 * n + 2);                      // 1/(2n+2)!
      c = fma(c, u, i0);
      sw = fma(sw, u, i1);
      d1 = fma(d1, u, i2);
      if (DERIV && n >= 1) {
        ds = fma(ds, u, n * i1);
        dd = fma(dd, u, n * i2);
      }
      if (n > 0) f2n /= static_cast<double>((2 * n) * (2 * n - 1));
    }
    C = c;
    Sw = L * sw;
    D1 = L * L * d1;
    if (DERIV) {
      dSw = L * L * L * ds;
      dD1 = L * L * L * L * dd;
    }
  } else {
    const double w = sqrt(fabs(K));
    if (K > 0) {
      double sn, cs;
      sincos(w * L, &sn, &cs);
      C = cs;
      Sw = sn / w;
    } else {
      C = cosh(w * L);
      Sw = sinh(w * L) / w;
    }
    D1 = (1.0 - C) / K;
    if (DERIV) {
      dSw = (L * C - Sw) / (2.0 * K);
      dD1 = (0.5 * L * Sw - D1) / K;
    }
  }
  if (DERIV) dC = -0.5 * L * Sw;
}

// one plane of a thick element forward; with `tangent` the plane's two
// tangent rows tq, tp (4 columns each) too
__device__ __forceinline__ void thick_plane_fwd(double &q, double &pq, double *tq, double *tp,
                                                double K, double L, double disp, bool tangent) {
  double C, Sw, D1, dC, dSw, dD1;
  thick_fns<false>(K, L, C, Sw, D1, dC, dSw, dD1);
  const double A = -K * Sw;
  const double q0 = q;
  q = fma(C, q0, fma(Sw, pq, disp * D1));
  pq = fma(A, q0, fma(C, pq, disp * Sw));
  if (tangent)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const double t = tq[j];
      tq[j] = fma(C, t, Sw * tp[j]);
      tp[j] = fma(A, t, C * tp[j]);
    }
}

// reverse of one plane of a thick element at the entry state (q, pq) and
// entry tangent rows (tq, tp; tangent mode): cotangents (qb, pqb) and the
// tangent-row cotangents (bq, bp) are mapped back through the transposed map;
// returns the cotangent of the plane's focusing strength K
__device__ __forceinline__ double thick_plane_rev(double &qb, double &pqb, double *bq, double *bp,
                                                  const double *tq, const double *tp, double q,
                                                  double pq, double K, double L, double disp,
                                                  bool tangent) {
  double C, Sw, D1, dC, dSw, dD1;
  thick_fns<true>(K, L, C, Sw, D1, dC, dSw, dD1);
  const double A = -K * Sw, dA = fma(-K, dSw, -Sw);
  double Kb = fma(qb, fma(dC, q, fma(dSw, pq, disp * dD1)),
                  pqb * fma(dA, q, fma(dC, pq, disp * dSw)));
  if (tangent) {
    double kt[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      kt[j] = fma(bq[j], fma(dC, tq[j], dSw * tp[j]), bp[j] * fma(dA, tq[j], dC * tp[j]));
      const double b = bq[j];
      bq[j] = fma(C, b, A * bp[j]);
      bp[j] = fma(Sw, b, C * bp[j]);
    }
    Kb += (kt[0] + kt[1]) + (kt[2] + kt[3]);
  }
  const double b = qb;
  qb = fma(C, b, A * pqb);
  pqb = fma(Sw, b, C * pqb);
  return Kb;
}

// tan of an edge's vertical angle: constant, or the fringe-field psi of the
// job's curvature (psi = e - 2 curv fint' / cos(e) (1 + sin^2 e), SLAC-75)
__device__ __forceinline__ double edge_t2(int flags, const double *c, double curv) {
  if (flags & DE_RTPSI)
    return tan(__ldg(c + 2) - 2.0 * curv * __ldg(c + 3) / __ldg(c + 4) * __ldg(c + 5));
  return __ldg(c + 2);
}

// tape slot of field f of kick k in turn tt (counted from the start of the
// group of segments being taped); rich-tape fields: x, y, Re S', Im S'.
// Warp-blocked: one warp's values for one turn are a contiguous run (the
// reverse walk prefetches them in bulk), a kick's field a 256-byte line.
constexpr int TLANES = 32;
__device__ __forceinline__ int64_t tidx(const DiffArgs &a, int tt, int k, int f, int nf, int j) {
  const int64_t warps = (a.n_jobs + TLANES - 1) / TLANES;
  return (((static_cast<int64_t>(tt) * warps + j / TLANES) * a.kicks_per_turn + k) * nf + f) *
             TLANES + (j % TLANES);
}

// one turn forward (one lane per job); with `tape` (tangent mode) x, y and
// the x/y rows of T at every kick are recorded as turn `tt`
__device__ void turn_forward(St &s, const DiffArgs &a, const double *T0, double o, bool tangent,
                             int j, int tt, bool tape) {
  int kidx = 0;
  const int nf = 10;
  for (int i = 0; i < a.n_ops; ++i) {
    const DOp op = a.ops[i];
    const double *c = T0 + op.toff;
    const double oo = op.achro ? 1.0 : o;
    switch (op.kind) {
      case D_DRIFT:
        fwd_drift(s, __ldg(c), tangent);
        break;
      case D_ALIGN:
        s.x -= __ldg(c);
        s.y -= __ldg(c + 1);
        break;
      case D_EDGE: {
        const double curv = __ldg(c) * oo, e1 = __ldg(c + 1), e2 = edge_t2(op.flags, c, curv);
        const double x0 = s.x, y0 = s.y;
        s.px = fma(x0 * curv, e1, s.px);
        s.py = fma(-(y0 * curv), e2, s.py);
        if (tangent)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            s.T[4 + q] = fma(s.T[q] * curv, e1, s.T[4 + q]);
            s.T[12 + q] = fma(-(s.T[8 + q] * curv), e2, s.T[12 + q]);
          }
        break;
      }
      case D_KICK:
      case D_TEAPOT: {
        const bool tp = op.kind == D_TEAPOT;
        const int N = tp ? op.N : 1;
        const double Lo = __ldg(c), Li = __ldg(c + 1), W = __ldg(c + 2), Lx = __ldg(c + 5);
        if (tp) fwd_drift(s, Lo, tangent);
        for (int sl = 0; sl < N; ++sl) {
          const int k = kidx++;
          if (tape) {  // tangent tape (the plain rich tape is written by the pair kernels)
            double *t = a.tape;
            t[tidx(a, tt, k, 0, nf, j)] = s.x;
            t[tidx(a, tt, k, 1, nf, j)] = s.y;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              t[tidx(a, tt, k, 2 + q, nf, j)] = s.T[q];
              t[tidx(a, tt, k, 6 + q, nf, j)] = s.T[8 + q];
            }
          }
          fwd_kick(s, c + KHDR, op.M, oo, tangent);
          if (tp && W != 0.0) fwd_weak(s, W, tangent);
          if (tp) fwd_drift(s, sl < N - 1 ? Li : Lx, tangent);
        }
        break;
      }
      case D_THICK: {
        const double L = __ldg(c), k1 = __ldg(c + 1), h = __ldg(c + 2);
        const int k = kidx;
        kidx += THICK_SLOTS;
        if (tape) {  // entry state and tangent: x, y, T rows x, y | px, py, T rows px, py
          double *t = a.tape;
          t[tidx(a, tt, k, 0, nf, j)] = s.x;
          t[tidx(a, tt, k, 1, nf, j)] = s.y;
          t[tidx(a, tt, k + 1, 0, nf, j)] = s.px;
          t[tidx(a, tt, k + 1, 1, nf, j)] = s.py;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            t[tidx(a, tt, k, 2 + q, nf, j)] = s.T[q];
            t[tidx(a, tt, k, 6 + q, nf, j)] = s.T[8 + q];
            t[tidx(a, tt, k + 1, 2 + q, nf, j)] = s.T[4 + q];
            t[tidx(a, tt, k + 1, 6 + q, nf, j)] = s.T[12 + q];
          }
        }
        const double disp = (op.flags & DT_BEND) ? (1.0 / o - 1.0) * h * oo : 0.0;
        thick_plane_fwd(s.x, s.px, s.T, s.T + 4, oo * fma(h, h, k1), L, disp, tangent);
        thick_plane_fwd(s.y, s.py, s.T + 8, s.T + 12, -oo * k1, L, 0.0, tangent);
        break;
      }
      default:
        break;
    }
  }
}

struct Bar {
  double x, px, y, py;
  double T[16];
};

__device__ __forceinline__ void rev_drift(Bar &b, double L, bool tangent) {
  b.px = fma(b.x, L, b.px);
  b.py = fma(b.y, L, b.py);
  if (tangent)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      b.T[4 + j] = fma(b.T[j], L, b.T[4 + j]);
      b.T[12 + j] = fma(b.T[8 + j], L, b.T[12 + j]);
    }
}

__device__ __forceinline__ void rev_weak(Bar &b, double W, bool tangent) {
  b.x = fma(-W, b.px, b.x);
  if (tangent)
#pragma unroll
    for (int j = 0; j < 4; ++j) b.T[j] = fma(-W, b.T[4 + j], b.T[j]);
}

// z^n for small n
__device__ __forceinline__ void zpow(double x, double y, int n, double &zr, double &zi) {
  zr = 1.0;
  zi = 0.0;
  for (int k = 0; k < n; ++k) {
    const double tr = fma(zr, x, -zi * y);
    zi = fma(zr, y, zi * x);
    zr = tr;
  }
}

// reverse of one kick at the taped (x, y) [and tangent rows]; adds the
// cotangents of the op's parameter coefficient to g0 (S term, weight z^pm) and
// g1 (S' term, weight z^(pm-1)), both still to be scaled by dK/dk / n!
__device__ __forceinline__ void rev_kick(Bar &b, const DiffArgs &a, int tt, int k, int j,
                                         const double *co, int M, double o, bool tangent, int pm,
                                         double &g0, double &g1) {
  const int nf = 10;
  const double x = a.tape[tidx(a, tt, k, 0, nf, j)], y = a.tape[tidx(a, tt, k, 1, nf, j)];
  double s0r, s0i, a1, b1, a2, b2;
  series<2>(co, M, x, y, s0r, s0i, a1, b1, a2, b2);
  a1 *= o;
  b1 *= o;
  // state: px' = px - Re S, py' = py + Im S
  double xb = fma(b.py, b1, fma(-b.px, a1, b.x));
  double yb = fma(b.px, b1, fma(b.py, a1, b.y));
  if (pm >= 0) {  // dS/dc = o z^pm / pm!
    double zr, zi;
    zpow(x, y, pm, zr, zi);
    g0 += o * fma(-b.px, zr, b.py * zi);
  }
  if (tangent) {
    a2 *= 2.0 * o;
    b2 *= 2.0 * o;
    double At[4], Bt[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const double dx = a.tape[tidx(a, tt, k, 2 + q, nf, j)];
      const double dy = a.tape[tidx(a, tt, k, 6 + q, nf, j)];
      const double pxb = b.T[4 + q], pyb = b.T[12 + q];
      // T_px -= a1 dx - b1 dy ; T_py += b1 dx + a1 dy
      b.T[q] = fma(pyb, b1, fma(-pxb, a1, b.T[q]));
      b.T[8 + q] = fma(pxb, b1, fma(pyb, a1, b.T[8 + q]));
      At[q] = fma(-pxb, dx, pyb * dy);
      Bt[q] = fma(pyb, dx, pxb * dy);
    }
    // summed in the order of the eight-lane form's butterfly
    const double Ab = (At[0] + At[1]) + (At[2] + At[3]);
    const double Bb = (Bt[0] + Bt[1]) + (Bt[2] + Bt[3]);
    // a1 + i b1 = S'(z): d/dx = S'' , d/dy = i S''
    xb = fma(Bb, b2, fma(Ab, a2, xb));
    yb = fma(Ab, -b2, fma(Bb, a2, yb));
    if (pm >= 1) {  // dS'/dc = o z^(pm-1) / (pm-1)!
      double zr, zi;
      zpow(x, y, pm - 1, zr, zi);
      g1 += o * fma(Ab, zr, Bb * zi);
    }
  }
  b.x = xb;
  b.y = yb;
}

// reverse of turn `tt` of the segment from its tape; accumulates parameter
// cotangents
__device__ void turn_reverse(Bar &b, const DiffArgs &a, const double *T0, double o, bool tangent,
                             int j, int tt) {
  int kidx = a.kicks_per_turn;
  for (int i = a.n_ops - 1; i >= 0; --i) {
    const DOp op = a.ops[i];
    const double *c = T0 + op.toff;
    const double oo = op.achro ? 1.0 : o;
    switch (op.kind) {
      case D_DRIFT:
        rev_drift(b, __ldg(c), tangent);
        break;
      case D_ALIGN:
        break;  // translation: cotangents unchanged
      case D_EDGE: {
        const double curv = __ldg(c) * oo, e1 = __ldg(c + 1), e2 = edge_t2(op.flags, c, curv);
        b.x = fma(b.px * curv, e1, b.x);
        b.y = fma(-(b.py * curv), e2, b.y);
        if (tangent)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            b.T[q] = fma(b.T[4 + q] * curv, e1, b.T[q]);
            b.T[8 + q] = fma(-(b.T[12 + q] * curv), e2, b.T[8 + q]);
          }
        break;
      }
      case D_KICK:
      case D_TEAPOT: {
        const bool tp = op.kind == D_TEAPOT;
        const int N = tp ? op.N : 1;
        const double Lo = __ldg(c), Li = __ldg(c + 1), W = __ldg(c + 2), Lx = __ldg(c + 5);
        const int pm = op.pslot >= 0 ? op.pm : -1;
        double g0 = 0.0, g1 = 0.0;
        for (int sl = N - 1; sl >= 0; --sl) {
          if (tp) rev_drift(b, sl < N - 1 ? Li : Lx, tangent);
          if (tp && W != 0.0) rev_weak(b, W, tangent);
          rev_kick(b, a, tt, --kidx, j, c + KHDR, op.M, oo, tangent, pm, g0, g1);
        }
        if (tp) rev_drift(b, Lo, tangent);
        if (op.pslot >= 0) {
          double &p = a.pbar[static_cast<int64_t>(op.pslot) * a.n_jobs + j];
          p = fma(g0, __ldg(c + 3), fma(g1, __ldg(c + 4), p));
        }
        break;
      }
      case D_THICK: {
        const double L = __ldg(c), k1 = __ldg(c + 1), h = __ldg(c + 2);
        kidx -= THICK_SLOTS;
        const int nf = 10;
        const double *t = a.tape;
        double ex[4], epx[4], ey[4], epy[4];  // entry tangent rows
        if (tangent)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            ex[q] = t[tidx(a, tt, kidx, 2 + q, nf, j)];
            ey[q] = t[tidx(a, tt, kidx, 6 + q, nf, j)];
            epx[q] = t[tidx(a, tt, kidx + 1, 2 + q, nf, j)];
            epy[q] = t[tidx(a, tt, kidx + 1, 6 + q, nf, j)];
          }
        const double x = t[tidx(a, tt, kidx, 0, nf, j)], y = t[tidx(a, tt, kidx, 1, nf, j)];
        const double px = t[tidx(a, tt, kidx + 1, 0, nf, j)];
        const double py = t[tidx(a, tt, kidx + 1, 1, nf, j)];
        const double disp = (op.flags & DT_BEND) ? (1.0 / o - 1.0) * h * oo : 0.0;
        const double kbx = thick_plane_rev(b.x, b.px, b.T, b.T + 4, ex, epx, x, px,
                                           oo * fma(h, h, k1), L, disp, tangent);
        const double kby = thick_plane_rev(b.y, b.py, b.T + 8, b.T + 12, ey, epy, y, py, -oo * k1,
                                           L, 0.0, tangent);
        if (op.pslot >= 0) {  // dK_x/dk1 = o, dK_y/dk1 = -o
          double &p = a.pbar[static_cast<int64_t>(op.pslot) * a.n_jobs + j];
          p = fma(oo, kbx - kby, p);
        }
        break;
      }
      default:
        break;
    }
  }
}

// z^pm for the parameter weight of the reverse kick: closed forms for the
// quadrupole and sextupole orders
__device__ __forceinline__ void zpow_small(double x, double y, int pm, double &zr, double &zi) {
  if (pm == 1) {
    zr = x;
    zi = y;
  } else if (pm == 2) {
    zr = fma(x, x, -y * y);
    zi = 2.0 * x * y;
  } else if (pm == 0) {
    zr = 1.0;
    zi = 0.0;
  } else {
    zpow(x, y, pm, zr, zi);
  }
}

// The reverse walk reads the tape backwards from HBM with one warp per SM,
// one dependent access per kick.  Lane 0 asks the copy engine to bring the
// warp's next chunks (CHUNK kicks, 64 KiB) into L2 ahead of use: fire and
// forget, nothing waits on it.
constexpr int CHUNK = 64;

__device__ __forceinline__ void prefetch_l2_bulk(const double *p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// chunk [k0, k0 + CHUNK) of turn tt (clipped at 0) of this lane's warp
__device__ __forceinline__ void prefetch_chunk(const DiffArgs &a, int tt, int k0, int j) {
  const int lo = k0 < 0 ? 0 : k0;
  const int hi = min(k0 + CHUNK, a.kicks_per_turn);  // stay inside this warp's turn
  if (hi <= lo || (j % TLANES) != 0) return;
  prefetch_l2_bulk(a.tape + tidx(a, tt, lo, 0, 4, j),
                   static_cast<uint32_t>((hi - lo) * 4 * TLANES * sizeof(double)));
}

__device__ void save_ckpt(const St &s, const DiffArgs &a, int c, int j, bool tangent) {
  double *d = a.ckpt + static_cast<int64_t>(c) * 20 * a.n_jobs + j;
  d[0] = s.x;
  d[a.n_jobs] = s.px;
  d[2 * a.n_jobs] = s.y;
  d[3 * a.n_jobs] = s.py;
  if (tangent)
#pragma unroll
    for (int k = 0; k < 16; ++k) d[(4 + k) * static_cast<int64_t>(a.n_jobs)] = s.T[k];
}

__device__ void load_ckpt(St &s, const DiffArgs &a, int c, int j, bool tangent) {
  const double *d = a.ckpt + static_cast<int64_t>(c) * 20 * a.n_jobs + j;
  s.x = d[0];
  s.px = d[a.n_jobs];
  s.y = d[2 * a.n_jobs];
  s.py = d[3 * a.n_jobs];
#pragma unroll
  for (int k = 0; k < 16; ++k)
    s.T[k] = tangent ? d[(4 + k) * static_cast<int64_t>(a.n_jobs)] : 0.0;
}

__global__ void diff_forward(DiffArgs a) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= a.n_jobs) return;
  const bool tangent = a.tangent;
  St s;
  s.x = a.z0[4 * j]; s.px = a.z0[4 * j + 1]; s.y = a.z0[4 * j + 2]; s.py = a.z0[4 * j + 3];
#pragma unroll
  for (int k = 0; k < 16; ++k) s.T[k] = (k % 5 == 0) ? 1.0 : 0.0;
  const double o = a.o[j];
  const double *T0 = a.tab + (a.seed ? static_cast<int64_t>(a.seed[j]) : 0) * a.tab_stride;
  const bool ck = a.ckpt != nullptr;
  for (int t = 0; t < a.turns; ++t) {
    if (ck && t % a.ck == 0) save_ckpt(s, a, t / a.ck, j, tangent);
    turn_forward(s, a, T0, o, tangent, j, 0, false);
  }
  if (ck && a.turns % a.ck == 0) save_ckpt(s, a, a.turns / a.ck, j, tangent);
  double *d = a.zT + 20 * static_cast<int64_t>(j);
  d[0] = s.x; d[1] = s.px; d[2] = s.y; d[3] = s.py;
#pragma unroll
  for (int k = 0; k < 16; ++k) d[4 + k] = tangent ? s.T[k] : 0.0;
}

__global__ void diff_reverse(DiffArgs a) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= a.n_jobs) return;
  const bool tangent = a.tangent;
  const double o = a.o[j];
  const double *T0 = a.tab + (a.seed ? static_cast<int64_t>(a.seed[j]) : 0) * a.tab_stride;
  for (int k = 0; k < a.n_params; ++k) a.pbar[static_cast<int64_t>(k) * a.n_jobs + j] = 0.0;
  Bar b;
  b.x = a.zbar[4 * j]; b.px = a.zbar[4 * j + 1]; b.y = a.zbar[4 * j + 2]; b.py = a.zbar[4 * j + 3];
#pragma unroll
  for (int k = 0; k < 16; ++k) b.T[k] = tangent ? a.Tbar[16 * j + k] : 0.0;
  const int last_seg = (a.turns - 1) / a.ck;
  for (int sg = last_seg; sg >= 0; --sg) {
    const int t0 = sg * a.ck;
    const int t1 = min(a.turns, t0 + a.ck);
    St s;
    load_ckpt(s, a, sg, j, tangent);
    for (int t = t0; t < t1; ++t) turn_forward(s, a, T0, o, tangent, j, t - t0, true);
    for (int t = t1 - 1; t >= t0; --t) turn_reverse(b, a, T0, o, tangent, j, t - t0);
  }
  a.zbar0[4 * j] = b.x; a.zbar0[4 * j + 1] = b.px; a.zbar0[4 * j + 2] = b.y;
  a.zbar0[4 * j + 3] = b.py;
}

// ---------------------------------------------------------------- lane pairs
// Plain (non-tangent) mode runs every job on two lanes of a warp: the even
// lane carries the horizontal plane (x, px), the odd lane the vertical one
// (y, py), so a warp holds 16 jobs and a sweep of J jobs has twice the warps
// (the SM sub-partitions are what the one-thread-per-job sweep leaves idle).
// Each quantity is computed by the same IEEE operations, in the same order, as
// in the one-lane code above; the lanes exchange values by warp shuffles where
// a quantity needs both planes (z = x + iy of a kick, the complex Horner
// steps, the momentum cotangents of the reverse kick).  Lanes of a job past
// the end keep running on a clamped job (every shuffle has all 32 lanes) and
// write nothing.
constexpr unsigned ALL_LANES = 0xffffffffu;

struct Half {
  double u, pu;  // this lane's plane: (x, px) on even lanes, (y, py) on odd lanes
};

__device__ __forceinline__ double other(double v) { return __shfl_xor_sync(ALL_LANES, v, 1); }

// -v by its sign bit: as a floating-point negation that no FMA absorbs it would
// take a slot of the FP64 pipe (and its 115-cycle way to a select or shuffle)
__device__ __forceinline__ double neg(double v) {
  return __hiloint2double(__double2hiint(v) ^ static_cast<int>(0x80000000u), __double2loint(v));
}
// v != 0 without the pipe's comparison
__device__ __forceinline__ bool nonzero(double v) {
  return ((__double2hiint(v) & 0x7fffffff) | __double2loint(v)) != 0;
}

// S(z)/o (and S'(z)/o with ND = 1) split over the pair: `r0` / `r1` are this
// lane's part (real on even lanes, imaginary on odd lanes).  Both parts of a
// Horner step are (own x + c) -+ other y, so a lane's own value goes straight
// into the next FMA (64.6 cycles) while the other lane's is on its way through
// the shuffle (about 75 more than that): sy = -y on even, y on odd lanes.
// Measured, 777 particles through the 1,024-element ring with errors: 2.58 ->
// 1.84 ms per turn forward, with the operands' signs changed outside the FP64
// pipe and the opcodes fetched ahead.
template <int ND>
__device__ __forceinline__ void series_pair(const double *__restrict__ a, int M, double x, double sy,
                                            bool even, double &r0, double &r1) {
  const double *c = even ? a : a + M;
  r0 = __ldg(c + M - 1);
  r1 = 0.0;
  for (int n = M - 2; n >= 0; --n) {
    const double o0 = other(r0);
    if (ND >= 1) {
      const double o1 = other(r1);
      r1 = fma(o1, sy, fma(r1, x, r0));
    }
    r0 = fma(o0, sy, fma(r0, x, __ldg(c + n)));
  }
}

// this lane's tape entry of kick 0 of turn tt (plain mode)
__device__ __forceinline__ double *tape_turn(const DiffArgs &a, int tt, int j) {
  return a.tape + tidx(a, tt, 0, 0, 4, j);
}

// a kick element of the pair with its M coefficients (this lane's part: the
// normal list on even lanes, the skew list on odd lanes) loaded into
// registers once for all N slices; the unrolled Horner issues no loads
template <int M, bool TAPE>
__device__ __forceinline__ void kick_elem_pair(Half &h, const double *c, bool tp, int N, double oo,
                                               bool even, bool write, double *&tape) {
  double cf[M];
  const double *src = c + KHDR + (even ? 0 : M);
#pragma unroll
  for (int n = 0; n < M; ++n) cf[n] = __ldg(src + n);
  const double Lo = __ldg(c), Li = __ldg(c + 1), W = __ldg(c + 2), Lx = __ldg(c + 5);
  const double so = even ? neg(oo) : oo, sw = neg(W);
  // the x plane's alone: 0 times an infinite y would be NaN
  const bool weak = tp && even && nonzero(W);
  if (tp) h.u = fma(h.pu, Lo, h.u);
  for (int sl = 0; sl < N; ++sl) {
    const double w = other(h.u);
    const double x = even ? h.u : w, sy = even ? neg(w) : h.u;
    double r0 = cf[M - 1], r1 = 0.0;
#pragma unroll
    for (int n = M - 2; n >= 0; --n) {
      const double o0 = other(r0);
      if (TAPE) {
        const double o1 = other(r1);
        r1 = fma(o1, sy, fma(r1, x, r0));
      }
      r0 = fma(o0, sy, fma(r0, x, cf[n]));
    }
    if (TAPE) {
      if (write) {
        tape[even ? 0 : TLANES] = h.u;
        tape[(even ? 2 : 3) * TLANES] = oo * r1;
      }
      tape += 4 * TLANES;
    }
    h.pu = fma(so, r0, h.pu);
    if (weak) h.pu = fma(sw, h.u, h.pu);
    if (tp) h.u = fma(h.pu, sl < N - 1 ? Li : Lx, h.u);
  }
}

// An opcode ahead of its use.  The list is the caller's, aligned like any int32
// array: word by word.
__device__ __forceinline__ DOp fetch(const DOp *p) {
  const int *w = reinterpret_cast<const int *>(p);
  return {__ldg(w),     __ldg(w + 1), __ldg(w + 2), __ldg(w + 3),
          __ldg(w + 4), __ldg(w + 5), __ldg(w + 6), __ldg(w + 7)};
}

// one turn forward of the pair; with TAPE the rich tape is written from `tape`
// on (x, Re S' by the even lane; y, Im S' by the odd lane)
template <bool TAPE>
__device__ void turn_forward_pair(Half &h, const DiffArgs &a, const double *T0, double o,
                                  bool even, bool write, double *tape) {
  DOp next = a.n_ops > 0 ? fetch(a.ops) : DOp{};
  for (int i = 0; i < a.n_ops; ++i) {
    const DOp op = next;
    if (i + 1 < a.n_ops) next = fetch(a.ops + i + 1);
    const double *c = T0 + op.toff;
    const double oo = op.achro ? 1.0 : o;
    switch (op.kind) {
      case D_DRIFT:
        h.u = fma(h.pu, __ldg(c), h.u);
        break;
      case D_ALIGN:
        h.u -= __ldg(c + (even ? 0 : 1));
        break;
      case D_EDGE: {
        const double curv = __ldg(c) * oo;
        const double t = h.u * curv;
        h.pu = fma(t, even ? __ldg(c + 1) : neg(edge_t2(op.flags, c, curv)), h.pu);
        break;
      }
      case D_THICK: {
        const double L = __ldg(c), k1 = __ldg(c + 1), hh = __ldg(c + 2);
        if (TAPE) {  // entry state: x, px by the even lane; y, py by the odd lane
          if (write) {
            tape[even ? 0 : TLANES] = h.u;
            tape[(even ? 2 : 3) * TLANES] = h.pu;
          }
          tape += THICK_SLOTS * 4 * TLANES;
        }
        const double K = even ? oo * fma(hh, hh, k1) : -oo * k1;
        const double disp = (even && (op.flags & DT_BEND)) ? (1.0 / o - 1.0) * hh * oo : 0.0;
        thick_plane_fwd(h.u, h.pu, nullptr, nullptr, K, L, disp, false);
        break;
      }
      case D_KICK:
      case D_TEAPOT: {
        const bool tp = op.kind == D_TEAPOT;
        const int N = tp ? op.N : 1;
        switch (op.M) {  // common orders: coefficients in registers
          case 1: kick_elem_pair<1, TAPE>(h, c, tp, N, oo, even, write, tape); continue;
          case 2: kick_elem_pair<2, TAPE>(h, c, tp, N, oo, even, write, tape); continue;
          case 3: kick_elem_pair<3, TAPE>(h, c, tp, N, oo, even, write, tape); continue;
          case 4: kick_elem_pair<4, TAPE>(h, c, tp, N, oo, even, write, tape); continue;
          case 5: kick_elem_pair<5, TAPE>(h, c, tp, N, oo, even, write, tape); continue;
          case 6: kick_elem_pair<6, TAPE>(h, c, tp, N, oo, even, write, tape); continue;
          case 7: kick_elem_pair<7, TAPE>(h, c, tp, N, oo, even, write, tape); continue;
          case 8: kick_elem_pair<8, TAPE>(h, c, tp, N, oo, even, write, tape); continue;
          default: break;
        }
        const double Lo = __ldg(c), Li = __ldg(c + 1), W = __ldg(c + 2), Lx = __ldg(c + 5);
        if (tp) h.u = fma(h.pu, Lo, h.u);
        for (int sl = 0; sl < N; ++sl) {
          const double w = other(h.u);
          const double x = even ? h.u : w, sy = even ? neg(w) : h.u;
          double s0, s1;
          series_pair<TAPE ? 1 : 0>(c + KHDR, op.M, x, sy, even, s0, s1);
          if (TAPE) {
            if (write) {
              tape[even ? 0 : TLANES] = h.u;
              tape[(even ? 2 : 3) * TLANES] = oo * s1;
            }
            tape += 4 * TLANES;
          }
          h.pu = fma(even ? neg(oo) : oo, s0, h.pu);
          if (tp && even && nonzero(W)) h.pu = fma(neg(W), h.u, h.pu);
          if (tp) h.u = fma(h.pu, sl < N - 1 ? Li : Lx, h.u);
        }
        break;
      }
      default:
        break;
    }
  }
}

// Reverse of a kick element of the pair with the tape values of its N slices
// (x, y, Re S', Im S') loaded up front, before the dependent cotangent chain;
// `tape` points past them and moves to the element's first slice.
//   xb += -pxb a1 + pyb b1,  yb += pyb a1 + pxb b1  (a1 + i b1 = S'):
// both parts are own a1 first, then the other lane's b1.
// A part of N slices; `last`: it ends with the element's last slice, `first`: it
// starts with the first.
template <int N>
__device__ __forceinline__ void rev_part_pair(Half &bh, const DiffArgs &a, const double *c, bool tp,
                                              bool last, bool first, bool even, int j, bool write,
                                              int tt, int pm, int &kidx, const double *&tape,
                                              double &g0) {
  double tx[N], ty[N], ta[N], tb[N];
#pragma unroll
  for (int q = 0; q < N; ++q) {
    const double *t0 = tape - (q + 1) * 4 * TLANES;
    tx[q] = t0[0];
    ty[q] = t0[TLANES];
    ta[q] = even ? neg(t0[2 * TLANES]) : t0[2 * TLANES];
    tb[q] = t0[3 * TLANES];
  }
  tape -= N * 4 * TLANES;
  const double Lo = __ldg(c), Li = __ldg(c + 1), W = __ldg(c + 2), Lx = __ldg(c + 5);
  const double sw = neg(W);
  const bool weak = tp && even && nonzero(W);
#pragma unroll
  for (int q = 0; q < N; ++q) {  // slice N-1-q
    if (tp) bh.pu = fma(bh.u, q == 0 && last ? Lx : Li, bh.pu);
    if (weak) bh.u = fma(sw, bh.pu, bh.u);
    --kidx;
    if (write && even && kidx % CHUNK == 0 && kidx >= 2 * CHUNK)
      prefetch_chunk(a, tt, kidx - 2 * CHUNK, j);
    const double w = other(bh.pu);
    bh.u = fma(w, tb[q], fma(bh.pu, ta[q], bh.u));
    if (pm >= 0) {
      double zr, zi;
      zpow_small(tx[q], ty[q], pm, zr, zi);
      const double pxb = even ? bh.pu : w, pyb = even ? w : bh.pu;
      g0 = fma(-pxb, zr, fma(pyb, zi, g0));
    }
  }
  if (tp && first) bh.pu = fma(bh.u, Lo, bh.pu);
}

// reverse of turn `tt` of the group from the rich tape, split over the pair
// (cotangents of x, px on even lanes, of y, py on odd lanes)
__device__ void turn_reverse_pair(Half &bh, const DiffArgs &a, const double *T0, double o,
                                  bool even, int j, bool write, int tt) {
  int kidx = a.kicks_per_turn;
  const int top = ((a.kicks_per_turn - 1) / CHUNK) * CHUNK;
  if (write && even) {
    prefetch_chunk(a, tt, top, j);
    prefetch_chunk(a, tt, top - CHUNK, j);
  }
  const double *tape = tape_turn(a, tt, j) + static_cast<int64_t>(kidx) * 4 * TLANES;
  DOp next = a.n_ops > 0 ? fetch(a.ops + a.n_ops - 1) : DOp{};
  for (int i = a.n_ops - 1; i >= 0; --i) {
    const DOp op = next;
    if (i > 0) next = fetch(a.ops + i - 1);
    const double *c = T0 + op.toff;
    const double oo = op.achro ? 1.0 : o;
    switch (op.kind) {
      case D_DRIFT:
        bh.pu = fma(bh.u, __ldg(c), bh.pu);
        break;
      case D_ALIGN:
        break;
      case D_EDGE: {
        const double curv = __ldg(c) * oo;
        const double t = bh.pu * curv;
        bh.u = fma(t, even ? __ldg(c + 1) : neg(edge_t2(op.flags, c, curv)), bh.u);
        break;
      }
      case D_THICK: {
        const double L = __ldg(c), k1 = __ldg(c + 1), hh = __ldg(c + 2);
        kidx -= THICK_SLOTS;
        tape -= THICK_SLOTS * 4 * TLANES;
        const int m = ((kidx + THICK_SLOTS - 1) / CHUNK) * CHUNK;  // a chunk start in range
        if (write && even && m >= kidx && m >= 2 * CHUNK) prefetch_chunk(a, tt, m - 2 * CHUNK, j);
        const double q = tape[even ? 0 : TLANES], pq = tape[(even ? 2 : 3) * TLANES];
        const double K = even ? oo * fma(hh, hh, k1) : -oo * k1;
        const double disp = (even && (op.flags & DT_BEND)) ? (1.0 / o - 1.0) * hh * oo : 0.0;
        const double kb = thick_plane_rev(bh.u, bh.pu, nullptr, nullptr, nullptr, nullptr, q, pq,
                                          K, L, disp, false);
        const double kb_other = other(kb);  // every lane: the shuffle needs the whole warp
        if (op.pslot >= 0 && write && even) {  // dK_x/dk1 = o, dK_y/dk1 = -o
          double &p = a.pbar[static_cast<int64_t>(op.pslot) * a.n_jobs + j];
          p = fma(oo, kb - kb_other, p);
        }
        break;
      }
      case D_KICK:
      case D_TEAPOT: {
        const bool tp = op.kind == D_TEAPOT;
        const int N = tp ? op.N : 1;
        const int pm = op.pslot >= 0 ? op.pm : -1;
        double g0 = 0.0;
        double p0 = 0.0;  // the parameter's sum so far, fetched ahead
        double *pp = nullptr;
        if (op.pslot >= 0 && write && even) {
          pp = a.pbar + static_cast<int64_t>(op.pslot) * a.n_jobs + j;
          p0 = *pp;
        }
        int left = N;
        for (; left >= 8; left -= 8)
          rev_part_pair<8>(bh, a, c, tp, left == N, left == 8, even, j, write, tt, pm, kidx, tape, g0);
        for (; left >= 4; left -= 4)
          rev_part_pair<4>(bh, a, c, tp, left == N, left == 4, even, j, write, tt, pm, kidx, tape, g0);
        for (; left >= 1; --left)
          rev_part_pair<1>(bh, a, c, tp, left == N, left == 1, even, j, write, tt, pm, kidx, tape, g0);
        if (tp && N < 1) bh.pu = fma(bh.u, __ldg(c), bh.pu);  // the outer drift alone
        if (pp) *pp = fma(g0 * oo, __ldg(c + 3), p0);
        break;
      }
      default:
        break;
    }
  }
}

// pair index of this thread: job j (clamped), lane parity, whether it writes
__device__ __forceinline__ void pair_of(int64_t t, int64_t jobs, int64_t &job, bool &even,
                                        bool &write) {
  job = t >> 1;
  even = (t & 1) == 0;
  write = job < jobs;
  if (!write) job = jobs - 1;
}

__global__ void diff_forward_pair(DiffArgs a) {
  const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if ((t & ~static_cast<int64_t>(31)) >= 2 * static_cast<int64_t>(a.n_jobs)) return;  // whole warp past the end
  int64_t jl;
  bool even, write;
  pair_of(t, a.n_jobs, jl, even, write);
  const int j = static_cast<int>(jl);
  Half h;
  h.u = a.z0[4 * j + (even ? 0 : 2)];
  h.pu = a.z0[4 * j + (even ? 1 : 3)];
  const double o = a.o[j];
  const double *T0 = a.tab + (a.seed ? static_cast<int64_t>(a.seed[j]) : 0) * a.tab_stride;
  const bool ck = a.ckpt != nullptr;
  const int f0 = even ? 0 : 2;
  for (int tt = 0; tt < a.turns; ++tt) {
    if (ck && tt % a.ck == 0 && write) {
      double *d = a.ckpt + static_cast<int64_t>(tt / a.ck) * 20 * a.n_jobs + j;
      d[f0 * static_cast<int64_t>(a.n_jobs)] = h.u;
      d[(f0 + 1) * static_cast<int64_t>(a.n_jobs)] = h.pu;
    }
    turn_forward_pair<false>(h, a, T0, o, even, write, nullptr);
  }
  if (write) {
    if (ck && a.turns % a.ck == 0) {
      double *d = a.ckpt + static_cast<int64_t>(a.turns / a.ck) * 20 * a.n_jobs + j;
      d[f0 * static_cast<int64_t>(a.n_jobs)] = h.u;
      d[(f0 + 1) * static_cast<int64_t>(a.n_jobs)] = h.pu;
    }
    double *d = a.zT + 20 * static_cast<int64_t>(j);
    d[f0] = h.u;
    d[f0 + 1] = h.pu;
    if (even)
      for (int k = 4; k < 20; ++k) d[k] = 0.0;
  }
}

__global__ void diff_tape_pair(DiffArgs a, int sg0, int G) {
  const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  const int64_t pairs = static_cast<int64_t>(G) * a.n_jobs;
  if ((t & ~static_cast<int64_t>(31)) >= 2 * pairs) return;
  int64_t q;
  bool even, write;
  pair_of(t, pairs, q, even, write);
  const int g = static_cast<int>(q / a.n_jobs), j = static_cast<int>(q % a.n_jobs);
  const int sg = sg0 + g;
  const int t0 = sg * a.ck;
  const bool live = t0 < a.turns;  // uniform per segment: whole warps agree unless G spans
  const int t1 = live ? min(a.turns, t0 + a.ck) : t0;
  const double o = a.o[j];
  const double *T0 = a.tab + (a.seed ? static_cast<int64_t>(a.seed[j]) : 0) * a.tab_stride;
  Half h;
  const int f0 = even ? 0 : 2;
  const int sl = live ? sg : 0;
  const double *d = a.ckpt + static_cast<int64_t>(sl) * 20 * a.n_jobs + j;
  h.u = d[f0 * static_cast<int64_t>(a.n_jobs)];
  h.pu = d[(f0 + 1) * static_cast<int64_t>(a.n_jobs)];
  // a warp may straddle two segments (J not a multiple of 16): every lane runs
  // the longer count; lanes past their own segment end do not write
  const int tmax = __reduce_max_sync(ALL_LANES, t1 - t0);
  for (int k = 0; k < tmax; ++k)
    turn_forward_pair<true>(h, a, T0, o, even, write && k < t1 - t0, tape_turn(a, g * a.ck + k, j));
}

__global__ void diff_reverse_plain_pair(DiffArgs a, int sg0, int sg_hi) {
  const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if ((t & ~static_cast<int64_t>(31)) >= 2 * static_cast<int64_t>(a.n_jobs)) return;
  int64_t jl;
  bool even, write;
  pair_of(t, a.n_jobs, jl, even, write);
  const int j = static_cast<int>(jl);
  const double o = a.o[j];
  const double *T0 = a.tab + (a.seed ? static_cast<int64_t>(a.seed[j]) : 0) * a.tab_stride;
  const int f0 = even ? 0 : 2;
  Half bh;
  bh.u = a.zbar0[4 * j + f0];
  bh.pu = a.zbar0[4 * j + f0 + 1];
  for (int sg = sg_hi; sg >= sg0; --sg) {
    const int t0 = sg * a.ck;
    const int t1 = min(a.turns, t0 + a.ck);
    for (int tt = t1 - 1; tt >= t0; --tt)
      turn_reverse_pair(bh, a, T0, o, even, j, write, (sg - sg0) * a.ck + (tt - t0));
  }
  if (write) {
    a.zbar0[4 * j + f0] = bh.u;
    a.zbar0[4 * j + f0 + 1] = bh.pu;
  }
}

// ---------------------------------------------------------------- eight lanes
// Tangent mode runs every job on eight lanes: plane (as the pairs above) x
// column of the 4x4 tangent; the state is carried by all four column lanes.
// The few jobs of an optics evaluation (three momenta per row) leave the GPU
// empty, so a turn's time is one lane's FP64 instructions: per kick of order M
// 75 with a job per lane, 28 with eight lanes (M = 6).  Measured on one GB300,
// 1,024-element ring with errors, 3 jobs, per turn: forward 7.9 -> 3.6 ms, taped
// forward and reverse 21.7 -> 10.1 ms.
struct Oct {
  double u, pu;  // this plane's coordinates (or their cotangents)
  double tu, tp; // this plane's two tangent rows in this lane's column
};

struct OctLane {
  bool even, write;  // plane; the lane's results are kept
  int col, j;
  double *tape;      // this lane's first entry of the turn
};

// this turn's tape entry of kick 0, field 0
__device__ __forceinline__ double *oct_tape(const DiffArgs &a, int tt, int j) {
  return a.tape + tidx(a, tt, 0, 0, 10, j);
}

// fields of a slot: x, y, T rows x and y (or, in a thick element's second slot,
// px, py and their rows)
__device__ __forceinline__ void oct_put(double *t, const OctLane &l, double v, double tv) {
  if (!l.write) return;
  if (l.col == 0) t[(l.even ? 0 : 1) * TLANES] = v;
  t[((l.even ? 2 : 6) + l.col) * TLANES] = tv;
}

__device__ __forceinline__ void oct_drift(Oct &s, double L) {
  s.u = fma(s.pu, L, s.u);
  s.tu = fma(s.tp, L, s.tu);
}

// a kick element; MM: its number of terms (0: M, at run time)
template <int MM, bool TAPE>
__device__ __forceinline__ void kick_elem_oct(Oct &s, const double *c, int M, bool tp, int N,
                                              double oo, const OctLane &l, double *&tape) {
  const bool even = l.even;
  constexpr int R = MM > 0 ? MM : 1;
  double cf[R];
#pragma unroll
  for (int n = 0; n < R; ++n) cf[n] = __ldg(c + KHDR + (even ? 0 : M) + n);
  const double Lo = __ldg(c), Li = __ldg(c + 1), W = __ldg(c + 2), Lx = __ldg(c + 5);
  const double so = even ? neg(oo) : oo, sw = neg(W);
  const bool weak = tp && even && nonzero(W);
  if (tp) oct_drift(s, Lo);
  for (int sl = 0; sl < N; ++sl) {
    if (TAPE) {
      oct_put(tape, l, s.u, s.tu);
      tape += 10 * TLANES;
    }
    const double w = other(s.u), ot = other(s.tu);
    const double x = even ? s.u : w, sy = even ? neg(w) : s.u;
    double s0, s1;
    if (MM > 0) {
      s0 = cf[R - 1];
      s1 = 0.0;
#pragma unroll
      for (int n = R - 2; n >= 0; --n) {
        const double o0 = other(s0), o1 = other(s1);
        s1 = fma(o1, sy, fma(s1, x, s0));
        s0 = fma(o0, sy, fma(s0, x, cf[n]));
      }
    } else {
      series_pair<1>(c + KHDR, M, x, sy, even, s0, s1);
    }
    s1 *= oo;
    s.pu = fma(so, s0, s.pu);
    const double o1 = other(s1);
    s.tp = fma(even ? o1 : s1, ot, fma(even ? neg(s1) : o1, s.tu, s.tp));
    if (weak) {
      s.pu = fma(sw, s.u, s.pu);
      s.tp = fma(sw, s.tu, s.tp);
    }
    if (tp) oct_drift(s, sl < N - 1 ? Li : Lx);
  }
}

template <bool TAPE>
__device__ void turn_forward_oct(Oct &s, const DiffArgs &a, const double *T0, double o,
                                 const OctLane &l, double *tape) {
  const bool even = l.even;
  DOp next = a.n_ops > 0 ? fetch(a.ops) : DOp{};
  for (int i = 0; i < a.n_ops; ++i) {
    const DOp op = next;
    if (i + 1 < a.n_ops) next = fetch(a.ops + i + 1);
    const double *c = T0 + op.toff;
    const double oo = op.achro ? 1.0 : o;
    switch (op.kind) {
      case D_DRIFT:
        oct_drift(s, __ldg(c));
        break;
      case D_ALIGN:
        s.u -= __ldg(c + (even ? 0 : 1));
        break;
      case D_EDGE: {
        const double curv = __ldg(c) * oo;
        const double e = even ? __ldg(c + 1) : neg(edge_t2(op.flags, c, curv));
        s.pu = fma(s.u * curv, e, s.pu);
        s.tp = fma(s.tu * curv, e, s.tp);
        break;
      }
      case D_KICK:
      case D_TEAPOT: {
        const bool tp = op.kind == D_TEAPOT;
        const int N = tp ? op.N : 1;
        switch (op.M) {  // common orders: coefficients in registers
          case 1: kick_elem_oct<1, TAPE>(s, c, op.M, tp, N, oo, l, tape); break;
          case 2: kick_elem_oct<2, TAPE>(s, c, op.M, tp, N, oo, l, tape); break;
          case 3: kick_elem_oct<3, TAPE>(s, c, op.M, tp, N, oo, l, tape); break;
          case 4: kick_elem_oct<4, TAPE>(s, c, op.M, tp, N, oo, l, tape); break;
          case 5: kick_elem_oct<5, TAPE>(s, c, op.M, tp, N, oo, l, tape); break;
          case 6: kick_elem_oct<6, TAPE>(s, c, op.M, tp, N, oo, l, tape); break;
          default: kick_elem_oct<0, TAPE>(s, c, op.M, tp, N, oo, l, tape); break;
        }
        break;
      }
      case D_THICK: {
        const double L = __ldg(c), k1 = __ldg(c + 1), h = __ldg(c + 2);
        if (TAPE) {
          oct_put(tape, l, s.u, s.tu);
          oct_put(tape + 10 * TLANES, l, s.pu, s.tp);
          tape += THICK_SLOTS * 10 * TLANES;
        }
        const double K = even ? oo * fma(h, h, k1) : -oo * k1;
        const double disp = (even && (op.flags & DT_BEND)) ? (1.0 / o - 1.0) * h * oo : 0.0;
        double C, Sw, D1, dC, dSw, dD1;
        thick_fns<false>(K, L, C, Sw, D1, dC, dSw, dD1);
        const double A = -K * Sw, u0 = s.u, t0 = s.tu;
        s.u = fma(C, u0, fma(Sw, s.pu, disp * D1));
        s.pu = fma(A, u0, fma(C, s.pu, disp * Sw));
        s.tu = fma(C, t0, Sw * s.tp);
        s.tp = fma(A, t0, C * s.tp);
        break;
      }
      default:
        break;
    }
  }
}

// sum over the four columns; every lane gets it
__device__ __forceinline__ double oct_sum(double v) {
  v += __shfl_xor_sync(ALL_LANES, v, 2);
  return v + __shfl_xor_sync(ALL_LANES, v, 4);
}

// reverse of one turn from the tape that turn_forward_oct<true> wrote
__device__ void turn_reverse_oct(Oct &b, const DiffArgs &a, const double *T0, double o,
                                 const OctLane &l, const double *tape) {
  const bool even = l.even;
  tape += static_cast<int64_t>(a.kicks_per_turn) * 10 * TLANES;
  const bool keeps = l.write && even && l.col == 0;  // the lane that owns the sums
  DOp next = a.n_ops > 0 ? fetch(a.ops + a.n_ops - 1) : DOp{};
  for (int i = a.n_ops - 1; i >= 0; --i) {
    const DOp op = next;
    if (i > 0) next = fetch(a.ops + i - 1);
    const double *c = T0 + op.toff;
    const double oo = op.achro ? 1.0 : o;
    switch (op.kind) {
      case D_DRIFT:
        b.pu = fma(b.u, __ldg(c), b.pu);
        b.tp = fma(b.tu, __ldg(c), b.tp);
        break;
      case D_ALIGN:
        break;  // translation: cotangents unchanged
      case D_EDGE: {
        const double curv = __ldg(c) * oo;
        const double e = even ? __ldg(c + 1) : neg(edge_t2(op.flags, c, curv));
        b.u = fma(b.pu * curv, e, b.u);
        b.tu = fma(b.tp * curv, e, b.tu);
        break;
      }
      case D_KICK:
      case D_TEAPOT: {
        const bool tp = op.kind == D_TEAPOT;
        const int N = tp ? op.N : 1;
        const double Lo = __ldg(c), Li = __ldg(c + 1), W = __ldg(c + 2), Lx = __ldg(c + 5);
        const double sw = neg(W);
        const bool weak = tp && even && nonzero(W);
        const int pm = op.pslot >= 0 ? op.pm : -1;
        const double *coef = c + KHDR + (even ? 0 : op.M);
        double g0 = 0.0, g1 = 0.0;
        for (int sl = N - 1; sl >= 0; --sl) {
          tape -= 10 * TLANES;
          const double x = tape[0], y = tape[TLANES];
          const double dx = tape[(2 + l.col) * TLANES], dy = tape[(6 + l.col) * TLANES];
          if (tp) {
            const double L = sl < N - 1 ? Li : Lx;
            b.pu = fma(b.u, L, b.pu);
            b.tp = fma(b.tu, L, b.tp);
          }
          if (weak) {
            b.u = fma(sw, b.pu, b.u);
            b.tu = fma(sw, b.tp, b.tu);
          }
          // this lane's parts of S, S', S''/2 (series<2>)
          const double sy = even ? neg(y) : y;
          double s0 = __ldg(coef + op.M - 1), s1 = 0.0, s2 = 0.0;
          for (int n = op.M - 2; n >= 0; --n) {
            const double o0 = other(s0), o1 = other(s1), o2 = other(s2);
            s2 = fma(o2, sy, fma(s2, x, s1));
            s1 = fma(o1, sy, fma(s1, x, s0));
            s0 = fma(o0, sy, fma(s0, x, __ldg(coef + n)));
          }
          s1 *= oo;
          s2 *= 2.0 * oo;
          const double o1 = other(s1), o2 = other(s2);
          const double A = even ? neg(s1) : o1, B = even ? o1 : s1;    // -+a1, b1
          const double A2 = even ? s2 : o2, B2 = even ? o2 : neg(s2);  // a2, +-b2
          const double w = other(b.pu), wt = other(b.tp);
          const double sum = oct_sum(fma(even ? neg(b.tp) : b.tp, dx, wt * dy));  // Ab | Bb
          const double osum = other(sum);
          if (pm >= 0) {
            const double pxb = even ? b.pu : w, pyb = even ? w : b.pu;
            double zr, zi;
            zpow_small(x, y, pm, zr, zi);
            g0 += oo * fma(-pxb, zr, pyb * zi);
            if (pm >= 1) {
              const double Ab = even ? sum : osum, Bb = even ? osum : sum;
              zpow_small(x, y, pm - 1, zr, zi);
              g1 += oo * fma(Ab, zr, Bb * zi);
            }
          }
          b.u = fma(w, B, fma(b.pu, A, b.u));
          b.tu = fma(wt, B, fma(b.tp, A, b.tu));
          b.u = fma(osum, B2, fma(sum, A2, b.u));
        }
        if (tp) {
          b.pu = fma(b.u, Lo, b.pu);
          b.tp = fma(b.tu, Lo, b.tp);
        }
        if (op.pslot >= 0 && keeps) {
          double &p = a.pbar[static_cast<int64_t>(op.pslot) * a.n_jobs + l.j];
          p = fma(g0, __ldg(c + 3), fma(g1, __ldg(c + 4), p));
        }
        break;
      }
      case D_THICK: {
        const double L = __ldg(c), k1 = __ldg(c + 1), h = __ldg(c + 2);
        tape -= THICK_SLOTS * 10 * TLANES;
        const double *t1 = tape + 10 * TLANES;
        const int v = (even ? 0 : 1) * TLANES, r = ((even ? 2 : 6) + l.col) * TLANES;
        const double q = tape[v], pq = t1[v], tq = tape[r], tpq = t1[r];
        const double K = even ? oo * fma(h, h, k1) : -oo * k1;
        const double disp = (even && (op.flags & DT_BEND)) ? (1.0 / o - 1.0) * h * oo : 0.0;
        double C, Sw, D1, dC, dSw, dD1;
        thick_fns<true>(K, L, C, Sw, D1, dC, dSw, dD1);
        const double A = -K * Sw, dA = fma(-K, dSw, -Sw);
        double Kb = fma(b.u, fma(dC, q, fma(dSw, pq, disp * dD1)),
                        b.pu * fma(dA, q, fma(dC, pq, disp * dSw)));
        Kb += oct_sum(fma(b.tu, fma(dC, tq, dSw * tpq), b.tp * fma(dA, tq, dC * tpq)));
        const double bu = b.u, bt = b.tu;
        b.u = fma(C, bu, A * b.pu);
        b.pu = fma(Sw, bu, C * b.pu);
        b.tu = fma(C, bt, A * b.tp);
        b.tp = fma(Sw, bt, C * b.tp);
        const double ko = other(Kb);
        if (op.pslot >= 0 && keeps) {  // dK_x/dk1 = o, dK_y/dk1 = -o
          double &p = a.pbar[static_cast<int64_t>(op.pslot) * a.n_jobs + l.j];
          p = fma(oo, Kb - ko, p);
        }
        break;
      }
      default:
        break;
    }
  }
}

__device__ __forceinline__ OctLane oct_lane(const DiffArgs &a) {
  const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  const int64_t job = t >> 3;
  OctLane l;
  l.even = (t & 1) == 0;
  l.col = static_cast<int>(t >> 1) & 3;
  l.write = job < a.n_jobs;  // lanes past the end run along on the last job
  l.j = static_cast<int>(l.write ? job : a.n_jobs - 1);
  return l;
}

// the rows of this lane in a [4 coordinates][16 tangent entries] record with
// `n` between entries
__device__ __forceinline__ void oct_save(const Oct &s, const OctLane &l, double *d, int64_t n) {
  if (!l.write) return;
  if (l.col == 0) {
    d[(l.even ? 0 : 2) * n] = s.u;
    d[(l.even ? 1 : 3) * n] = s.pu;
  }
  d[(4 + (l.even ? 0 : 8) + l.col) * n] = s.tu;
  d[(4 + (l.even ? 4 : 12) + l.col) * n] = s.tp;
}

__global__ void __launch_bounds__(32) diff_forward_oct(DiffArgs a) {
  const OctLane l = oct_lane(a);
  Oct s;
  s.u = a.z0[4 * l.j + (l.even ? 0 : 2)];
  s.pu = a.z0[4 * l.j + (l.even ? 1 : 3)];
  s.tu = l.col == (l.even ? 0 : 2) ? 1.0 : 0.0;
  s.tp = l.col == (l.even ? 1 : 3) ? 1.0 : 0.0;
  const double o = a.o[l.j];
  const double *T0 = a.tab + (a.seed ? static_cast<int64_t>(a.seed[l.j]) : 0) * a.tab_stride;
  const int64_t J = a.n_jobs;
  for (int t = 0; t < a.turns; ++t) {
    if (a.ckpt && t % a.ck == 0)
      oct_save(s, l, a.ckpt + static_cast<int64_t>(t / a.ck) * 20 * J + l.j, J);
    turn_forward_oct<false>(s, a, T0, o, l, nullptr);
  }
  if (a.ckpt && a.turns % a.ck == 0)
    oct_save(s, l, a.ckpt + static_cast<int64_t>(a.turns / a.ck) * 20 * J + l.j, J);
  oct_save(s, l, a.zT + 20 * static_cast<int64_t>(l.j), 1);
}

__global__ void __launch_bounds__(32) diff_reverse_oct(DiffArgs a) {
  const OctLane l = oct_lane(a);
  const double o = a.o[l.j];
  const double *T0 = a.tab + (a.seed ? static_cast<int64_t>(a.seed[l.j]) : 0) * a.tab_stride;
  const int64_t J = a.n_jobs;
  if (l.write)
    for (int k = threadIdx.x & 7; k < a.n_params; k += 8) a.pbar[k * J + l.j] = 0.0;
  Oct b;
  b.u = a.zbar[4 * l.j + (l.even ? 0 : 2)];
  b.pu = a.zbar[4 * l.j + (l.even ? 1 : 3)];
  b.tu = a.Tbar[16 * static_cast<int64_t>(l.j) + (l.even ? 0 : 8) + l.col];
  b.tp = a.Tbar[16 * static_cast<int64_t>(l.j) + (l.even ? 4 : 12) + l.col];
  __syncwarp();
  for (int sg = (a.turns - 1) / a.ck; sg >= 0; --sg) {
    const int t0 = sg * a.ck, t1 = min(a.turns, t0 + a.ck);
    const double *d = a.ckpt + static_cast<int64_t>(sg) * 20 * J + l.j;
    Oct s;
    s.u = d[(l.even ? 0 : 2) * J];
    s.pu = d[(l.even ? 1 : 3) * J];
    s.tu = d[(4 + (l.even ? 0 : 8) + l.col) * J];
    s.tp = d[(4 + (l.even ? 4 : 12) + l.col) * J];
    for (int t = t0; t < t1; ++t)
      turn_forward_oct<true>(s, a, T0, o, l, oct_tape(a, t - t0, l.j));
    __syncwarp();  // the tape's entries are read by other lanes than wrote them
    for (int t = t1 - 1; t >= t0; --t) turn_reverse_oct(b, a, T0, o, l, oct_tape(a, t - t0, l.j));
    __syncwarp();
  }
  if (l.write && l.col == 0) {
    a.zbar0[4 * l.j + (l.even ? 0 : 2)] = b.u;
    a.zbar0[4 * l.j + (l.even ? 1 : 3)] = b.pu;
  }
}

}  // namespace ufo_diff

// ---------------------------------------------------------------- C ABI
extern "C" {

// All pointers are device pointers; `ops` int32[n_ops][8] (DOp), `tab` f64.
// Asynchronous on `stream`.  Returns 0, -1 (bad arguments) or -2 (launch
// error).
// the kernels use no shared memory: give the whole on-chip store to L1, where
// the opcode list and one seed's constants (~200 kB for a 1,000-element ring)
// then stay resident
static void prefer_l1() {
  static bool done = false;
  if (done) return;
  cudaFuncSetAttribute(ufo_diff::diff_forward, cudaFuncAttributePreferredSharedMemoryCarveout, 0);
  cudaFuncSetAttribute(ufo_diff::diff_reverse, cudaFuncAttributePreferredSharedMemoryCarveout, 0);
  cudaFuncSetAttribute(ufo_diff::diff_forward_pair,
                       cudaFuncAttributePreferredSharedMemoryCarveout, 0);
  cudaFuncSetAttribute(ufo_diff::diff_tape_pair, cudaFuncAttributePreferredSharedMemoryCarveout, 0);
  cudaFuncSetAttribute(ufo_diff::diff_reverse_plain_pair,
                       cudaFuncAttributePreferredSharedMemoryCarveout, 0);
  done = true;
}

// Eight lanes per job while their warps are at most two per sub-partition: two
// queue for the FP64 pipe in the time the one-lane form's single warp takes.
static bool oct_lanes_pay(int n_jobs) {
  int device = 0, sms = 0;
  if (cudaGetDevice(&device) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
    return false;
  return n_jobs <= 32 * sms;
}

int ufo_diff_forward(const int32_t *ops, int n_ops, const double *tab, int64_t tab_stride,
                     const int32_t *seed, int n_params, int kicks_per_turn, int n_jobs,
                     const double *z0, const double *o, int turns, int ck, int tangent,
                     double *ckpt, double *zT, void *stream) {
  if (n_jobs <= 0) return 0;
  if (!ops || n_ops < 0 || !tab || !z0 || !o || !zT || turns < 0 || ck < 1) return -1;
  prefer_l1();
  ufo_diff::DiffArgs a{};
  a.ops = reinterpret_cast<const ufo_diff::DOp *>(ops);
  a.n_ops = n_ops;
  a.tab = tab;
  a.tab_stride = tab_stride;
  a.seed = seed;
  a.n_params = n_params;
  a.kicks_per_turn = kicks_per_turn;
  a.n_jobs = n_jobs;
  a.z0 = z0;
  a.o = o;
  a.turns = turns;
  a.ck = ck;
  a.tangent = tangent;
  a.ckpt = ckpt;
  a.zT = zT;
  const int tpb = 32;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (tangent && oct_lanes_pay(n_jobs)) {
    ufo_diff::diff_forward_oct<<<(n_jobs + 3) / 4, tpb, 0, st>>>(a);
  } else if (tangent) {
    ufo_diff::diff_forward<<<(n_jobs + tpb - 1) / tpb, tpb, 0, st>>>(a);
  } else {  // two lanes per job
    const int64_t threads = 2 * static_cast<int64_t>(n_jobs);
    ufo_diff::diff_forward_pair<<<static_cast<unsigned>((threads + tpb - 1) / tpb), tpb, 0, st>>>(a);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int ufo_diff_reverse(const int32_t *ops, int n_ops, const double *tab, int64_t tab_stride,
                     const int32_t *seed, int n_params, int kicks_per_turn, int n_jobs,
                     const double *o, int turns, int ck, int tangent, const double *ckpt,
                     const double *zbar, const double *Tbar, double *tape, int tape_segments,
                     double *zbar0, double *pbar, void *stream) {
  if (n_jobs <= 0) return 0;
  if (!ops || n_ops < 0 || !tab || !o || !ckpt || !zbar || !tape || !zbar0 ||
      (n_params > 0 && !pbar) || turns < 1 || ck < 1 || (tangent && !Tbar) || tape_segments < 1)
    return -1;
  prefer_l1();
  ufo_diff::DiffArgs a{};
  a.ops = reinterpret_cast<const ufo_diff::DOp *>(ops);
  a.n_ops = n_ops;
  a.tab = tab;
  a.tab_stride = tab_stride;
  a.seed = seed;
  a.n_params = n_params;
  a.kicks_per_turn = kicks_per_turn;
  a.n_jobs = n_jobs;
  a.o = o;
  a.turns = turns;
  a.ck = ck;
  a.tangent = tangent;
  a.ckpt = const_cast<double *>(ckpt);
  a.zbar = zbar;
  a.Tbar = Tbar;
  a.tape = tape;
  a.zbar0 = zbar0;
  a.pbar = pbar;
  const int tpb = 32;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (tangent) {
    if (oct_lanes_pay(n_jobs))
      ufo_diff::diff_reverse_oct<<<(n_jobs + 3) / 4, tpb, 0, st>>>(a);
    else
      ufo_diff::diff_reverse<<<(n_jobs + tpb - 1) / tpb, tpb, 0, st>>>(a);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
  }
  // plain mode: groups of up to tape_segments segments, last group first
  if (n_params > 0 &&
      cudaMemsetAsync(pbar, 0, sizeof(double) * n_params * static_cast<size_t>(n_jobs), st) !=
          cudaSuccess)
    return -2;
  if (cudaMemcpyAsync(zbar0, zbar, sizeof(double) * 4 * static_cast<size_t>(n_jobs),
                      cudaMemcpyDeviceToDevice, st) != cudaSuccess)
    return -2;
  const int last_seg = (turns - 1) / ck;
  for (int hi = last_seg; hi >= 0; hi -= tape_segments) {
    const int lo = hi - tape_segments + 1 < 0 ? 0 : hi - tape_segments + 1;
    const int G = hi - lo + 1;
    const int64_t threads = 2 * static_cast<int64_t>(G) * n_jobs;  // two lanes per job
    ufo_diff::diff_tape_pair<<<static_cast<unsigned>((threads + tpb - 1) / tpb), tpb, 0, st>>>(
        a, lo, G);
    const int64_t rthreads = 2 * static_cast<int64_t>(n_jobs);
    ufo_diff::diff_reverse_plain_pair<<<static_cast<unsigned>((rthreads + tpb - 1) / tpb), tpb, 0,
                                        st>>>(a, lo, hi);
    if (cudaGetLastError() != cudaSuccess) return -2;
  }
  return 0;
}

}  // extern "C"
