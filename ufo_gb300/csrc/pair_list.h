// pair_list.h -- the two-lane kernel's opcode list and its host side: which form
// an op takes, made from the public opcodes and constants.  Plain C++, so that a
// CPU test can read what the kernel (pair.cuh) is going to walk.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstring>
#include <unordered_map>
#include <vector>

#include "../../include/ufo_gb300.h"
#include "opcodes.h"

#ifdef __CUDACC__
#define UFO_HOST_DEV __host__ __device__ inline
#else
#define UFO_HOST_DEV inline
#endif

namespace ufo {

// ---- opcode words of this kernel, built on the host (decode_pair)
//   head  bits 0-7 variant, 8-15 exponent shift of div_shift, PF_* flags
//   toff  first constant in the table row
//   a     slices; first field in the coefficient cache; observation
//         index; first op of a segment in the public list
//   b     general kicks: normal mask | skew mask << 16; end of the segment; with
//         PF_THEN the first constant of a plain drift that follows the op
struct PairOp {
  int head, toff, a, b;
};
enum : int {
  PF_NEG = 1 << 16,    // div_shift subtracts
  PF_ACHRO = 1 << 17, PF_SPLITO = 1 << 18,
  PF_X = 1 << 19, PF_Y = 1 << 20,  // the plane has the term (align, edge)
  PF_CONST = 1 << 21, PF_PSER = 1 << 22,
  PF_DIV = 1 << 23,    // the table holds [A, d, 1/d, A/d] for the inner drift
  PF_FILL = 1 << 24,   // this op fills its cache fields
  PF_THEN = 1 << 25,   // a plain drift follows, run with this op (strict list only)
  // general teapots: the alignment shifts around them run with them (PF_X, PF_Y
  // as in an align op), two dispatches fewer per magnet (FODO ring with errors,
  // 1,000 particles, FMA 192 -> 183 us per turn, light-source ring 2,066 ->
  // 1,907); their constants lie right before and after the element's, or
  // (.._EDGE) beyond an empty edge's three
  PF_PRE = 1 << 26, PF_POST = 1 << 27, PF_PRE_EDGE = 1 << 28, PF_POST_EDGE = 1 << 29
};
enum : int {
  PV_SEGMENT = 0, PV_DRIFT, PV_DRIFT2, PV_DRIFT_DIV, PV_ALIGN, PV_EDGE, PV_EDGE_PSI, PV_THICKQ,
  PV_THICKB, PV_CIRCLE, PV_OBSERVE, PV_LINEAR, PV_WIDE,
  PV_KICK = 16,   // + pattern (0..3, see teapot in ops.cuh)
  PV_TEAPOT = 20  // + pattern (0..3) + 4 * division form (0..2) + 12 * weak
};
constexpr int PAIR_SEGMENT = 16;
// forms of the inner drift of a teapot: x += px L; x += (px A) / d with one
// FMA (see div_shift); the same by Markstein's correction (divc)
enum : int { DIV_NONE = 0, DIV_SHIFT = 1, DIV_GENERAL = 2, DIV_ANY = 3 };
// cached fields of a thick element, per lane
enum : int { TC_C = 0, TC_S, TC_K, TC_R, TC_Z, TC_D, TC_DP, TC_FIELDS };

// ------------------------------------------------ two-lane opcode list
// The exponent shift of div_shift for the divisor d (RN(1/d) = r in the
// table), or 0 when no power of two serves: with eps = (1/d - r) / ulp(r) and M
// the significand of 1/d, the candidate k = +-2^-j must satisfy |k - eps| <
// 1/(2 d') over operand significands up to 2/M (quotients below the next power
// of two) and up to 2 halved (above it); 0.95 leaves room for the terms of
// order 2^-53 that the bound drops.
inline int shift_form(double d, double r, bool &negative) {
  if (!(d > 1.0 && d < 1048576.0) || d != std::floor(d) || r != 1.0 / d) return 0;
  long odd = static_cast<long>(d);
  while (odd % 2 == 0) odd /= 2;
  if (odd == 1) return 0;
  int ez = 0;
  const double m = 2.0 * std::frexp(r, &ez);  // r = m 2^(ez-1), m in [1, 2)
  --ez;
  const double eps = std::ldexp(std::fma(-d, r, 1.0) / d, 52 - ez);
  negative = eps < 0.0;
  const double bound = 0.95 / (2.0 * static_cast<double>(odd));
  for (int j = 1; j <= 8; ++j) {
    const double k = std::ldexp(negative ? -1.0 : 1.0, -j);
    const double off = std::fabs(k - eps);
    if (off * (2.0 / m) < bound && off < bound) return 52 + j - ez;
  }
  return 0;
}

// kick pattern of the interpreters (teapot in ops.cuh)
inline int kick_pattern(int nn, int ns, int32_t mn) {
  return ns != 0 ? 0 : (nn == 2 && mn == 2) ? 1 : (nn == 3 && mn == 4) ? 2 : mn == 0 ? 3 : 0;
}

// What the two-lane lists need to know of every row's constants.
struct RowScan {
  bool plain = true;     // strengths whose half and negative are exact, in every row
  bool same = true;      // an inner drift's division is row 0's in every row
  int twin = -1;         // an earlier op with the same cacheable constants in every row
};

// What is to hold in every row for a part of an op's RowScan to stand.  The rows
// are looked through by the host, or by the GPU once the table is there
// (check_rows_kernel).
struct RowCheck {
  enum : int { PLAIN = 0, SAME, TWIN };
  int kind, op;
  int a, b, n;  // TWIN: n constants at a and at b; else the constant at a
};

UFO_HOST_DEV bool plain_strength(double k) {
  k = fabs(k);
  return k == 0.0 || (k > 1e-280 && k < 1e280);
}

UFO_HOST_DEV bool same_bits(double x, double y) {
  union { double d; uint64_t u; } p{x}, q{y};
  return p.u == q.u;
}

UFO_HOST_DEV bool check_row(const RowCheck &c, const double *row, const double *row0) {
  if (c.kind == RowCheck::PLAIN) return plain_strength(row[c.a]);
  if (c.kind == RowCheck::SAME) return row[c.a] == row0[c.a] && row[c.a + 1] == row0[c.a + 1];
  bool same = true;
  for (int k = 0; k < c.n; ++k) same = same && same_bits(row[c.a + k], row[c.b + k]);
  return same;
}

// The scan as the first row has it, and what to check in the rows.
inline std::vector<RowScan> scan_first_row(const int32_t *ops, int n_ops, const double *row0,
                                           std::vector<RowCheck> &checks) {
  std::vector<RowScan> scan(static_cast<size_t>(n_ops));
  std::unordered_multimap<uint64_t, int> seen;  // constants -> op
  auto word = [&](int i) { return ops + static_cast<size_t>(i) * UFO_OP_WORDS; };
  for (int i = 0; i < n_ops; ++i) {
    const int32_t *w = word(i);
    RowScan &s = scan[static_cast<size_t>(i)];
    if (w[0] == OP_KICK ||
        (w[0] == OP_TEAPOT && !(w[1] & (F_YOSHIDA | F_EXACT)))) {
      const bool teapot = w[0] == OP_TEAPOT;
      const bool div = teapot && w[3] > 1 && ((w[1] >> SH_FINNER) & 3) == DF_DIV;
      const int pattern = kick_pattern(w[teapot ? 4 : 3], w[teapot ? 5 : 4], w[teapot ? 6 : 5]);
      if (pattern == 1 || pattern == 2) {  // a short form's strength
        const int at = w[2] + (!teapot ? 0 : w[3] <= 1 ? 1 : div ? 5 : 2);
        checks.push_back({RowCheck::PLAIN, i, at, 0, 1});
      }
      if (div) checks.push_back({RowCheck::SAME, i, w[2] + 2, 0, 2});  // [d, 1/d]
    } else if (w[0] == OP_THICKQ || w[0] == OP_THICKB ||
               (w[0] == OP_EDGE && (w[1] & F_RTPSI))) {
      const int n = static_cast<int>(op_consts(w));
      uint64_t h = 1469598103934665603ull ^ static_cast<uint64_t>(w[0] * 31 + w[1]);
      for (int k = 0; k < n; ++k) {
        uint64_t bits;
        std::memcpy(&bits, row0 + w[2] + k, sizeof bits);
        h = (h ^ bits) * 1099511628211ull;
        h ^= h >> 29;
      }
      const auto range = seen.equal_range(h);
      for (auto it = range.first; it != range.second && s.twin < 0; ++it) {
        const int32_t *v = word(it->second);
        if (v[0] == w[0] && v[1] == w[1] &&
            check_row({RowCheck::TWIN, i, v[2], w[2], n}, row0, row0))
          s.twin = it->second;
      }
      if (s.twin < 0)
        seen.emplace(h, i);
      else
        checks.push_back({RowCheck::TWIN, i, word(s.twin)[2], w[2], n});
    }
  }
  return scan;
}

// Row by row (check by check, each look misses the cache: 20,000 rows of 833 ops
// took 170 ms more); `bad`: one byte per check, set where a row fails it.
inline void check_rows(const std::vector<RowCheck> &checks, const double *table, int64_t stride,
                       int n_seeds, std::vector<unsigned char> &bad) {
  bad.assign(checks.size(), 0);
  for (int r = 0; r < n_seeds; ++r)
    for (size_t k = 0; k < checks.size(); ++k)
      if (!bad[k]) bad[k] = !check_row(checks[k], table + static_cast<int64_t>(r) * stride, table);
}

inline void apply_checks(const std::vector<RowCheck> &checks,
                         const std::vector<unsigned char> &bad, std::vector<RowScan> &scan) {
  for (size_t k = 0; k < checks.size(); ++k) {
    if (!bad[k]) continue;
    RowScan &s = scan[static_cast<size_t>(checks[k].op)];
    if (checks[k].kind == RowCheck::PLAIN) s.plain = false;
    if (checks[k].kind == RowCheck::SAME) s.same = false;
    if (checks[k].kind == RowCheck::TWIN) s.twin = -1;
  }
}

struct PairLists {
  std::vector<PairOp> ops;  // the strict list, then at fma_at the FMA one
  size_t fma_at = 0;
  int n_ops = 0;            // public ops
  int cache_fields = 0;     // doubles per lane of the coefficient cache
  int wide[2] = {0, 0};     // entries run by the one-lane code, per list
  bool fma_ready = false;   // general kicks carry the series that FMA launches read
  bool general = false;     // most kicks are general
  bool thick = false;       // most magnets are thick
};

// where a list's cache-filling ops start
inline size_t pair_fill_at(int n_ops) { return 2 * static_cast<size_t>(n_ops) + 4; }

// Translate a validated opcode list for the two-lane kernel; false when an op
// is a Yoshida or exact-drift element, which would run as one-lane code on
// half-empty warps (a program has them everywhere or nowhere; pair_pays bounds
// the share of the other ops without a two-lane form).  Structurally empty ops
// (zero-angle edges) are left out: they matter to non-finite coordinates alone.
// Thick elements and fringe edges with the same constants in every row share
// their cache fields; at most `most_fields` are given out, and an element that
// gets none goes through the one-lane code, in a segment of its own.
inline bool decode_list(const int32_t *ops, int n_ops, const double *row0,
                        const std::vector<RowScan> &scan, int most_fields, bool fold_drifts,
                        PairLists &lists) {
  std::vector<PairOp> &out = lists.ops;
  int &cache_fields = lists.cache_fields, &wides = lists.wide[fold_drifts ? 0 : 1];
  cache_fields = wides = 0;
  lists.fma_ready = true;
  int kicks = 0, general = 0, thick = 0;
  std::vector<int> field_of(static_cast<size_t>(n_ops), -1);
  size_t head = 0;  // the current segment's header
  int64_t last_end = -1;  // where the constants of the last general teapot end
  auto open = [&](int first) {
    head = out.size();
    out.push_back({PV_SEGMENT, 0, first, first});
  };
  open(0);
  for (int i = 0; i < n_ops; ++i) {
    const int32_t *w = ops + static_cast<size_t>(i) * UFO_OP_WORDS;
    const int flags = w[1];
    const int common = (flags & F_ACHRO) ? PF_ACHRO : 0;
    PairOp op{PV_WIDE, w[2], i, 0};
    int fields = 0;
    bool keep = true;
    switch (w[0]) {
      case OP_NOP: keep = false; break;
      case OP_DRIFT:
        if (flags & F_EXACT) return false;
        op.head = w[3] == DF_MUL ? PV_DRIFT
                  : w[3] == DF_MUL2 ? PV_DRIFT2 : PV_DRIFT_DIV;
        break;
      case OP_KICK:
      case OP_TEAPOT: {
        const bool teapot = w[0] == OP_TEAPOT;
        const int32_t *k = w + (teapot ? 4 : 3);  // nn, ns, mn, ms
        const int pattern = (k[2] | k[3]) ? kick_pattern(k[0], k[1], k[2]) : 3;
        if (pattern == 0 && !(flags & F_PSER)) lists.fma_ready = false;
        ++kicks;
        general += pattern == 0;
        if (teapot && (flags & (F_EXACT | F_YOSHIDA))) return false;
        if (teapot && (((flags >> SH_FOUTER) & 3) != DF_MUL ||
                       ((flags >> SH_FINNER) & 3) == DF_MUL2))
          return false;
        if ((k[2] >> 16) || (k[3] >> 16)) break;  // orders above 15
        const bool div = teapot && w[3] > 1 && ((flags >> SH_FINNER) & 3) == DF_DIV;
        // the half and negative strengths formed on constants must be exact
        if (!scan[static_cast<size_t>(i)].plain) break;
        op.a = teapot ? w[3] : i;
        op.b = pattern == 0 ? k[2] | k[3] << 16 : 0;
        if (!teapot) {
          if (pattern == 3) keep = false;
          op.head = (PV_KICK + pattern) | common;
          break;
        }
        int form = DIV_NONE, shift = 0;
        bool negative = false;
        if (div) {
          form = DIV_GENERAL;
          const double *q = row0 + w[2] + 1;  // [A, d, 1/d, A/d]
          if (scan[static_cast<size_t>(i)].same) shift = shift_form(q[1], q[2], negative);
          if (shift) form = DIV_SHIFT;
        }
        op.head = (PV_TEAPOT + pattern + 4 * form + ((flags & F_WEAK) ? 12 : 0)) |
                  shift << 8 | (shift && negative ? PF_NEG : 0) | (div ? PF_DIV : 0) |
                  ((flags & F_SPLITO) ? PF_SPLITO : 0) | common |
                  ((flags & F_PSER) ? PF_PSER : 0);
        if (pattern == 0) {
          // the shift before a general teapot runs with it: see PF_PRE
          last_end = w[2] + op_consts(w);
          const PairOp &before = out.back();
          const int gap = w[2] - before.toff;
          if (out.size() - 1 > head && (before.head & 0xff) == PV_ALIGN &&
              !(before.head & PF_THEN) && (gap == 2 || gap == 5)) {
            op.head |= PF_PRE | (gap == 5 ? PF_PRE_EDGE : 0) |
                       (before.head & (PF_X | PF_Y));
            out.pop_back();
          }
        }
        break;
      }
      case OP_ALIGN:
        op.head = PV_ALIGN | ((flags & F_AX) ? PF_X : 0) |
                  ((flags & F_AY) ? PF_Y : 0);
        {  // the shift after a general teapot
          PairOp &before = out.back();
          const int variant = (before.head & 0xff) - PV_TEAPOT;
          const int planes = op.head & (PF_X | PF_Y);
          const int64_t gap = w[2] - last_end;
          if (out.size() - 1 > head && variant >= 0 && variant % 4 == 0 &&
              !(before.head & PF_POST) && (gap == 0 || gap == 3) &&
              (!(before.head & PF_PRE) ||
               (before.head & (PF_X | PF_Y)) == planes)) {
            before.head |= PF_POST | (gap == 3 ? PF_POST_EDGE : 0) | planes;
            keep = false;
          }
        }
        break;
      case OP_EDGE:
        keep = flags & (F_T1 | F_T2 | F_RTPSI);
        op.head = ((flags & F_RTPSI) ? PV_EDGE_PSI : PV_EDGE) | common |
                  ((flags & F_T1) ? PF_X : 0) | ((flags & F_T2) ? PF_Y : 0);
        if (flags & F_RTPSI) {
          if (!(flags & F_T2)) return false;
          fields = 1;
        }
        break;
      case OP_THICKQ:
      case OP_THICKB:
        op.head = (w[0] == OP_THICKQ ? PV_THICKQ : PV_THICKB) | common |
                  ((flags & F_CONST) ? PF_CONST : 0);
        fields = w[0] == OP_THICKQ ? TC_D : TC_FIELDS;
        ++thick;
        break;
      case OP_APERTURE:
        if (flags & F_CIRCLE) op.head = PV_CIRCLE;
        break;
      case OP_OBSERVE:
        op.head = PV_OBSERVE;
        op.a = w[3];
        break;
      case OP_LINEAR: op.head = PV_LINEAR; break;
      default: break;  // wires, dynamic kicks: the one-lane code
    }
    if (fields) {
      const int twin = scan[static_cast<size_t>(i)].twin;
      const int field = twin >= 0 ? field_of[static_cast<size_t>(twin)] : -1;
      op.a = field;
      if (field < 0 && fields <= most_fields - cache_fields) {
        op.a = cache_fields;
        op.head |= PF_FILL;
        cache_fields += fields;
      }
      field_of[static_cast<size_t>(i)] = op.a;
      if (op.a < 0) op = {PV_WIDE, w[2], i, 0};  // no room: by the one-lane code
    }
    // A plain drift goes with the op before it (strict list): an op of its own
    // costs its dispatch, about 200 cycles beside the 129 of its arithmetic.
    PairOp &before = out.back();
    const int variant = before.head & 0xff;
    if (fold_drifts && keep && op.head == PV_DRIFT && out.size() - 1 > head &&
        !(before.head & PF_THEN) &&
        (variant == PV_DRIFT || variant == PV_ALIGN || variant == PV_EDGE ||
         variant == PV_EDGE_PSI || variant == PV_THICKQ || variant == PV_THICKB ||
         (variant >= PV_TEAPOT && (variant - PV_TEAPOT) % 4 != 0))) {
      before.head |= PF_THEN;
      before.b = op.toff;
      keep = false;
    }
    // the kernel loads the constant at toff with the op, read or not
    if (op_consts(w) == 0) op.toff = 0;
    if (keep) {
      // an op without a two-lane form is a segment of its own
      const bool wide = op.head == PV_WIDE;
      const int kept = static_cast<int>(out.size() - 1 - head);
      if (kept > 0 && (wide || out.back().head == PV_WIDE || kept == PAIR_SEGMENT))
        open(i);
      out.push_back(op);
      wides += wide;
    }
    out[head].b = i + 1;
  }
  if (out[head].b > out[head].a) open(n_ops);  // the end
  out.push_back({PV_SEGMENT, 0, 0, 0});   // the kernel fetches two ops ahead
  out.push_back({PV_SEGMENT, 0, 0, 0});
  lists.general = 2 * general > kicks;
  lists.thick = thick > kicks;
  return true;
}

// Both lists, at fixed places whatever the constants make of them (a captured
// graph keeps their addresses): the second at `fma_at`, each padded to two
// entries per op -- every op a segment of its own -- and the ends, and followed
// by the ops that fill the cache (pair_fill walks those alone: one turn of three
// particles through 1,600 ops 997 us with the whole list, 893 us).
inline bool decode_pair(const int32_t *ops, int n_ops, const double *row0,
                        const std::vector<RowScan> &scan, int most_fields, PairLists &lists) {
  std::vector<PairOp> &out = lists.ops;
  out.clear();
  const size_t fill_at = pair_fill_at(n_ops);
  lists.n_ops = n_ops;
  lists.fma_at = fill_at + n_ops + 1;
  for (const bool strict : {true, false}) {
    const size_t start = out.size();
    if (!decode_list(ops, n_ops, row0, scan, most_fields, strict, lists)) return false;
    const size_t end = out.size();
    out.resize(start + fill_at);
    for (size_t i = start; i < end; ++i)
      if (out[i].head & PF_FILL) out.push_back(out[i]);
    out.resize(start + lists.fma_at);  // an end at least
  }
  return true;
}

// Which launches take the two-lane kernel (measured on one GB300, us per turn,
// one-lane kernel -> two-lane kernel; 152 SMs, 16 particles per warp):
//  strict arithmetic: always.  Its operations come in pairs of planes, so the
//   two-lane form issues no more of them at any size, and the constant division
//   and the coefficient cache shorten it: FODO ring (128 elements) 1,024
//   particles 167 -> 61, 65,536 particles 475 -> 382; light-source ring (1,024)
//   65,536 particles 5,352 -> 4,273; thick 768-element ring, 1,000 particles
//   1,355 -> 318, 65,536 particles 4,481 -> 1,765.
//   A ring with general error kicks on most magnets (a coefficient enters one
//   lane's sum, so half its products are idle) gains up to 12 warps per SM:
//   light-source ring with errors 1,000 particles 15,590 -> 8,480, 20,500 to
//   24,000 18,770 -> 19,230 (a third warp on some sub-partitions), 29,184 20,240
//   -> 19,310, 30,000 even.
//  FMA: up to 9 warps per SM; where most kicks are general 13, or 11 if a row of
//   constants passes 64 KB, which the two-lane kernel's warps, twice as many, read
//   every turn.  The sextupole form and the composed linear elements cost the
//   two-lane code more instructions (6 for 5, 8 for 5 per 32 particles), so the
//   one-lane kernel wins once its pipe is full: light-source ring 333 particles
//   652 -> 345, 20,000 (8.2 warps per SM) 699 -> 615, 21,888 755 -> 772, 24,000
//   (9.9) 705 -> 770; FODO ring with errors on every magnet 1,000 346 -> 192,
//   31,616 (13) 435 -> 412, 34,000 (14) 435 -> 443; light-source ring with errors
//   (161 KB) 27,000 (11.1) 3,960 -> 3,740, 29,184 (12) 3,960 -> 4,250, 33,000
//   4,240 -> 4,370.
//  Dynamic-aperture scans of such a ring that nobody tuned: always.  Where few
//  survive the refill of twice as many, half-size warps wins (196,608 particles,
//  128 turns, ms: 15 % survive 87.5 -> 64.9); where most do it costs up to 5 %
//  (31 % 119 -> 123, 66 % 225 -> 236), which a launch cannot know beforehand.  A
//  tuned scan (StableAperture's second phase, of survivors) goes by its size.
//  Uneven turn counts on such a ring: strict always; FMA up to 44 warps per SM.
//   The last, longest particles run in few warps, and twice as many half-size
//   warps leave the queue more evenly: error seeds of 64 to 256 turns, ms, 39,967
//   particles 122 -> 99, 79,967 185 -> 148, 99,966 205 -> 189, but 119,968 219 ->
//   222 and 159,879 295 -> 307; of 1,000 to 4,096 turns / 32, 1,145,971 particles
//   1,013 -> 1,082 (strict 5,892 -> 5,887).
//  Few ops without a two-lane form (wires, general apertures, dynamic kicks,
//   orders above 15, elements without room in the cache): each is a segment that
//   both lanes of a pair compute in full, twice the FP64 instructions of the one-
//   lane kernel.  The share that still pays falls with the warps per SM (FODO
//   ring with a rectangular aperture, or a wire, after every k-th magnet, strict;
//   share of ops, particles): 14 %, 12,000 270 -> 227, 278 -> 260; 8 %, 16,000
//   236 -> 171, 245 -> 212; 8 %, 30,000 299 -> 301, 339 -> 402; 2 %, 65,536
//   490 -> 434, 523 -> 492; but 25 %, 65,536 675 -> 1,034, 1,210 -> 1,929.  FMA 5 %,
//   16,000 65 -> 49, 67 -> 58, 20,000 65 -> 73, 70 -> 84.  General magnets and
//   thick elements, the longer part of their turn, bear more: errors on every
//   magnet, FMA 17 %, 16,000 584 -> 511, 24,000 613 -> 761; thick ring 24 %, 1,000
//   2,246 -> 1,558, 16,000 2,397 -> 1,856, 24,000 2,554 -> 2,641.
struct PairUse {
  int64_t n;
  int sm_count;
  bool fma, uneven, untuned_scan;
  int64_t row_bytes;  // constants of one seed
};

// the least ops per op without a two-lane form; 0: none may be
inline int least_ops_per_wide(const PairLists &p, const PairUse &u, int64_t groups) {
  const int64_t sms = u.sm_count;
  if (p.thick) return groups <= 8 * sms ? 4 : 5;
  if (p.general) return groups <= 8 * sms ? 5 : 32;
  if (groups <= 5 * sms) return u.fma ? 8 : 6;
  if (groups <= 8 * sms) return u.fma ? 12 : 10;
  return u.fma ? 0 : 32;
}

inline bool pair_pays(const PairLists &p, const PairUse &u) {
  if (u.fma && !p.fma_ready) return false;
  const int64_t groups = (u.n + 15) / 16;
  const int64_t wide = p.wide[u.fma ? 1 : 0];
  const int per_wide = least_ops_per_wide(p, u, groups);
  if (wide && (!per_wide || p.n_ops < per_wide * wide)) return false;
  if (!u.fma && !p.general) return true;
  if (p.general && (u.untuned_scan || (u.uneven && !u.fma))) return true;
  const int most = !p.general ? 9 : !u.fma ? 12 : u.uneven ? 44 : u.row_bytes <= 65536 ? 13 : 11;
  return groups <= most * static_cast<int64_t>(u.sm_count);
}
// Resident warps per SM of the two-lane kernel, 16 particles each: the tuning
// counts warps of the one-lane kernel, so twice as many, at most the 16 that the
// registers allow.  A dynamic-aperture scan that nobody tuned gets 8 when it has
// more than 10 per SM: most of its particles are lost in the first turns, and
// lanes that refill from a longer queue stay fuller, while two warps per sub-
// partition still fill most of the FP64 pipe.  FODO ring with errors, strict, 24
// turns (ms with 8, 16, and on the one-lane kernel): 21 % survive, 24,000
// particles 30, 37, 47, 30,000 34, 54, 53, 49,152 35, 68, 72.  If nearly all
// survive the queue is a second round, which up to 10 per SM would cost more than
// the refill can gain: 20,000 53, 39, 47, 24,000 54, 41, 50, 30,000 62, 57, 58,
// 36,864 63, 65, 65, 49,152 92, 87, 85.
inline int pair_warps_per_sm(int64_t n, int sm_count, int tuning, bool untuned_scan) {
  const int64_t groups = (n + 15) / 16;
  return untuned_scan && groups > 10 * static_cast<int64_t>(sm_count) ? 8
                                                                      : std::min(16, 2 * tuning);
}

// Time slices (Slices in pair.cuh) for a two-lane launch of equal turns with
// more groups of 16 particles than 8 warps per SM: as many warps as fill every
// sub-partition evenly (a multiple of 4 per SM) and leave groups in hand.  Below
// that a sub-partition's first and second warp hide each other's latency, so an
// uneven second one costs nothing.  Measured (us per turn, strict, without ->
// with): FODO ring 65,536 particles 434 -> 379, light-source ring 4,991 -> 4,259,
// thick ring 1,948 -> 1,777, 30,000 particles of the FODO ring 182 -> 175.  The
// one-lane kernel keeps whole runs: the 12 warps per SM that leave it groups in
// hand cost it more than the even end gains (FMA, light-source ring 1,511 ->
// 1,685).
// At most 32 groups per SM.  A slice's group keeps its lanes, lost or not, while
// a lane of a whole run takes the next particle: beams of which a part is lost
// run longer in slices, and up to here (where the one-lane kernel holds them all
// at once and refills nothing either) never longer than on that kernel.  Light-
// source ring, 30 turns (ms: slices, whole runs, one-lane kernel): 77,824
// particles of which 14 % survive 141, 79, 183, none lost 151, 150, 180; 262,144
// particles 469, 122, 210 and 510, 524, 629; thick ring, 40 turns, 262,144
// particles, 3 % survive 120, 52, 224.
struct SlicePlan {
  int groups = 0;  // 0: whole runs
  int count = 0, turns = 0;  // slices per group, turns per slice
  int warps_per_sm = 0;
};

inline SlicePlan slice_plan(int64_t n, int turns, int n_ops, int sm_count, int most_warps,
                            int64_t most_groups) {
  SlicePlan s;
  const int64_t groups = (n + 15) / 16;
  const int64_t w = std::min<int64_t>(most_warps, (groups - 1) / sm_count) / 4 * 4;
  if (turns < 2 || w < 8 || groups > std::min<int64_t>(most_groups, 32 * sm_count)) return s;
  s.groups = static_cast<int>(groups);
  // slice length: a launch ends within about half a slice (a share of Q / 2T),
  // and each slice costs about 5 us of exchange against some 0.6 us per op and
  // turn: the sum is least near Q = sqrt(16 T / ops)
  s.turns = std::max(1, static_cast<int>(std::sqrt(16.0 * turns / std::max(1, n_ops))));
  // in 64 bits: turns near INT_MAX mean "until all are lost"
  s.count = static_cast<int>((static_cast<int64_t>(turns) + s.turns - 1) / s.turns);
  s.warps_per_sm = static_cast<int>(w);
  return s;
}

}  // namespace ufo
