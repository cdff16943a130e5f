// opcodes.h -- the opcode table's words, and how many constants an op reads
// (host and device; no CUDA).
#pragma once
#include <cstdint>

namespace ufo {

enum : int {
  OP_NOP = 0, OP_DRIFT, OP_KICK, OP_TEAPOT, OP_ALIGN, OP_EDGE, OP_THICKQ, OP_THICKB, OP_WIRE,
  OP_APERTURE, OP_OBSERVE, OP_DYNKICK, OP_LINEAR
};
enum : int { DF_MUL = 0, DF_MUL2 = 1, DF_DIV = 2 };
enum : int {
  F_ACHRO = 1 << 0, F_EXACT = 1 << 1, F_WEAK = 1 << 2, F_RTPSI = 1 << 3, F_T1 = 1 << 4,
  F_T2 = 1 << 5, F_CONST = 1 << 6, F_AX = 1 << 7, F_AY = 1 << 8, F_T1Z = 1 << 9,
  F_T2Z = 1 << 10, F_WEAKZ = 1 << 11, F_YOSHIDA = 1 << 12, F_CIRCLE = 1 << 13, F_SPLITO = 1 << 14,
  F_PSER = 1 << 15
};
constexpr int SH_FOUTER = 16, SH_FINNER = 18;

struct Op {
  int kind, flags, toff, i0, i1, i2, i3, i4;
};

inline int popc32(uint32_t v) { return __builtin_popcount(v); }

inline bool mask_fits(int n, int32_t mask) {
  if (n < 0 || n > 32) return false;
  const uint32_t m = static_cast<uint32_t>(mask);
  return n == 32 || (m >> n) == 0u;
}

// constants of the dense power series of a general kick (F_PSER): 2 per
// order up to the highest coefficient; -1 if the flag is set without one
inline int64_t pser_consts(int flags, int32_t mn, int32_t ms) {
  if (!(flags & F_PSER)) return 0;
  const uint32_t m = static_cast<uint32_t>(mn) | static_cast<uint32_t>(ms);
  if (m == 0u) return -1;
  return 2 * static_cast<int64_t>(32 - __builtin_clz(m));
}

inline int drift_consts(int form, bool exact) {
  if (exact) return 1;
  return form == DF_MUL ? 1 : form == DF_MUL2 ? 2 : form == DF_DIV ? 4 : -1;
}

// Number of table constants an op reads (exactly what the kernels read), or
// -1 if the op's shape is invalid.  Every op must fit inside the stride so
// that no kernel read leaves its seed's row.
inline int64_t op_consts(const int32_t *w) {
  const int kind = w[0], flags = w[1];
  const bool exact = flags & F_EXACT;
  switch (kind) {
    case OP_NOP:
    case OP_OBSERVE:
      return 0;
    case OP_DRIFT:
      return drift_consts(w[3], exact);
    case OP_KICK: {
      if (!mask_fits(w[3], w[5]) || !mask_fits(w[4], w[6])) return -1;
      const int64_t ps = pser_consts(flags, w[5], w[6]);
      if (ps < 0) return -1;
      return popc32(w[5]) + popc32(w[6]) + ps;
    }
    case OP_TEAPOT: {
      const int64_t ps = pser_consts(flags, w[6], w[7]);
      if (ps < 0) return -1;
      if (flags & F_YOSHIDA) {  // [4 drifts][3 weights][kick][W][series]
        if (exact || w[3] < 1 || !mask_fits(w[4], w[6]) || !mask_fits(w[5], w[7])) return -1;
        return 7 + popc32(w[6]) + popc32(w[7]) + ((flags & F_WEAK) ? 1 : 0) + ps;
      }
      if (w[3] < 1 || !mask_fits(w[4], w[6]) || !mask_fits(w[5], w[7])) return -1;
      if ((flags & F_PSER) && exact) return -1;
      const int fo = (flags >> SH_FOUTER) & 3, fi = (flags >> SH_FINNER) & 3;
      const int co = drift_consts(fo, exact), ci = w[3] > 1 ? drift_consts(fi, exact) : 0;
      if (co < 0 || ci < 0) return -1;
      return co + ci + popc32(w[6]) + popc32(w[7]) + ((flags & F_WEAK) ? 1 : 0) +
             ((flags & F_SPLITO) ? 1 : 0) + ps;
    }
    case OP_ALIGN:
      return 2;
    case OP_EDGE:
      return (flags & F_RTPSI) ? 6 : 3;
    case OP_THICKQ:
      return (flags & F_CONST) ? 7 : 2;
    case OP_THICKB:
      return (flags & F_CONST) ? 16 : 3;
    case OP_WIRE:
      return 3;
    case OP_APERTURE:
      if (flags & F_CIRCLE) return 1;
      return w[3] >= 0 ? 2 * static_cast<int64_t>(w[3]) : -1;
    case OP_DYNKICK:
      if (w[3] < 0 || w[4] < 0 || w[3] > 32 || w[4] > 32 || w[5] < w[3] + w[4]) return -1;
      return w[5];
    case OP_LINEAR:
      return 5;
    default:
      return -1;
  }
}

}  // namespace ufo
