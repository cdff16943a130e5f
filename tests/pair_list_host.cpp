// The two-lane kernel's host side behind a C interface, for tests on the CPU.
#include <algorithm>

#include "../ufo_gb300/csrc/pair_list.h"

extern "C" {

// The lists of decode_pair, four words per entry.  info: accepted, entries,
// start of the FMA list, cache fields, FMA lists usable, most kicks general.
int pair_lists(const int32_t *ops, int n_ops, const double *table, int64_t stride, int n_seeds,
               int most_fields, int32_t *out, int64_t capacity, int64_t *info) {
  std::vector<ufo::PairOp> list;
  size_t fma_at = 0;
  int fields = 0;
  bool fma = false, general = false;
  const bool ok = ufo::decode_pair(ops, n_ops, table, stride, n_seeds, most_fields, list, fma_at,
                                   fields, fma, general);
  info[0] = ok;
  info[1] = static_cast<int64_t>(list.size());
  info[2] = static_cast<int64_t>(fma_at);
  info[3] = fields;
  info[4] = fma;
  info[5] = general;
  if (static_cast<int64_t>(list.size()) * 4 > capacity) return -1;
  std::memcpy(out, list.data(), sizeof(ufo::PairOp) * list.size());
  return 0;
}

}  // extern "C"
