// The two-lane kernel's host side behind a C interface, for tests on the CPU.
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

// groups, slices per group, turns per slice, warps per SM
void pair_slices(int64_t n, int turns, int n_ops, int sm_count, int most_warps,
                 int64_t most_groups, int64_t *out) {
  const ufo::SlicePlan p = ufo::slice_plan(n, turns, n_ops, sm_count, most_warps, most_groups);
  out[0] = p.groups;
  out[1] = p.count;
  out[2] = p.turns;
  out[3] = p.warps_per_sm;
}

}  // extern "C"
