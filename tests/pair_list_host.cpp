// The two-lane kernel's host side behind a C interface, for tests on the CPU.
#include "../ufo_gb300/csrc/pair_list.h"

extern "C" {

// The lists of decode_pair, four words per entry.  info: accepted, entries,
// start of the FMA list, cache fields, FMA lists usable, most kicks general,
// entries run by the one-lane code in the strict and the FMA list.
int pair_lists(const int32_t *ops, int n_ops, const double *table, int64_t stride, int n_seeds,
               int most_fields, int32_t *out, int64_t capacity, int64_t *info) {
  ufo::PairLists p;
  std::vector<ufo::RowCheck> checks;
  std::vector<unsigned char> bad;
  std::vector<ufo::RowScan> scan = ufo::scan_first_row(ops, n_ops, table, checks);
  ufo::check_rows(checks, table, stride, n_seeds, bad);
  ufo::apply_checks(checks, bad, scan);
  info[0] = ufo::decode_pair(ops, n_ops, table, scan, most_fields, p);
  info[1] = static_cast<int64_t>(p.ops.size());
  info[2] = static_cast<int64_t>(p.fma_at);
  info[3] = p.cache_fields;
  info[4] = p.fma_ready;
  info[5] = p.general;
  info[6] = p.wide[0];
  info[7] = p.wide[1];
  if (static_cast<int64_t>(p.ops.size()) * 4 > capacity) return -1;
  std::memcpy(out, p.ops.data(), sizeof(ufo::PairOp) * p.ops.size());
  return 0;
}

// Whether a launch of n particles of such lists takes the two-lane kernel.
int pair_use(int n_ops, int wide, int thick, int general, int64_t n, int sm_count, int fma,
             int uneven, int scan, int64_t row_bytes) {
  ufo::PairLists p;
  p.n_ops = n_ops;
  p.wide[0] = p.wide[1] = wide;
  p.thick = thick != 0;
  p.general = general != 0;
  p.fma_ready = true;
  return ufo::pair_pays(p, {n, sm_count, fma != 0, uneven != 0, scan != 0, row_bytes});
}

int pair_resident(int64_t n, int sm_count, int tuning, int scan) {
  return ufo::pair_warps_per_sm(n, sm_count, tuning, scan != 0);
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
