// row_span.h at the ends of its range: every entry of a row_ptr is written once,
// and the closing position of 2^32 - 1 rows ends.
#include <cstdio>
#include <vector>

#include "../../matrix_format_performance_b200/csrc/row_span.h"

static bool covers(uint32_t rows, const std::vector<uint32_t> &ids) {
  uint64_t next = 0;
  for (uint64_t p = 0; p <= ids.size(); ++p) {
    const mfp::row_span s =
        mfp::rows_starting_at(p, ids.size(), p ? ids[p - 1] : 0u, p < ids.size() ? ids[p] : 0u, rows);
    if (s.first != next || s.end < s.first) return false;
    next = s.end;
  }
  return next == (uint64_t)rows + 1u;
}

int main() {
  const uint32_t most = 0xffffffffu;
  const bool ok = covers(1, {0}) && covers(5, {0, 0, 3}) && covers(5, {4}) && covers(most, {0}) &&
                  covers(most, {0, 7, most - 1u}) && covers(most, {most - 1u, most - 1u});
  std::printf(ok ? "ok\n" : "FAILED\n");
  return ok ? 0 : 1;
}
