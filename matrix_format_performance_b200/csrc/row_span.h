// The rows whose elements start at a position of a row-sorted element list.
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define MFP_HD __host__ __device__
#else
#define MFP_HD
#endif

namespace mfp {

// [first, end): 64 bits, since `end` is rows + 1 for the closing position and
// a matrix may have 2^32 - 1 rows.
struct row_span {
  uint64_t first, end;
};

// Position p of nnz elements with sorted row ids: the rows after the element
// before it (`prev`, unused at p = 0) up to its own row `cur`; at p = nnz, up to
// row_ptr's last entry, rows (`cur` unused).
MFP_HD inline row_span rows_starting_at(uint64_t p, uint64_t nnz, uint32_t prev, uint32_t cur, uint32_t rows) {
  return {p ? (uint64_t)prev + 1u : 0u, (uint64_t)(p < nnz ? cur : rows) + 1u};
}

}  // namespace mfp
