// Aligned quads of a CSR's elements.
#pragma once

#include <cstdint>

#if !defined(MFP_HD)
#if defined(__CUDACC__)
#define MFP_HD __host__ __device__
#else
#define MFP_HD
#endif
#endif

namespace mfp {

// Whether the quad from element e < nnz on lies within the nnz elements (e + 4
// wraps at the end of 2^32 - 1 elements).
MFP_HD inline bool whole_quad(uint32_t e, uint32_t nnz) { return nnz - e >= 4u; }

}  // namespace mfp
