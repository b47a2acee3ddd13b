// quads.h for every remainder of the last quad, up to 2^32 - 1 elements.
#include <cstdio>
#include <initializer_list>

#include "../../matrix_format_performance_b200/csrc/quads.h"

int main() {
  bool ok = true;
  for (uint64_t nnz : {1ull, 3ull, 4ull, 5ull, 1000ull, 0xfffffffcull, 0xfffffffdull, 0xfffffffeull, 0xffffffffull})
    for (uint64_t e = nnz > 64 ? (nnz - 60) & ~3ull : 0; e < nnz; e += 4)
      ok = ok && mfp::whole_quad((uint32_t)e, (uint32_t)nnz) == (e + 4 <= nnz);
  std::printf(ok ? "ok\n" : "FAILED\n");
  return ok ? 0 : 1;
}
