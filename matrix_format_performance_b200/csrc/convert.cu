// On-device format conversion: the reference's host converters
// (common/matrix_converter.cpp, common/scoo_matrix_class.cpp) as CUDA kernels
// over device arrays.  Every output array is identical, element for element,
// to the host converters in formats.cpp (and so to the reference's).
//
// Building blocks:
//   - an exclusive scan of a per-item count (row lengths, tail lengths, radix
//     histograms): block sums, one CTA over the block sums, block-local scans;
//   - a row expansion for COO-shaped outputs: a 2048-element output tile marks
//     the first position of every row that starts inside it with the row id,
//     then an inclusive max-scan over the tile gives each position its row
//     (empty rows never mark a position, long rows span tiles);
//   - a stable LSD radix sort (digits of up to 9 bits, one launch per digit:
//     tiles rank their keys, look back for the counts of the tiles before them
//     and scatter) for COO triplets -> CSR on the composite key (row, column).
#include "host_common.h"
#include "row_span.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <vector>

using namespace mfp;

namespace {

constexpr uint32_t kThreads = 256;
constexpr uint32_t kWarps = kThreads / 32;
constexpr uint32_t kItems = 8;
constexpr uint32_t kTile = kThreads * kItems;  // items per CTA in scans and expansions
constexpr uint32_t kRadixThreads = 512;
constexpr uint32_t kRadixWarps = kRadixThreads / 32;
constexpr uint32_t kRadixRounds = 12;
constexpr uint32_t kRadixTile = kRadixThreads * kRadixRounds;  // keys per CTA in a radix pass
constexpr uint32_t kRadixBits = 9;                             // widest digit
constexpr uint32_t kRadixBins = 1u << kRadixBits;
static_assert(kRadixBins == kRadixThreads, "one thread per digit");
constexpr uint32_t kRadixPasses = 8;                      // 64-bit keys
constexpr uint32_t kRadixPolls = 1u << 20;                // look-back limit, about a second
constexpr uint32_t kStop = 0x80000000u;                   // in a tile counter: no more tiles

int cuda_fail(cudaError_t e, const char *what) {
  return fail(MFP_ERROR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}
#define CV_TRY(expr, what)                               \
  do {                                                   \
    cudaError_t _e = (expr);                             \
    if (_e != cudaSuccess) return cuda_fail(_e, what);   \
  } while (0)

inline cudaStream_t as_stream(void *s) { return reinterpret_cast<cudaStream_t>(s); }
inline uint32_t blocks_for(uint64_t n, uint64_t per) { return (uint32_t)((n + per - 1) / per); }
inline uint32_t bits_for(uint32_t x) { return x ? 32u - (uint32_t)__builtin_clz(x) : 0u; }

// shared-memory index with one pad word per 32 (conflict-free strided reads)
__device__ __forceinline__ uint32_t pad(uint32_t i) { return i + (i >> 5); }

__device__ __forceinline__ uint32_t warp_incl_sum(uint32_t v) {
  const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
  for (uint32_t o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}
__device__ __forceinline__ uint32_t warp_incl_max(uint32_t v) {
  const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
  for (uint32_t o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v = max(v, t);
  }
  return v;
}

// Exclusive block prefix (sum or max) of one value per thread; *total gets the
// block's reduction.  s holds kWarps words.
template <bool MAX>
__device__ __forceinline__ uint32_t block_excl(uint32_t v, uint32_t *s, uint32_t *total) {
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  const uint32_t inc = MAX ? warp_incl_max(v) : warp_incl_sum(v);
  if (lane == 31) s[w] = inc;
  __syncthreads();
  if (w == 0) {
    uint32_t t = lane < kWarps ? s[lane] : 0u;
    t = MAX ? warp_incl_max(t) : warp_incl_sum(t);
    if (lane < kWarps) s[lane] = t;
  }
  __syncthreads();
  const uint32_t before = w ? s[w - 1] : 0u;
  if (total) *total = s[kWarps - 1];
  __syncthreads();
  if (MAX) {
    const uint32_t ex = __shfl_up_sync(0xffffffffu, inc, 1);
    return max(before, lane ? ex : 0u);
  }
  return before + inc - v;
}

// ---------------------------------------------------------------------------
// Exclusive scan of f(i), i in [0, n): out[0..n], out[n] = the total.
// ---------------------------------------------------------------------------
// in-row positions >= start of row i (coo_matrix_class tail, matrix_converter.cpp:242-257)
struct f_tail {
  const uint32_t *rp;
  uint32_t start;
  __device__ uint32_t operator()(uint32_t i) const {
    const uint32_t len = rp[i + 1] - rp[i];
    return len > start ? len - start : 0u;
  }
};

template <typename F>
__global__ void __launch_bounds__(kThreads) scan_reduce_kernel(uint32_t n, F f, uint32_t *sums) {
  __shared__ uint32_t s[kWarps];
  const uint64_t base = (uint64_t)blockIdx.x * kTile;
  uint32_t acc = 0;
#pragma unroll
  for (uint32_t j = 0; j < kItems; ++j) {
    const uint64_t i = base + j * kThreads + threadIdx.x;
    if (i < n) acc += f((uint32_t)i);
  }
  uint32_t total;
  block_excl<false>(acc, s, &total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// One CTA: sums[0..nb) -> exclusive offsets in place; *grand = the total.
__global__ void __launch_bounds__(kThreads) scan_sums_kernel(uint32_t nb, uint32_t *sums, uint32_t *grand) {
  __shared__ uint32_t s[kWarps];
  uint32_t carry = 0;
  for (uint32_t b0 = 0; b0 < nb; b0 += kThreads) {
    const uint32_t i = b0 + threadIdx.x;
    const uint32_t v = i < nb ? sums[i] : 0u;
    uint32_t total;
    const uint32_t ex = block_excl<false>(v, s, &total);
    if (i < nb) sums[i] = carry + ex;
    carry += total;
  }
  if (threadIdx.x == 0) *grand = carry;
}

template <typename F>
__global__ void __launch_bounds__(kThreads) scan_apply_kernel(uint32_t n, F f, const uint32_t *offsets,
                                                              uint32_t *out) {
  __shared__ uint32_t tile[kTile + kTile / 32];
  __shared__ uint32_t s[kWarps];
  const uint64_t base = (uint64_t)blockIdx.x * kTile;
#pragma unroll
  for (uint32_t j = 0; j < kItems; ++j) {
    const uint32_t p = j * kThreads + threadIdx.x;
    tile[pad(p)] = base + p < n ? f((uint32_t)(base + p)) : 0u;
  }
  __syncthreads();
  uint32_t v[kItems], acc = 0;
#pragma unroll
  for (uint32_t k = 0; k < kItems; ++k) {
    v[k] = acc;
    acc += tile[pad(threadIdx.x * kItems + k)];
  }
  const uint32_t ex = block_excl<false>(acc, s, nullptr) + offsets[blockIdx.x];
#pragma unroll
  for (uint32_t k = 0; k < kItems; ++k) tile[pad(threadIdx.x * kItems + k)] = ex + v[k];
  __syncthreads();
#pragma unroll
  for (uint32_t j = 0; j < kItems; ++j) {
    const uint32_t p = j * kThreads + threadIdx.x;
    if (base + p < n) out[base + p] = tile[pad(p)];
  }
}

// Scratch comes from a per-device memory pool private to the converters.  Its
// release threshold is unlimited, so freed scratch stays mapped for the next
// conversion (the device's default pool would hand it back to the driver at
// every synchronisation and map it again on the next call, which costs
// milliseconds per GB); mfp_dev_scratch_release returns it.
std::mutex g_pool_mu;
std::map<int, cudaMemPool_t> g_pools;

int scratch_pool(cudaMemPool_t *out) {
  int dev = 0;
  CV_TRY(cudaGetDevice(&dev), "cudaGetDevice");
  std::lock_guard<std::mutex> lk(g_pool_mu);
  auto it = g_pools.find(dev);
  if (it != g_pools.end()) {
    *out = it->second;
    return MFP_SUCCESS;
  }
  cudaMemPoolProps props{};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  cudaMemPool_t pool;
  CV_TRY(cudaMemPoolCreate(&pool, &props), "cudaMemPoolCreate");
  uint64_t keep = UINT64_MAX;
  CV_TRY(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep), "cudaMemPoolSetAttribute");
  g_pools[dev] = pool;
  *out = pool;
  return MFP_SUCCESS;
}

// Scratch that lives for one converter call, freed in stream order.
struct scratch {
  cudaStream_t st;
  cudaMemPool_t pool = nullptr;
  std::vector<void *> ptrs;
  explicit scratch(cudaStream_t s) : st(s) {}
  ~scratch() {
    for (void *p : ptrs) cudaFreeAsync(p, st);
  }
  template <typename T>
  int get(T **p, size_t count) {
    *p = nullptr;
    if (!count) return MFP_SUCCESS;
    if (!pool) {
      const int s = scratch_pool(&pool);
      if (s) return s;
    }
    void *q = nullptr;
    CV_TRY(cudaMallocFromPoolAsync(&q, count * sizeof(T), pool, st), "cudaMallocFromPoolAsync");
    ptrs.push_back(q);
    *p = static_cast<T *>(q);
    return MFP_SUCCESS;
  }
};

template <typename F>
int exclusive_scan(uint32_t n, F f, uint32_t *out, scratch &sc) {
  if (n == 0) {
    CV_TRY(cudaMemsetAsync(out, 0, sizeof(uint32_t), sc.st), "cudaMemsetAsync");
    return MFP_SUCCESS;
  }
  const uint32_t nb = blocks_for(n, kTile);
  uint32_t *sums = nullptr;
  int st = sc.get(&sums, nb);
  if (st) return st;
  scan_reduce_kernel<F><<<nb, kThreads, 0, sc.st>>>(n, f, sums);
  scan_sums_kernel<<<1, kThreads, 0, sc.st>>>(nb, sums, out + n);
  scan_apply_kernel<F><<<nb, kThreads, 0, sc.st>>>(n, f, sums, out);
  CV_TRY(cudaGetLastError(), "scan launch");
  return MFP_SUCCESS;
}

// ---------------------------------------------------------------------------
// Row expansion: output element j in [0, total) belongs to the row r with
// tp[r] <= j < tp[r+1] and copies source element rp[r] + start + (j - tp[r]).
// With tp == rp and start == 0 (plain COO / SCOO) the values and columns are
// the CSR arrays themselves, copied whole; only the row ids are written here.
// ---------------------------------------------------------------------------
// tr[i] = the row holding output position i * kTile (i < ntiles) or total - 1
// (i = ntiles): the largest r < rows with tp[r] <= pos.
__global__ void __launch_bounds__(kThreads) tile_rows_kernel(uint32_t rows, uint32_t total, const uint32_t *tp,
                                                             uint32_t ntiles, uint32_t *tr) {
  const uint32_t i = blockIdx.x * kThreads + threadIdx.x;
  if (i > ntiles) return;
  const uint32_t pos = i < ntiles ? i * kTile : total - 1u;
  uint32_t lo = 0, hi = rows - 1;
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo + 1) / 2;
    if (tp[mid] <= pos) lo = mid; else hi = mid - 1;
  }
  tr[i] = lo;
}

template <typename T, bool COPY>
__global__ void __launch_bounds__(kThreads) expand_kernel(uint32_t total, const uint32_t *tr, const uint32_t *tp,
                                                          const uint32_t *rp, uint32_t start,
                                                          const uint32_t *__restrict__ cols,
                                                          const T *__restrict__ vals, T *__restrict__ od,
                                                          uint32_t *__restrict__ oc, uint32_t *__restrict__ orow) {
  __shared__ uint32_t s_row[kTile + kTile / 32];
  __shared__ uint32_t s[kWarps];
  const uint32_t j0 = blockIdx.x * kTile;
  const uint32_t n = min(kTile, total - j0);
  const uint32_t r0 = tr[blockIdx.x], r1 = tr[blockIdx.x + 1];
  for (uint32_t p = threadIdx.x; p < kTile; p += kThreads) s_row[pad(p)] = 0u;
  __syncthreads();
  // mark the first position of every row starting in this tile (r0 covers
  // position 0; rows up to r1 may start in the next tile and are skipped)
  for (uint32_t r = r0 + threadIdx.x; r <= r1 && r >= r0; r += kThreads) {
    const uint32_t b = tp[r], e = tp[r + 1];
    if (b < e && b < j0 + n) s_row[pad(max(b, j0) - j0)] = r;
  }
  __syncthreads();
  // inclusive max-scan over the tile: each position takes the last row mark
  uint32_t v[kItems], m = 0;
#pragma unroll
  for (uint32_t k = 0; k < kItems; ++k) {
    m = max(m, s_row[pad(threadIdx.x * kItems + k)]);
    v[k] = m;
  }
  const uint32_t before = block_excl<true>(m, s, nullptr);
#pragma unroll
  for (uint32_t k = 0; k < kItems; ++k) s_row[pad(threadIdx.x * kItems + k)] = max(before, v[k]);
  __syncthreads();
  // all loads of a thread are issued before its stores
  uint32_t src[kItems];
#pragma unroll
  for (uint32_t k = 0; k < kItems; ++k) {
    const uint32_t p = k * kThreads + threadIdx.x;
    v[k] = p < n ? s_row[pad(p)] : 0u;
    if (COPY) src[k] = p < n ? rp[v[k]] + start + (j0 + p - tp[v[k]]) : 0u;
  }
  if (COPY) {
    T dv[kItems];
    uint32_t dc[kItems];
#pragma unroll
    for (uint32_t k = 0; k < kItems; ++k)
      if (k * kThreads + threadIdx.x < n) {
        dv[k] = vals[src[k]];
        dc[k] = cols[src[k]];
      }
#pragma unroll
    for (uint32_t k = 0; k < kItems; ++k)
      if (k * kThreads + threadIdx.x < n) {
        od[j0 + k * kThreads + threadIdx.x] = dv[k];
        oc[j0 + k * kThreads + threadIdx.x] = dc[k];
      }
  }
#pragma unroll
  for (uint32_t k = 0; k < kItems; ++k) {
    const uint32_t p = k * kThreads + threadIdx.x;
    if (p < n) orow[j0 + p] = v[k];
  }
}

// ELL: thread per row, slots in order, column-major stores (coalesced across
// the warp).  When a CTA's CSR segment fits kEllCap elements and is not much
// longer than the slots it fills, it is first staged in shared memory with
// coalesced loads (one pad word per 32: conflict-free for rows of 32).
constexpr uint32_t kEllCap = 8192;
template <typename T>
constexpr size_t ell_smem_bytes() {
  return (size_t)(kEllCap + kEllCap / 32) * (sizeof(T) + sizeof(uint32_t));
}

template <typename T>
__global__ void __launch_bounds__(kThreads) ell_kernel(uint32_t rows, uint32_t width, const uint32_t *__restrict__ rp,
                                                       const uint32_t *__restrict__ cols,
                                                       const T *__restrict__ vals, T *__restrict__ ed,
                                                       uint32_t *__restrict__ ec) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *sv = reinterpret_cast<T *>(smem_raw);
  uint32_t *sc = reinterpret_cast<uint32_t *>(sv + kEllCap + kEllCap / 32);
  const uint32_t r0 = blockIdx.x * kThreads;
  const uint32_t nr = min(kThreads, rows - r0);
  const uint32_t seg0 = rp[r0], seg1 = rp[r0 + nr];
  const uint32_t r = r0 + threadIdx.x;
  const bool has = r < rows;
  const uint32_t b = has ? rp[r] : 0u;
  const uint32_t len = has ? min(rp[r + 1] - b, width) : 0u;
  const bool staged = seg1 - seg0 <= kEllCap && (uint64_t)(seg1 - seg0) <= 2ull * nr * width;
  if (staged) {
    // 8 loads in flight per thread before their shared-memory stores
    for (uint32_t e0 = seg0 + threadIdx.x; e0 < seg1; e0 += 8u * kThreads) {
      T vv[8];
      uint32_t cc[8];
#pragma unroll
      for (uint32_t k = 0; k < 8; ++k) {
        const uint32_t e = e0 + k * kThreads;
        if (e < seg1) {
          vv[k] = vals[e];
          cc[k] = cols[e];
        }
      }
#pragma unroll
      for (uint32_t k = 0; k < 8; ++k) {
        const uint32_t e = e0 + k * kThreads;
        if (e < seg1) {
          sv[pad(e - seg0)] = vv[k];
          sc[pad(e - seg0)] = cc[k];
        }
      }
    }
    __syncthreads();
  }
  if (!has) return;
  for (uint32_t s = 0; s < width; ++s) {
    const size_t o = (size_t)s * rows + r;
    if (s < len) {
      ed[o] = staged ? sv[pad(b - seg0 + s)] : vals[b + s];
      ec[o] = staged ? sc[pad(b - seg0 + s)] : cols[b + s];
    } else {
      ed[o] = T(0);
      ec[o] = 0u;
    }
  }
}

// slices_ptr: a slice starts every slice_size rows (scoo_matrix_class.cpp:76-100);
// entries after the last real slice stay 0.
__global__ void __launch_bounds__(kThreads) scoo_slices_kernel(uint32_t nnz, const uint32_t *rp, uint32_t slice_size,
                                                               uint32_t count, uint32_t real, uint32_t *sp) {
  const uint32_t i = blockIdx.x * kThreads + threadIdx.x;
  if (i > count) return;
  sp[i] = i < real ? rp[(size_t)i * slice_size] : (i == real ? nnz : 0u);
}

// ---------------------------------------------------------------------------
// Row statistics: min / max / sum of row lengths, then the sum of squared
// deviations from the integer average as an exact 64-bit integer.
// ---------------------------------------------------------------------------
// Grid-stride over rows, then one atomic per block and quantity (same-address
// atomics from every warp would serialise in L2).
constexpr uint32_t kStatBlocks = 148 * 4;

template <typename T>
__device__ __forceinline__ T block_reduce_op(T v, T *s, int op) {  // op 0 sum, 1 min, 2 max, 3 or
  for (uint32_t o = 16; o; o >>= 1) {
    const T u = __shfl_xor_sync(0xffffffffu, v, o);
    v = op == 0 ? v + u : op == 1 ? min(v, u) : op == 2 ? max(v, u) : (v | u);
  }
  if ((threadIdx.x & 31u) == 0) s[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0)
    for (uint32_t w = 1; w < kWarps; ++w) v = op == 0 ? v + s[w] : op == 1 ? min(v, s[w]) : op == 2 ? max(v, s[w]) : (v | s[w]);
  __syncthreads();
  return v;  // valid in thread 0
}

__global__ void __launch_bounds__(kThreads) row_minmax_kernel(uint32_t rows, const uint32_t *rp,
                                                              unsigned long long *acc) {
  __shared__ unsigned long long s[kWarps];
  unsigned long long mn = 0xffffffffull, mx = 0ull, sm = 0ull;
  for (uint64_t r = (uint64_t)blockIdx.x * kThreads + threadIdx.x; r < rows; r += (uint64_t)gridDim.x * kThreads) {
    const unsigned long long n = rp[r + 1] - rp[r];
    mn = min(mn, n);
    mx = max(mx, n);
    sm += n;
  }
  mn = block_reduce_op(mn, s, 1);
  mx = block_reduce_op(mx, s, 2);
  sm = block_reduce_op(sm, s, 0);
  if (threadIdx.x == 0) {
    atomicMin(&acc[0], mn);
    atomicMax(&acc[1], mx);
    atomicAdd(&acc[2], sm);
  }
}
// acc[3] += (n - avg)^2; acc[4] flags a deviation >= 2^26 (its square may not
// be exact in double, so the exact-sum shortcut does not apply)
__global__ void __launch_bounds__(kThreads) row_sqdev_kernel(uint32_t rows, const uint32_t *rp, uint32_t avg,
                                                             unsigned long long *acc) {
  __shared__ unsigned long long s[kWarps];
  unsigned long long q = 0, big = 0;
  for (uint64_t r = (uint64_t)blockIdx.x * kThreads + threadIdx.x; r < rows; r += (uint64_t)gridDim.x * kThreads) {
    const uint32_t n = rp[r + 1] - rp[r];
    const unsigned long long d = n > avg ? n - avg : avg - n;
    q += d * d;
    big |= d >= (1ull << 26);
  }
  q = block_reduce_op(q, s, 0);
  big = block_reduce_op(big, s, 3);
  if (threadIdx.x == 0) {
    atomicAdd(&acc[3], q);
    if (big) atomicOr(&acc[4], 1ull);
  }
}
// acc[0] += sum over rows of max(0, len - start)
__global__ void __launch_bounds__(kThreads) tail_count_kernel(uint32_t rows, const uint32_t *rp, uint32_t start,
                                                              unsigned long long *acc) {
  __shared__ unsigned long long s[kWarps];
  unsigned long long c = 0;
  for (uint64_t r = (uint64_t)blockIdx.x * kThreads + threadIdx.x; r < rows; r += (uint64_t)gridDim.x * kThreads) {
    const uint32_t n = rp[r + 1] - rp[r];
    c += n > start ? n - start : 0u;
  }
  c = block_reduce_op(c, s, 0);
  if (threadIdx.x == 0) atomicAdd(acc, c);
}

// Checks a device CSR: row_ptr[0] = 0, non-decreasing, row_ptr[rows] = nnz,
// columns < cols.  err[0] |= 1 (row_ptr) / 2 (column), err[1] = min bad index.
__global__ void __launch_bounds__(kThreads) check_csr_kernel(uint32_t rows, uint32_t nnz, uint32_t cols,
                                                             const uint32_t *rp, const uint32_t *ci, uint32_t *err) {
  const uint64_t i = (uint64_t)blockIdx.x * kThreads + threadIdx.x;
  if (i <= rows) {
    const uint32_t a = rp[i];
    const bool bad = (i == 0 && a != 0) || (i == rows && a != nnz) || (i < rows && rp[i + 1] < a);
    if (bad) {
      atomicOr(&err[0], 1u);
      atomicMin(&err[1], (uint32_t)i);
    }
  }
  if (i < nnz && ci[i] >= cols && !(cols == 0 && ci[i] == 0)) {
    atomicOr(&err[0], 2u);
    atomicMin(&err[2], (uint32_t)i);
  }
}

// Per-slice column window [min, max + 1) (mfp_scoo_x_windows on the device).
__global__ void __launch_bounds__(kThreads) scoo_windows_kernel(uint32_t nnz, const uint32_t *ci, const uint32_t *sp,
                                                                uint32_t *win) {
  __shared__ uint32_t s_lo[kWarps], s_hi[kWarps];
  const uint32_t sl = blockIdx.x;
  const uint32_t b = sp[sl], e = sp[sl + 1];
  uint32_t lo = 0xffffffffu, hi = 0u;
  const bool any = b < e && e <= nnz;
  if (any)
    for (uint32_t k = b + threadIdx.x; k < e; k += kThreads) {
      lo = min(lo, ci[k]);
      hi = max(hi, ci[k] + 1u);
    }
  for (uint32_t o = 16; o; o >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if ((threadIdx.x & 31u) == 0) {
    s_lo[threadIdx.x >> 5] = lo;
    s_hi[threadIdx.x >> 5] = hi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (uint32_t w = 1; w < kWarps; ++w) {
      lo = min(lo, s_lo[w]);
      hi = max(hi, s_hi[w]);
    }
    win[2 * sl] = any ? lo : 0u;
    win[2 * sl + 1] = any ? hi : 0u;
  }
}

// ---------------------------------------------------------------------------
// COO triplets -> CSR: keys (row << cb | col) with the value converted to T as
// payload, a stable LSD radix sort when the input is not already in CSR
// order, then row_ptr from the row boundaries of the sorted rows.
//
// One launch per digit, as in the published one-sweep radix sort (Adinets and
// Merrill, 2022), with the decoupled look-back of Merrill and Garland (2016).  A
// pass reads and writes 12 bytes per FP32 element (24 in all); the histograms of
// every digit come from one read of the ids before the passes, the first pass
// reads the triplets themselves and the last one writes the CSR arrays.  B200,
// 15.1M elements of 2M rows (42 key bits), FP32: 894 us: 75 for the
// histograms and 145 a pass (2.4 TB/s; shared memory at 54% and instruction issue
// at 53% of their rates, 31 warps per SM).  It was 1,340
// us with five launches per 8-bit digit (histogram 39 us, scans 12, scatter
// 137, whose __match_any_sync kept one pipe 74% busy), 130 for making the keys
// and 100 for splitting them.  Equal digits found with a shared-memory atomicOr
// instead of ballots: 988 us; 256 threads with 16 keys each: 1,259 us (spills,
// runs of 8 keys).
// ---------------------------------------------------------------------------
constexpr uint32_t kKeyBlocks = 148 * 6;

struct radix_digits {
  uint32_t passes = 0, bits = 0;  // digits per key, bits per digit
  radix_digits() = default;
  explicit radix_digits(uint32_t key_bits) {
    passes = (key_bits + kRadixBits - 1u) / kRadixBits;
    bits = key_bits <= 8u * passes ? 8u : 9u;
  }
};

// Where a pass takes its keys and payloads, and where it puts them.
template <typename T>
struct triplets_in {
  const uint32_t *__restrict__ r, *__restrict__ c;
  const double *__restrict__ v;
  uint32_t cb;
  __device__ unsigned long long key(uint64_t i) const { return ((unsigned long long)r[i] << cb) | c[i]; }
  __device__ T pay(uint64_t i) const { return static_cast<T>(v[i]); }
};
template <typename P>
struct pairs_in {
  const unsigned long long *__restrict__ k;
  const P *__restrict__ p;
  __device__ unsigned long long key(uint64_t i) const { return k[i]; }
  __device__ P pay(uint64_t i) const { return p[i]; }
};
template <typename P>
struct pairs_out {
  unsigned long long *__restrict__ k;
  P *__restrict__ p;
  __device__ void key(uint32_t g, unsigned long long v) const { k[g] = v; }
  __device__ void pay(uint32_t g, P v) const { p[g] = v; }
};
template <typename T>
struct csr_out {
  uint32_t *__restrict__ rows, *__restrict__ cols;
  T *__restrict__ data;
  uint32_t cb;
  __device__ void key(uint32_t g, unsigned long long v) const {
    rows[g] = (uint32_t)(v >> cb);
    cols[g] = (uint32_t)(v & ((1ull << cb) - 1ull));
  }
  __device__ void pay(uint32_t g, T v) const { data[g] = v; }
};

template <uint32_t BITS>
__device__ __forceinline__ uint32_t digit_of(unsigned long long k, uint32_t shift) {
  const uint32_t lo = (uint32_t)k, hi = (uint32_t)(k >> 32);
  return (shift < 32u ? __funnelshift_r(lo, hi, shift) : hi >> (shift - 32u)) & ((1u << BITS) - 1u);
}

// Exclusive prefix over the CTA of a radix pass; s holds kRadixWarps words.
__device__ __forceinline__ uint32_t radix_excl(uint32_t v, uint32_t *s) {
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  const uint32_t inc = warp_incl_sum(v);
  if (lane == 31) s[w] = inc;
  __syncthreads();
  if (w == 0) {
    const uint32_t t = warp_incl_sum(lane < kRadixWarps ? s[lane] : 0u);
    if (lane < kRadixWarps) s[lane] = t;
  }
  __syncthreads();
  return (w ? s[w - 1] : 0u) + inc - v;
}

// Histograms of every digit: hist[pass][bin] (zeroed, as err).  CHECK (triplets):
// err[0] |= 1 (row id) / 2 (col id), err[1] = ~ the first bad element, err[2] = 1
// when some key is smaller than its predecessor (input not in CSR order).
template <bool CHECK, uint32_t BITS, typename In>
__global__ void __launch_bounds__(kThreads) radix_hist_kernel(uint32_t n, In in, uint32_t rows, uint32_t cols,
                                                              uint32_t passes, uint32_t *hist, uint32_t *err) {
  __shared__ uint32_t h[kRadixPasses * kRadixBins];
  for (uint32_t i = threadIdx.x; i < passes * kRadixBins; i += kThreads) h[i] = 0u;
  __syncthreads();
  bool unsorted = false;
  // tiles of 4 keys per thread, their loads issued together
  const uint64_t step = (uint64_t)gridDim.x * kThreads * 4u;
  for (uint64_t b = (uint64_t)blockIdx.x * kThreads * 4u; b < n; b += step) {
    unsigned long long k[4];
    bool bad[4];
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
      const uint64_t i = b + j * kThreads + threadIdx.x;
      bad[j] = false;
      if constexpr (CHECK) {
        const uint32_t r = i < n ? in.r[i] : 0u, c = i < n ? in.c[i] : 0u;
        k[j] = ((unsigned long long)r << in.cb) | c;
        bad[j] = i < n && (r >= rows || c >= cols);
      } else {
        k[j] = i < n ? in.key(i) : 0ull;
      }
    }
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
      const uint64_t i = b + j * kThreads + threadIdx.x;
      if constexpr (CHECK) {
        unsigned long long prev = __shfl_up_sync(0xffffffffu, k[j], 1);
        if ((threadIdx.x & 31u) == 0) prev = i && i < n ? in.key(i - 1) : 0ull;
        unsorted |= i < n && prev > k[j];
        if (bad[j]) {
          atomicOr(&err[0], in.r[i] >= rows ? 1u : 2u);
          atomicMax(&err[1], ~(uint32_t)i);
        }
      }
      if (i < n) {
#pragma unroll
        for (uint32_t p = 0; p < kRadixPasses; ++p)
          if (p < passes) atomicAdd(&h[p * kRadixBins + digit_of<BITS>(k[j], p * BITS)], 1u);
      }
    }
  }
  if (CHECK && unsorted) err[2] = 1u;
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < passes * kRadixBins; i += kThreads)
    if (h[i]) atomicAdd(&hist[i], h[i]);
}

// Status words of the look-back, one per (tile, digit): the high half says
// what the low half counts, by pass (stale words of earlier passes say less).
__device__ __forceinline__ unsigned long long status_word(uint32_t pass, bool prefix, uint32_t v) {
  return ((unsigned long long)(2u * pass + (prefix ? 2u : 1u)) << 32) | v;
}
__device__ __forceinline__ unsigned long long ld_status(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_status(unsigned long long *p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// A digit's look-back ran out: the error word, and no more tiles of later passes.
__device__ __noinline__ void radix_give_up(uint32_t pass, uint32_t *counter, uint32_t *err) {
  atomicOr(&err[3], 1u);
  for (uint32_t p = pass + 1u; p < kRadixPasses; ++p) atomicOr(counter + (p - pass), kStop);
}

// One digit: stable scatter of a 6,144-key tile.  Keys go, in tile order, after
// every key of a smaller digit and after the same digit's keys of earlier
// tiles.  Warp w ranks its contiguous 384 keys with a warp-private digit
// histogram (equal digits found bit by bit with ballots), thread t scans digit
// t over the warps and looks back for its count in the tiles before, the tile
// is placed in shared memory in digit order and written out as contiguous digit
// runs; payloads follow through the same shared memory.  Tiles are numbered in
// the order their CTAs start, so a tile only ever waits for CTAs that are
// running.  The wait is bounded: a digit that gives up after `polls` looks in vain
// goes on with the part of its count that it has, which is too small, so its keys
// stay inside the array but leave holes in it; it sets err[3] and marks the tile
// counters of the later passes (`counter` is this pass's of kRadixPasses), whose
// tiles return at once instead of taking digits from the holes.
struct radix_smem {
  unsigned long long key[kRadixTile];  // or payloads
  uint32_t wh[kRadixWarps][kRadixBins];
  uint32_t gbase[kRadixBins];
  uint32_t red[kRadixWarps], red2[kRadixWarps];
  uint32_t tile;
};
template <uint32_t BITS, typename P, typename In, typename Out>
__global__ void __launch_bounds__(kRadixThreads, 2) radix_pass_kernel(uint32_t n, In in, Out out, uint32_t pass,
                                                                      const uint32_t *hist, uint32_t *counter,
                                                                      unsigned long long *status, uint32_t polls,
                                                                      uint32_t *err) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  radix_smem &S = *reinterpret_cast<radix_smem *>(smem_raw);
  constexpr uint32_t kPerWarp = kRadixTile / kRadixWarps;
  const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
  if (t == 0) S.tile = atomicAdd(counter, 1u);
#pragma unroll
  for (uint32_t i = 0; i < kRadixWarps; ++i) S.wh[i][t] = 0u;
  const uint32_t hv = hist[t];
  __syncthreads();
  // (shuffled, so that the compiler knows the warp leaves as one: 18 us of 915)
  const uint32_t tile = __shfl_sync(0xffffffffu, S.tile, 0), shift = pass * BITS;
  if (tile & kStop) return;
  const uint64_t base = (uint64_t)tile * kRadixTile;
  const uint32_t tn = (uint32_t)min((uint64_t)kRadixTile, n - base);
  const uint32_t wbase = warp * kPerWarp + lane;
  unsigned long long k[kRadixRounds];
#pragma unroll
  for (uint32_t j = 0; j < kRadixRounds; ++j) k[j] = wbase + j * 32u < tn ? in.key(base + wbase + j * 32u) : ~0ull;
  // the keys of smaller digits in the whole array
  const uint32_t below = radix_excl(hv, S.red);
  uint32_t rk[kRadixRounds];
  uint32_t *wh = S.wh[warp];
#pragma unroll
  for (uint32_t j = 0; j < kRadixRounds; ++j) {
    const uint32_t d = digit_of<BITS>(k[j], shift);
    const bool valid = wbase + j * 32u < tn;
    uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
    for (uint32_t b = 0; b < BITS; ++b) {
      const uint32_t other = 0u - ((d >> b) & 1u ^ 1u);  // all ones where the bit is 0
      peers &= __ballot_sync(0xffffffffu, (d >> b) & 1u) ^ other;
    }
    const uint32_t before = wh[d];
    __syncwarp();
    const uint32_t mine = peers & ((1u << lane) - 1u);
    if (valid && mine == 0u) wh[d] = before + __popc(peers);
    __syncwarp();
    rk[j] = before + __popc(mine);
  }
  __syncthreads();
  uint32_t tot = 0;  // thread t: digit t, summed over the warps
#pragma unroll
  for (uint32_t w = 0; w < kRadixWarps; ++w) tot += S.wh[w][t];
  unsigned long long *mine = status + (size_t)tile * kRadixBins + t;
  st_status(mine, status_word(pass, tile == 0, tot));
  const uint32_t start = radix_excl(tot, S.red2);
  {
    uint32_t at = start;
#pragma unroll
    for (uint32_t w = 0; w < kRadixWarps; ++w) {
      const uint32_t c = S.wh[w][t];
      S.wh[w][t] = at;
      at += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (uint32_t j = 0; j < kRadixRounds; ++j)
    if (wbase + j * 32u < tn) {
      rk[j] += wh[digit_of<BITS>(k[j], shift)];  // the key's place in the tile
      S.key[rk[j]] = k[j];
    }
  // the same digit's keys in earlier tiles
  uint32_t excl = 0;
  if (tile) {
    const unsigned long long *st = status + t;
    for (uint32_t w = tile - 1u, waits = 0;;) {
      const unsigned long long v = ld_status(st + (size_t)w * kRadixBins);
      const uint32_t flag = (uint32_t)(v >> 32);
      if (flag <= 2u * pass || polls == 0u) {  // not there yet
        if (++waits > polls) {
          radix_give_up(pass, counter, err);
          break;
        }
        continue;
      }
      excl += (uint32_t)v;
      if (flag == 2u * pass + 2u || w == 0) break;
      --w;
    }
    st_status(mine, status_word(pass, true, excl + tot));
  }
  S.gbase[t] = below + excl - start;
  __syncthreads();
  uint32_t g[kRadixRounds];
#pragma unroll
  for (uint32_t j = 0; j < kRadixRounds; ++j) {
    const uint32_t p = j * kRadixThreads + t;
    if (p < tn) {
      const unsigned long long kk = S.key[p];
      g[j] = S.gbase[digit_of<BITS>(kk, shift)] + p;
      out.key(g[j], kk);
    }
  }
  P v[kRadixRounds];
#pragma unroll
  for (uint32_t j = 0; j < kRadixRounds; ++j)
    v[j] = wbase + j * 32u < tn ? in.pay(base + wbase + j * 32u) : P(0);
  __syncthreads();
  P *sp = reinterpret_cast<P *>(S.key);
#pragma unroll
  for (uint32_t j = 0; j < kRadixRounds; ++j)
    if (wbase + j * 32u < tn) sp[rk[j]] = v[j];
  __syncthreads();
#pragma unroll
  for (uint32_t j = 0; j < kRadixRounds; ++j)
    if (j * kRadixThreads + t < tn) out.pay(g[j], sp[j * kRadixThreads + t]);
}

// row_ptr from sorted rows: position p starts the rows (rows[p-1], rows[p]]
// (p = nnz closes the rows after the last element's row).  Nothing after a sort
// that gave up, whose rows are not ids.
__global__ void __launch_bounds__(kThreads) rowptr_from_rows_kernel(uint32_t nnz, uint32_t rows,
                                                                    const uint32_t *__restrict__ ri, uint32_t *rp,
                                                                    const uint32_t *err) {
  const uint64_t p = (uint64_t)blockIdx.x * kThreads + threadIdx.x;
  if (p > nnz) return;
  const row_span span = rows_starting_at(p, nnz, p ? ri[p - 1] : 0u, p < nnz ? ri[p] : 0u, rows);
  if (__ldg(err + 3)) return;
  for (uint64_t q = span.first; q < span.end; ++q) rp[q] = (uint32_t)p;
}

// Triplets already in CSR order.
template <typename T>
__global__ void __launch_bounds__(kThreads) csr_copy_kernel(uint32_t nnz, const uint32_t *__restrict__ ci,
                                                            const double *__restrict__ v, uint32_t *__restrict__ cols_out,
                                                            T *__restrict__ data_out) {
  const uint32_t p = blockIdx.x * kThreads + threadIdx.x;
  if (p >= nnz) return;
  cols_out[p] = ci[p];
  data_out[p] = static_cast<T>(v[p]);
}

bool valid_vt(int vt) { return vt == MFP_F32 || vt == MFP_F64; }

template <typename T>
int coo_from_csr_t(uint32_t rows, const uint32_t *rp, const uint32_t *ci, const T *vals, uint32_t start, T *od,
                   uint32_t *oc, uint32_t *orow, void *stream) {
  cudaStream_t st = as_stream(stream);
  scratch sc(st);
  if (rows == 0) return ok();
  const uint32_t *tp = rp;
  uint32_t *tpw = nullptr;
  int s;
  if (start) {
    if ((s = sc.get(&tpw, (size_t)rows + 1))) return s;
    if ((s = exclusive_scan(rows, f_tail{rp, start}, tpw, sc))) return s;
    tp = tpw;
  }
  uint32_t total = 0;
  CV_TRY(cudaMemcpyAsync(&total, tp + rows, sizeof(uint32_t), cudaMemcpyDeviceToHost, st), "cudaMemcpyAsync");
  CV_TRY(cudaStreamSynchronize(st), "cudaStreamSynchronize");
  if (total == 0) return ok();
  if (!od || !oc || !orow) return fail(MFP_ERROR_INVALID_VALUE, "null output array");
  const uint32_t ntiles = blocks_for(total, kTile);
  uint32_t *tr = nullptr;
  if ((s = sc.get(&tr, (size_t)ntiles + 1))) return s;
  tile_rows_kernel<<<blocks_for((uint64_t)ntiles + 1, kThreads), kThreads, 0, st>>>(rows, total, tp, ntiles, tr);
  if (start) {
    expand_kernel<T, true><<<ntiles, kThreads, 0, st>>>(total, tr, tp, rp, start, ci, vals, od, oc, orow);
  } else {
    CV_TRY(cudaMemcpyAsync(od, vals, (size_t)total * sizeof(T), cudaMemcpyDeviceToDevice, st), "cudaMemcpyAsync");
    CV_TRY(cudaMemcpyAsync(oc, ci, (size_t)total * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st), "cudaMemcpyAsync");
    expand_kernel<T, false><<<ntiles, kThreads, 0, st>>>(total, tr, tp, rp, 0u, ci, vals, od, oc, orow);
  }
  CV_TRY(cudaGetLastError(), "expand_kernel");
  return ok();
}

// Device words of one sort, zeroed by begin(): status words, histograms, tile
// counters and error words, each from a 128-byte boundary (whole warps read a
// tile's row of status words: 48 bytes off, a pass took 4% longer).
struct radix_state {
  unsigned long long *status = nullptr;
  uint32_t *err = nullptr, *hist = nullptr, *counters = nullptr;
  uint32_t tiles = 0;
  int begin(uint32_t n, scratch &sc) {
    tiles = blocks_for(n, kRadixTile);
    const size_t words = (size_t)tiles * kRadixBins, bytes = words * 8u + (kRadixPasses * kRadixBins + 32u + 4u) * 4u;
    unsigned char *p = nullptr;
    const int s = sc.get(&p, bytes);
    if (s) return s;
    status = reinterpret_cast<unsigned long long *>(p);
    hist = reinterpret_cast<uint32_t *>(p + words * 8u);
    counters = hist + kRadixPasses * kRadixBins;
    err = counters + 32;
    CV_TRY(cudaMemsetAsync(p, 0, bytes, sc.st), "cudaMemsetAsync");
    return MFP_SUCCESS;
  }
};
// The histograms of `in`, with the other device words made ready.
template <bool CHECK, typename In>
int radix_histograms(uint32_t n, const In &in, uint32_t rows, uint32_t cols, const radix_digits &dg, radix_state &R,
                     scratch &sc) {
  const int s = R.begin(n, sc);
  if (s) return s;
  auto k = dg.bits == 8u ? radix_hist_kernel<CHECK, 8, In> : radix_hist_kernel<CHECK, 9, In>;
  k<<<std::min(kKeyBlocks, blocks_for(n, 4u * kThreads)), kThreads, 0, sc.st>>>(
      n, in, rows, cols, dg.passes, R.hist, R.err);
  CV_TRY(cudaGetLastError(), "radix_hist_kernel");
  return MFP_SUCCESS;
}
template <typename P, typename In, typename Out>
int radix_pass(uint32_t n, const In &in, const Out &out, const radix_digits &dg, uint32_t pass, const radix_state &R,
               uint32_t polls, scratch &sc) {
  auto k = dg.bits == 8u ? radix_pass_kernel<8, P, In, Out> : radix_pass_kernel<9, P, In, Out>;
  CV_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(radix_smem)),
         "cudaFuncSetAttribute");
  k<<<R.tiles, kRadixThreads, sizeof(radix_smem), sc.st>>>(n, in, out, pass, R.hist + pass * kRadixBins,
                                                           R.counters + pass, R.status, polls, R.err);
  CV_TRY(cudaGetLastError(), "radix_pass_kernel");
  return MFP_SUCCESS;
}
int radix_error(uint32_t flag) {
  return flag ? fail(MFP_ERROR_DEVICE_WAIT, "a radix tile gave up waiting for the tiles before it") : MFP_SUCCESS;
}

// Stable LSD radix sort of n (key, payload) pairs on the low `bits` key bits;
// k0 / p0 hold the input and, on return, the sorted pairs (buffers swap).
template <typename P>
int radix_sort_pairs(uint32_t n, uint32_t bits, unsigned long long *&k0, P *&p0, scratch &sc) {
  if (n == 0 || bits == 0) return MFP_SUCCESS;
  const radix_digits dg(bits);
  unsigned long long *k1 = nullptr;
  P *p1 = nullptr;
  uint32_t h_err[4];
  radix_state R;
  int s;
  if ((s = sc.get(&k1, n)) || (s = sc.get(&p1, n)) ||
      (s = radix_histograms<false>(n, pairs_in<P>{k0, p0}, 0u, 0u, dg, R, sc)))
    return s;
  for (uint32_t pass = 0; pass < dg.passes; ++pass) {
    if ((s = radix_pass<P>(n, pairs_in<P>{k0, p0}, pairs_out<P>{k1, p1}, dg, pass, R, kRadixPolls, sc))) return s;
    std::swap(k0, k1);
    std::swap(p0, p1);
  }
  CV_TRY(cudaMemcpyAsync(h_err, R.err, sizeof(h_err), cudaMemcpyDeviceToHost, sc.st), "cudaMemcpyAsync");
  CV_TRY(cudaStreamSynchronize(sc.st), "cudaStreamSynchronize");
  return radix_error(h_err[3]);
}

struct byte_range {
  const void *p;
  size_t bytes;
  bool overlaps(const byte_range &o) const {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p), b = reinterpret_cast<uintptr_t>(o.p);
    return a < b + o.bytes && b < a + bytes;
  }
};
// An input that an output overlaps moves to scratch.
template <typename I>
int unshare(const I *&in, size_t n, const byte_range (&outs)[3], scratch &sc) {
  const byte_range r{in, n * sizeof(I)};
  if (!r.overlaps(outs[0]) && !r.overlaps(outs[1]) && !r.overlaps(outs[2])) return MFP_SUCCESS;
  I *copy = nullptr;
  const int s = sc.get(&copy, n);
  if (s) return s;
  CV_TRY(cudaMemcpyAsync(copy, in, r.bytes, cudaMemcpyDeviceToDevice, sc.st), "cudaMemcpyAsync");
  in = copy;
  return MFP_SUCCESS;
}

template <typename T>
int csr_from_coo_t(uint32_t rows, uint32_t cols, uint32_t nnz, const uint32_t *ri, const uint32_t *ci,
                   const double *v, uint32_t *rp, uint32_t *co, T *data, uint32_t polls, void *stream) {
  cudaStream_t st = as_stream(stream);
  scratch sc(st);
  if (!rp) return fail(MFP_ERROR_INVALID_VALUE, "null row_ptr");
  if (nnz && (!ri || !ci || !v || !co || !data)) return fail(MFP_ERROR_INVALID_VALUE, "null array");
  if (nnz == 0) {
    CV_TRY(cudaMemsetAsync(rp, 0, ((size_t)rows + 1) * sizeof(uint32_t), st), "cudaMemsetAsync");
    CV_TRY(cudaStreamSynchronize(st), "cudaStreamSynchronize");
    return ok();
  }
  const uint32_t rb = rows > 1 ? bits_for(rows - 1) : 0u, cb = cols > 1 ? bits_for(cols - 1) : 0u;
  const radix_digits dg(rb + cb);
  radix_state R;
  int s;
  if ((s = radix_histograms<true>(nnz, triplets_in<T>{ri, ci, v, cb}, rows, cols, dg, R, sc))) return s;
  uint32_t h_err[4];
  CV_TRY(cudaMemcpyAsync(h_err, R.err, sizeof(h_err), cudaMemcpyDeviceToHost, st), "cudaMemcpyAsync");
  CV_TRY(cudaStreamSynchronize(st), "cudaStreamSynchronize");
  if (h_err[0] & 1u) return fail(MFP_ERROR_INVALID_VALUE, "row id >= rows %u at element %u", rows, ~h_err[1]);
  if (h_err[0] & 2u) return fail(MFP_ERROR_INVALID_VALUE, "col id >= cols %u at element %u", cols, ~h_err[1]);
  // a kernel that reads the triplets and writes the CSR needs them apart (several
  // passes read them all into scratch first)
  if (!h_err[2] || dg.passes == 1u) {
    const byte_range outs[3] = {{rp, ((size_t)rows + 1) * 4u}, {co, (size_t)nnz * 4u}, {data, (size_t)nnz * sizeof(T)}};
    if ((s = unshare(ri, nnz, outs, sc)) || (s = unshare(ci, nnz, outs, sc)) || (s = unshare(v, nnz, outs, sc))) return s;
  }
  const triplets_in<T> in{ri, ci, v, cb};
  const uint32_t *sorted_rows = ri;
  if (!h_err[2]) {  // in CSR order already: a stable sort would keep it
    csr_copy_kernel<T><<<blocks_for(nnz, kThreads), kThreads, 0, st>>>(nnz, ci, v, co, data);
  } else {
    unsigned long long *k[2] = {nullptr, nullptr};
    T *p[2] = {nullptr, nullptr};
    uint32_t *out_rows = nullptr;
    for (uint32_t b = 0; b < 2u && b + 1u < dg.passes; ++b)
      if ((s = sc.get(&k[b], nnz)) || (s = sc.get(&p[b], nnz))) return s;
    // the last pass leaves the rows in the key buffer that it does not read
    out_rows = reinterpret_cast<uint32_t *>(k[(dg.passes - 1u) & 1u]);
    if (!out_rows && (s = sc.get(&out_rows, nnz))) return s;
    const csr_out<T> out{out_rows, co, data, cb};
    for (uint32_t pass = 0; pass < dg.passes; ++pass) {
      const bool first = pass == 0, last = pass + 1u == dg.passes;
      const pairs_in<T> mid_in{k[(pass + 1u) & 1u], p[(pass + 1u) & 1u]};
      const pairs_out<T> mid_out{k[pass & 1u], p[pass & 1u]};
      if (first)
        s = last ? radix_pass<T>(nnz, in, out, dg, pass, R, polls, sc)
                 : radix_pass<T>(nnz, in, mid_out, dg, pass, R, polls, sc);
      else
        s = last ? radix_pass<T>(nnz, mid_in, out, dg, pass, R, polls, sc)
                 : radix_pass<T>(nnz, mid_in, mid_out, dg, pass, R, polls, sc);
      if (s) return s;
    }
    sorted_rows = out_rows;
  }
  rowptr_from_rows_kernel<<<blocks_for((uint64_t)nnz + 1, kThreads), kThreads, 0, st>>>(nnz, rows, sorted_rows, rp, R.err);
  CV_TRY(cudaGetLastError(), "rowptr_from_rows_kernel");
  if (h_err[2])  // sorted here: whether a tile gave up
    CV_TRY(cudaMemcpyAsync(h_err, R.err, sizeof(h_err), cudaMemcpyDeviceToHost, st), "cudaMemcpyAsync");
  CV_TRY(cudaStreamSynchronize(st), "cudaStreamSynchronize");
  if (h_err[3]) return radix_error(h_err[3]);
  return ok();
}

// SCOO sort_cols: keys (slice << cb | col) with the element index as payload;
// after the stable sort, values and rows are gathered by index.
__global__ void __launch_bounds__(kThreads) slice_keys_kernel(uint32_t nnz, const uint32_t *__restrict__ ri,
                                                              const uint32_t *__restrict__ ci, uint32_t slice_size,
                                                              uint32_t cb, unsigned long long *__restrict__ keys,
                                                              uint32_t *__restrict__ idx) {
  const uint32_t i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= nnz) return;
  keys[i] = ((unsigned long long)(ri[i] / slice_size) << cb) | ci[i];
  idx[i] = i;
}
template <typename T>
__global__ void __launch_bounds__(kThreads) slice_gather_kernel(uint32_t nnz, const unsigned long long *__restrict__ keys,
                                                                const uint32_t *__restrict__ idx,
                                                                unsigned long long cmask, const T *__restrict__ v_in,
                                                                const uint32_t *__restrict__ r_in, T *__restrict__ v_out,
                                                                uint32_t *__restrict__ c_out, uint32_t *__restrict__ r_out) {
  const uint32_t p = blockIdx.x * kThreads + threadIdx.x;
  if (p >= nnz) return;
  const uint32_t j = idx[p];
  c_out[p] = (uint32_t)(keys[p] & cmask);
  v_out[p] = v_in[j];
  r_out[p] = r_in[j];
}

template <typename T>
int scoo_sort_cols_t(uint32_t rows, uint32_t cols, uint32_t slice_size, uint32_t nnz, T *v, uint32_t *ci,
                     uint32_t *ri, cudaStream_t st) {
  scratch sc(st);
  if (nnz == 0) return ok();
  if (!v || !ci || !ri) return fail(MFP_ERROR_INVALID_VALUE, "null array");
  if (slice_size == 0) return fail(MFP_ERROR_INVALID_VALUE, "slice_size 0");
  const uint32_t cb = cols > 1 ? bits_for(cols - 1) : 0u;
  const uint32_t sb = rows > slice_size ? bits_for((rows - 1) / slice_size) : 0u;
  unsigned long long *k0 = nullptr;
  uint32_t *p0 = nullptr;
  T *vcopy = nullptr;
  uint32_t *rcopy = nullptr;
  int s;
  if ((s = sc.get(&k0, nnz)) || (s = sc.get(&p0, nnz)) || (s = sc.get(&vcopy, nnz)) || (s = sc.get(&rcopy, nnz)))
    return s;
  CV_TRY(cudaMemcpyAsync(vcopy, v, (size_t)nnz * sizeof(T), cudaMemcpyDeviceToDevice, st), "cudaMemcpyAsync");
  CV_TRY(cudaMemcpyAsync(rcopy, ri, (size_t)nnz * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st), "cudaMemcpyAsync");
  slice_keys_kernel<<<blocks_for(nnz, kThreads), kThreads, 0, st>>>(nnz, ri, ci, slice_size, cb, k0, p0);
  CV_TRY(cudaGetLastError(), "slice_keys_kernel");
  if ((s = radix_sort_pairs<uint32_t>(nnz, sb + cb, k0, p0, sc))) return s;
  slice_gather_kernel<T><<<blocks_for(nnz, kThreads), kThreads, 0, st>>>(nnz, k0, p0, (1ull << cb) - 1ull, vcopy, rcopy,
                                                                         v, ci, ri);
  CV_TRY(cudaGetLastError(), "slice_gather_kernel");
  CV_TRY(cudaStreamSynchronize(st), "cudaStreamSynchronize");
  return ok();
}

}  // namespace

extern "C" {

int mfp_dev_rows_statistics(uint32_t rows, const uint32_t *rp, mfp_rows_statistic *out, void *stream) {
  if (!rp || !out) return fail(MFP_ERROR_INVALID_VALUE, "null argument");
  if (rows == 0) return fail(MFP_ERROR_INVALID_VALUE, "rows == 0");
  cudaStream_t st = as_stream(stream);
  scratch sc(st);
  unsigned long long *acc = nullptr;
  int s = sc.get(&acc, 5);
  if (s) return s;
  // min starts at UINT_MAX - 1 like the reference (matrix_converter.cpp:100)
  const unsigned long long init[5] = {0xfffffffeull, 0ull, 0ull, 0ull, 0ull};
  CV_TRY(cudaMemcpyAsync(acc, init, sizeof(init), cudaMemcpyHostToDevice, st), "cudaMemcpyAsync");
  const uint32_t sb = std::min(kStatBlocks, blocks_for(rows, kThreads));
  row_minmax_kernel<<<sb, kThreads, 0, st>>>(rows, rp, acc);
  unsigned long long h[5];
  CV_TRY(cudaMemcpyAsync(h, acc, sizeof(h), cudaMemcpyDeviceToHost, st), "cudaMemcpyAsync");
  CV_TRY(cudaStreamSynchronize(st), "cudaStreamSynchronize");
  mfp_rows_statistic r{};
  r.min_elements_in_rows = (uint32_t)h[0];
  r.max_elements_in_rows = (uint32_t)h[1];
  // the reference sums in unsigned int (matrix_converter.cpp:102-116)
  r.avg_elements_in_rows = (uint32_t)h[2] / rows;
  row_sqdev_kernel<<<sb, kThreads, 0, st>>>(rows, rp, r.avg_elements_in_rows, acc);
  CV_TRY(cudaMemcpyAsync(h, acc, sizeof(h), cudaMemcpyDeviceToHost, st), "cudaMemcpyAsync");
  CV_TRY(cudaStreamSynchronize(st), "cudaStreamSynchronize");
  if (h[4] == 0 && h[3] < (1ull << 53)) {
    // every partial sum of the reference's double loop is an integer below
    // 2^53, so that loop is exact and equals this integer sum
    r.elements_in_rows_std_deviation = std::sqrt((double)h[3] / rows);
  } else {
    // outside the exact range: run the reference's sequential loop on the host
    std::vector<uint32_t> hp((size_t)rows + 1);
    CV_TRY(cudaMemcpy(hp.data(), rp, hp.size() * sizeof(uint32_t), cudaMemcpyDeviceToHost), "cudaMemcpy D2H");
    return mfp_get_rows_statistics(rows, hp.data(), out);
  }
  *out = r;
  return ok();
}

int mfp_dev_check_csr(uint32_t rows, uint32_t cols, uint32_t nnz, const uint32_t *rp, const uint32_t *ci,
                      void *stream) {
  if (!rp || (nnz && !ci)) return fail(MFP_ERROR_INVALID_VALUE, "null array");
  cudaStream_t st = as_stream(stream);
  scratch sc(st);
  uint32_t *err = nullptr;
  int s = sc.get(&err, 3);
  if (s) return s;
  const uint32_t init[3] = {0u, 0xffffffffu, 0xffffffffu};
  CV_TRY(cudaMemcpyAsync(err, init, sizeof(init), cudaMemcpyHostToDevice, st), "cudaMemcpyAsync");
  const uint64_t n = std::max<uint64_t>((uint64_t)rows + 1, nnz);
  check_csr_kernel<<<blocks_for(n, kThreads), kThreads, 0, st>>>(rows, nnz, cols, rp, ci, err);
  CV_TRY(cudaGetLastError(), "check_csr_kernel");
  uint32_t h[3];
  CV_TRY(cudaMemcpyAsync(h, err, sizeof(h), cudaMemcpyDeviceToHost, st), "cudaMemcpyAsync");
  CV_TRY(cudaStreamSynchronize(st), "cudaStreamSynchronize");
  if (h[0] & 1u) return fail(MFP_ERROR_INVALID_VALUE, "row_ptr is not a CSR row pointer (entry %u)", h[1]);
  if (h[0] & 2u) return fail(MFP_ERROR_INVALID_VALUE, "column id >= cols %u at element %u", cols, h[2]);
  return ok();
}

int mfp_dev_coo_count(uint32_t rows, const uint32_t *rp, uint32_t start, uint32_t *count, void *stream) {
  if (!rp || !count) return fail(MFP_ERROR_INVALID_VALUE, "null argument");
  *count = 0;
  if (rows == 0) return ok();
  cudaStream_t st = as_stream(stream);
  if (start == 0) {  // every element: row_ptr[rows] - row_ptr[0]
    uint32_t ends[2];
    CV_TRY(cudaMemcpyAsync(&ends[0], rp, sizeof(uint32_t), cudaMemcpyDeviceToHost, st), "cudaMemcpyAsync");
    CV_TRY(cudaMemcpyAsync(&ends[1], rp + rows, sizeof(uint32_t), cudaMemcpyDeviceToHost, st), "cudaMemcpyAsync");
    CV_TRY(cudaStreamSynchronize(st), "cudaStreamSynchronize");
    *count = ends[1] - ends[0];
    return ok();
  }
  scratch sc(st);
  unsigned long long *acc = nullptr;
  int s;
  if ((s = sc.get(&acc, 1))) return s;
  CV_TRY(cudaMemsetAsync(acc, 0, sizeof(unsigned long long), st), "cudaMemsetAsync");
  tail_count_kernel<<<std::min(kStatBlocks, blocks_for(rows, kThreads)), kThreads, 0, st>>>(rows, rp, start, acc);
  CV_TRY(cudaGetLastError(), "tail_count_kernel");
  unsigned long long h = 0;
  CV_TRY(cudaMemcpyAsync(&h, acc, sizeof(h), cudaMemcpyDeviceToHost, st), "cudaMemcpyAsync");
  CV_TRY(cudaStreamSynchronize(st), "cudaStreamSynchronize");
  *count = (uint32_t)h;
  return ok();
}

int mfp_dev_coo_from_csr(int vt, uint32_t rows, const uint32_t *rp, const uint32_t *ci, const void *vals,
                         uint32_t start, void *od, uint32_t *oc, uint32_t *orow, void *stream) {
  if (!valid_vt(vt)) return fail(MFP_ERROR_INVALID_VALUE, "bad value type");
  if (!rp) return fail(MFP_ERROR_INVALID_VALUE, "null row_ptr");
  if (vt == MFP_F64)
    return coo_from_csr_t<double>(rows, rp, ci, static_cast<const double *>(vals), start, static_cast<double *>(od),
                                  oc, orow, stream);
  return coo_from_csr_t<float>(rows, rp, ci, static_cast<const float *>(vals), start, static_cast<float *>(od), oc,
                               orow, stream);
}

int mfp_dev_ell_from_csr(int vt, uint32_t rows, const uint32_t *rp, const uint32_t *ci, const void *vals,
                         uint32_t width, void *ed, uint32_t *ec, void *stream) {
  if (!valid_vt(vt)) return fail(MFP_ERROR_INVALID_VALUE, "bad value type");
  if (!rp || ((uint64_t)rows * width && (!ed || !ec))) return fail(MFP_ERROR_INVALID_VALUE, "null array");
  if (rows == 0 || width == 0) return ok();
  cudaStream_t st = as_stream(stream);
  if (vt == MFP_F64) {
    CV_TRY(cudaFuncSetAttribute(ell_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)ell_smem_bytes<double>()),
           "cudaFuncSetAttribute");
    ell_kernel<double><<<blocks_for(rows, kThreads), kThreads, ell_smem_bytes<double>(), st>>>(
        rows, width, rp, ci, static_cast<const double *>(vals), static_cast<double *>(ed), ec);
  } else {
    CV_TRY(cudaFuncSetAttribute(ell_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)ell_smem_bytes<float>()),
           "cudaFuncSetAttribute");
    ell_kernel<float><<<blocks_for(rows, kThreads), kThreads, ell_smem_bytes<float>(), st>>>(
        rows, width, rp, ci, static_cast<const float *>(vals), static_cast<float *>(ed), ec);
  }
  CV_TRY(cudaGetLastError(), "ell_kernel");
  return ok();
}

int mfp_dev_scoo_from_csr(int vt, uint32_t rows, uint32_t nnz, const uint32_t *rp, const uint32_t *ci,
                          const void *vals, const mfp_scoo_params *prm, void *ov, uint32_t *oc, uint32_t *orow,
                          uint32_t *sp, void *stream) {
  if (!valid_vt(vt)) return fail(MFP_ERROR_INVALID_VALUE, "bad value type");
  if (!rp || !prm || !sp) return fail(MFP_ERROR_INVALID_VALUE, "null array");
  if (prm->slice_size == 0 && rows) return fail(MFP_ERROR_INVALID_VALUE, "slice_size 0");
  const uint32_t real = rows ? (uint32_t)(((uint64_t)rows + prm->slice_size - 1) / prm->slice_size) : 0u;
  if (real > prm->slices_count) return fail(MFP_ERROR_INVALID_VALUE, "too many slices");
  cudaStream_t st = as_stream(stream);
  scoo_slices_kernel<<<blocks_for((uint64_t)prm->slices_count + 1, kThreads), kThreads, 0, st>>>(
      nnz, rp, prm->slice_size, prm->slices_count, real, sp);
  CV_TRY(cudaGetLastError(), "scoo_slices_kernel");
  // values, c_index and r_index are the CSR arrays in CSR order with row ids
  return mfp_dev_coo_from_csr(vt, rows, rp, ci, vals, 0, ov, oc, orow, stream);
}

int mfp_dev_scoo_sort_cols(int vt, uint32_t rows, uint32_t cols, uint32_t slice_size, uint32_t nnz, void *values,
                           uint32_t *c_index, uint32_t *r_index, void *stream) {
  if (!valid_vt(vt)) return fail(MFP_ERROR_INVALID_VALUE, "bad value type");
  if (vt == MFP_F64)
    return scoo_sort_cols_t<double>(rows, cols, slice_size, nnz, static_cast<double *>(values), c_index, r_index,
                                    as_stream(stream));
  return scoo_sort_cols_t<float>(rows, cols, slice_size, nnz, static_cast<float *>(values), c_index, r_index,
                                 as_stream(stream));
}

int mfp_dev_scoo_x_windows(uint32_t nnz, const uint32_t *ci, const uint32_t *sp, uint32_t slices, uint32_t *win,
                           void *stream) {
  if (!sp || !win || (nnz && !ci)) return fail(MFP_ERROR_INVALID_VALUE, "null argument");
  if (slices == 0) return ok();
  scoo_windows_kernel<<<slices, kThreads, 0, as_stream(stream)>>>(nnz, ci, sp, win);
  CV_TRY(cudaGetLastError(), "scoo_windows_kernel");
  return ok();
}

int mfp_dev_scratch_release(void) {
  cudaMemPool_t pool;
  const int s = scratch_pool(&pool);
  if (s) return s;
  CV_TRY(cudaDeviceSynchronize(), "cudaDeviceSynchronize");
  CV_TRY(cudaMemPoolTrimTo(pool, 0), "cudaMemPoolTrimTo");
  return ok();
}

int mfp_dev_scratch_bytes(uint64_t *reserved) {
  if (!reserved) return fail(MFP_ERROR_INVALID_VALUE, "null argument");
  cudaMemPool_t pool;
  const int s = scratch_pool(&pool);
  if (s) return s;
  CV_TRY(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, reserved), "cudaMemPoolGetAttribute");
  return ok();
}

int mfp_dev_csr_from_coo(int vt, uint32_t rows, uint32_t cols, uint32_t nnz, const uint32_t *ri, const uint32_t *ci,
                         const double *v, uint32_t *rp, uint32_t *co, void *data, void *stream) {
  return mfp_dev_csr_from_coo_limited(vt, rows, cols, nnz, ri, ci, v, rp, co, data, kRadixPolls, stream);
}

int mfp_dev_csr_from_coo_limited(int vt, uint32_t rows, uint32_t cols, uint32_t nnz, const uint32_t *ri,
                                 const uint32_t *ci, const double *v, uint32_t *rp, uint32_t *co, void *data,
                                 uint32_t polls, void *stream) {
  if (!valid_vt(vt)) return fail(MFP_ERROR_INVALID_VALUE, "bad value type");
  if (vt == MFP_F64)
    return csr_from_coo_t<double>(rows, cols, nnz, ri, ci, v, rp, co, static_cast<double *>(data), polls, stream);
  return csr_from_coo_t<float>(rows, cols, nnz, ri, ci, v, rp, co, static_cast<float *>(data), polls, stream);
}

}  // extern "C"
