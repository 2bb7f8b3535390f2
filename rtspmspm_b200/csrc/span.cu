// Symbolic rows whose columns lie in a narrow span: a bitmap of the span in
// the warp's shared memory instead of a hash table of the columns.
//
// A hash step probes, claims and retries in branches that split the warp (the
// lanes wait for the longest chain among them), and a table for many distinct
// columns is half full; here a step is one word read and, for a column not yet
// seen, one atomic OR, at the price of counting and clearing the span's words.
// Erdos-Renyi 65,536 x 32 (1,024 products a row over 2,048 words): 1.64 ->
// 0.52 ms; 27-point stencil 61^3 0.56 -> 0.36 ms, 96^3 (1,165 words) 2.03 ->
// 1.73 ms.  Bound: the atomics, a shared-memory wavefront a lane (l1tex 93 %
// on the stencil at 830 instructions a row).
//
// The same bitmap with counts as the numeric accumulator (an entry's place by
// population count, no sort) was measured slower than the hash rows and
// dropped: stencil 96^3 2.94 -> 4.65 ms.  It reads the rows of B twice and its
// 9 KB a warp leave 24 warps an SM.
#include <algorithm>

#include "common.cuh"
#include "kernels.hpp"

namespace spg {

// First column of the row's bitmap (a multiple of 32): the smallest column of
// its products.
template <bool R32>
__device__ __forceinline__ int32_t span_start(const DCsr& A, const DCsr& B, int64_t s, int64_t e) {
  unsigned lo = 0x7fffffffu;
  for (int64_t p = s + lane_id(); p < e; p += 32) {
    const int32_t k = A.col[p];
    const auto bs = RowOff<R32>::at(B, k);
    if (RowOff<R32>::at(B, k + 1) > bs) lo = min(lo, (unsigned)B.col[bs]);
  }
  return (int32_t)(__reduce_min_sync(kFull, lo) & ~31u);
}

// Sets the bit of every product's column; false (in some lane) when one lies
// outside the `words` words.  No order: segments are taken four at a time.
template <bool R32>
__device__ __forceinline__ bool span_mark(const DCsr& A, const DCsr& B, int64_t s, int64_t e, int32_t lo, int words,
                                          uint32_t* bits) {
  using Off = typename RowOff<R32>::T;
  const int lane = lane_id();
  const uint32_t last = (uint32_t)words * 32u - 1u;
  uint32_t far = 0;
  auto mark = [&](int32_t c) {
    uint32_t off = (uint32_t)(c - lo);
    far = max(far, off);
    off = min(off, last);
    const uint32_t bit = 1u << (off & 31);
    if (!(bits[off >> 5] & bit)) atomicOr(&bits[off >> 5], bit);
  };
  for (int64_t base = s; base < e; base += 32) {
    const int64_t p = base + lane;
    Off bs = 0;
    int len = 0;
    if (p < e) {
      const int32_t k = A.col[p];
      bs = RowOff<R32>::at(B, k);
      len = (int)(RowOff<R32>::at(B, k + 1) - bs);
    }
    const int n = (int)min((int64_t)32, e - base);
    if (__any_sync(kFull, lane < n && (len < kPackBelow || len > 32))) {
      for_each_col(B.col, bs, len, mark);
      continue;
    }
    for (int i = 0; i < n; i += 4) {
      int32_t c[4];
      int l[4];
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int from = min(i + x, n - 1);  // past the end: the last segment once more
        const Off b = __shfl_sync(kFull, bs, from);
        l[x] = __shfl_sync(kFull, len, from);
        c[x] = B.col[b + min(lane, l[x] - 1)];
      }
#pragma unroll
      for (int x = 0; x < 4; ++x) mark(c[x]);
    }
  }
  __syncwarp();
  return far <= last;
}

// Warp per row: the exact count of its columns.
template <bool R32>
__global__ void __launch_bounds__(256) k_sym_span(DCsr A, DCsr B, const int32_t* rows, int64_t nrows, int words,
                                                  int64_t* nnz, int* flags) {
  extern __shared__ __align__(16) uint32_t sm_span[];
  const int lane = lane_id();
  uint32_t* bits = sm_span + (size_t)(threadIdx.x >> 5) * words;
  for (int i = lane; i < words; i += 32) bits[i] = 0u;
  __syncwarp();
  const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  uint4* b4 = reinterpret_cast<uint4*>(bits);
  for (int64_t idx = gw; idx < nrows; idx += nw) {
    const int32_t row = rows[idx];
    const int64_t s = A.rp[row], e = A.rp[row + 1];
    const int32_t lo = span_start<R32>(A, B, s, e);
    const bool ok = span_mark<R32>(A, B, s, e, lo, words, bits);
    int c = 0;
    for (int i = lane; i < words / 4; i += 32) {
      const uint4 w = b4[i];
      c += __popc(w.x) + __popc(w.y) + __popc(w.z) + __popc(w.w);
      b4[i] = make_uint4(0u, 0u, 0u, 0u);
    }
    c = __reduce_add_sync(kFull, c);
    if (lane == 0) nnz[row] = c;
    if (!ok) raise_flag(flags, kFlagBadIndex);
    __syncwarp();
  }
}

// ---- launchers ---------------------------------------------------------------

// CTAs of 4 warps, as many an SM as fit, no more than the rows need.
constexpr int kSpanWarps = 4;
static_assert(kSpanWarps * span_bin_words(kNumSpanBins - 1) * 4 <= 48 * 1024, "within every kernel's default limit");
template <typename Kernel>
static int span_grid(Kernel kernel, size_t smem, int64_t nrows, const LaunchCtx& lc) {
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kSpanWarps * 32, smem);
  return (int)std::max<int64_t>(
      1, std::min<int64_t>((nrows + kSpanWarps - 1) / kSpanWarps, (int64_t)lc.sms * std::max(1, per_sm)));
}

template <bool R32>
static void sym_span_one(int words, const DCsr& A, const DCsr& B, const int32_t* rows, int64_t nrows, int64_t* nnz,
                         int* flags, const LaunchCtx& lc) {
  const size_t smem = (size_t)kSpanWarps * words * 4;
  const int blocks = span_grid(k_sym_span<R32>, smem, nrows, lc);
  k_sym_span<R32><<<blocks, kSpanWarps * 32, smem, lc.stream>>>(A, B, rows, nrows, words, nnz, flags);
}

void launch_sym_span(int bin, const DCsr& A, const DCsr& B, const int32_t* rows, int64_t nrows, int64_t* nnz,
                     int* flags, const LaunchCtx& lc) {
  if (nrows == 0) return;
  const int words = span_bin_words(bin - kBinSpan);
  if (B.rp32) sym_span_one<true>(words, A, B, rows, nrows, nnz, flags, lc);
  else sym_span_one<false>(words, A, B, rows, nrows, nnz, flags, lc);
}

}  // namespace spg
