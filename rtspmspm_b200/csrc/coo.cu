// COO -> CSR on the GPU: entries in any order become CSR with sorted
// columns, duplicate (i, j) pairs summed in FP32 in the order given.
//
// Replaces the reference's conversion step: it uploads the parsed COO and
// calls cusparseXcoo2csr (cuSparse/src/main.cpp:439-442), which needs
// row-sorted input and keeps duplicates; the reference's files come
// column-major (the reader sorts them on the host first).  Here the entries
// are ordered by a stable LSD radix sort on the key (row << 32) | column,
// 8 bits per pass over the bits the shape needs, so equal keys keep their
// input order; each run of equal keys is then folded left to right (the
// first value, plus the second, ...) exactly as the host reader folds
// duplicates, and row pointers come from the sorted rows.
#include <algorithm>
#include <cstring>
#include <vector>

#include "context.hpp"

namespace spg {
namespace {

constexpr int kSortThreads = 512;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 8;                         // per lane
constexpr int kSortTile = kSortThreads * kSortItems;  // entries per CTA
constexpr int kDigits = 256;
static_assert(kSortThreads >= kDigits, "a thread per digit");
constexpr int kScatterSmem = kSortTile * (8 + 4);  // the tile's keys and values in digit order

// Where a sort pass reads its entries: the first one from the COO arrays
// (entries outside the matrix get key 0 and raise a flag in the counting
// kernel), the others from the previous pass.
struct CooIn {
  const int32_t* ri;
  const int32_t* ci;
  int64_t rows, cols;
  int* flags;
  const uint64_t* key;
  const float* val;
};

template <bool FIRST>
__device__ __forceinline__ uint64_t entry_key(const CooIn& in, int64_t i, bool check) {
  if (!FIRST) return in.key[i];
  const int32_t r = in.ri[i], c = in.ci[i];
  if (r < 0 || r >= in.rows || c < 0 || c >= in.cols) {
    if (check) atomicOr(in.flags, kFlagBadIndex);
    return 0;
  }
  return ((uint64_t)(uint32_t)r << 32) | (uint32_t)c;
}

// Digit counts of each tile: hist[d * ntiles + tile].
template <bool FIRST>
__global__ void __launch_bounds__(kSortThreads) k_radix_hist(CooIn in, int64_t n, int shift, int64_t ntiles,
                                                             int64_t* hist) {
  __shared__ int cnt[kDigits];
  if (threadIdx.x < kDigits) cnt[threadIdx.x] = 0;
  __syncthreads();
  const int64_t t0 = blockIdx.x * (int64_t)kSortTile;
  for (int q = threadIdx.x; q < kSortTile; q += kSortThreads) {
    const int64_t i = t0 + q;
    if (i < n) atomicAdd(&cnt[(int)((entry_key<FIRST>(in, i, true) >> shift) & 0xffu)], 1);
  }
  __syncthreads();
  if (threadIdx.x < kDigits) hist[(int64_t)threadIdx.x * ntiles + blockIdx.x] = cnt[threadIdx.x];
}

// Stable scatter of one tile: warp w owns entries [w * 32 * kSortItems, (w + 1) * 32 * kSortItems)
// of the tile, taken 32 consecutive at a time, so an entry's rank among the
// tile's entries of its digit follows (warp, step, lane) = input order.  The
// tile is first ordered by digit in shared memory (entry at tile position
// lp = the digit's first position in the tile + the counts of earlier warps
// + the entry's rank), then written out by consecutive threads, so each
// digit's run of the tile goes to consecutive global positions (coalesced
// stores; scattering straight from registers ran at 1.1 TB/s).
//
// Bound: __match_any_sync, whose time grows with the distinct digits of a warp
// (2^23 entries: 98 us a pass of 8-bit digits, 66 us of 4-bit ones; the 24
// bytes an entry moves take 31 us at the copy peak).  So it runs once an
// entry, the rank kept in a register (143 -> 98 us against matching again for
// the positions); eight ballots in its place were slower (153 us with two
// rounds).  512 threads a tile: 256 took as long here but made twice the tiles
// to count and scan (2^26 entries: 6.5 against 6.0 ms a call), 1,024 and 16
// entries a lane were slower.  off:
// exclusive scan of hist (digit-major), the first output position of each
// (digit, tile).  ALONE: the only tile, which needs none (one entry: 82 -> 68 us a
// call) and raises the flags that the counting kernel does.  Dynamic shared memory: kSortTile keys and values.
template <bool FIRST, bool ALONE>
__global__ void __launch_bounds__(kSortThreads) k_radix_scatter(CooIn in, int64_t n, int shift, int64_t ntiles,
                                                                const int64_t* off, uint64_t* kout, float* vout) {
  __shared__ int base[kSortWarps][kDigits];
  __shared__ int first[kDigits];  // the digit's first position in the tile's digit order
  extern __shared__ uint64_t sm_sort[];
  uint64_t* sk = sm_sort;
  float* sv = reinterpret_cast<float*>(sm_sort + kSortTile);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  for (int d = lane; d < kDigits; d += 32) base[w][d] = 0;
  __syncwarp();
  const int64_t t0 = blockIdx.x * (int64_t)kSortTile;
  const int64_t w0 = t0 + (int64_t)w * (kSortItems * 32);
  uint64_t k[kSortItems];
  float v[kSortItems];
#pragma unroll
  for (int j = 0; j < kSortItems; ++j) {
    const int64_t i = w0 + j * 32 + lane;
    k[j] = i < n ? entry_key<FIRST>(in, i, ALONE) : 0;
    v[j] = i < n ? in.val[i] : 0.f;
  }
  // the warp's count per digit and, from the counts so far, each entry's rank
  // among the warp's entries of its digit
  int rank[kSortItems];
#pragma unroll
  for (int j = 0; j < kSortItems; ++j) {
    const bool act = w0 + j * 32 + lane < n;
    const int d = act ? (int)((k[j] >> shift) & 0xffu) : kDigits + lane;
    const unsigned grp = __match_any_sync(kFull, d);
    const int before = act ? base[w][d] : 0;
    rank[j] = before + __popc(grp & lt);
    __syncwarp();
    if (act && (grp & lt) == 0u) base[w][d] = before + __popc(grp);
    __syncwarp();
  }
  __syncthreads();
  // per digit: its total in the tile and, per warp, the start of the warp's entries
  {
    constexpr int kDigitWarps = kDigits / 32;
    __shared__ int wtot[kDigitWarps];
    const int d = threadIdx.x;
    int run = 0, incl = 0;
    if (d < kDigits) {
#pragma unroll
      for (int x = 0; x < kSortWarps; ++x) {
        const int c = base[x][d];
        base[x][d] = run;
        run += c;
      }
      // exclusive scan of the digit totals across the CTA (digit d = thread d)
      incl = warp_incl_scan(run);
      if (lane == 31) wtot[w] = incl;
    }
    __syncthreads();
    if (d < kDigits) {
      int pre = incl - run;
#pragma unroll
      for (int x = 0; x < kDigitWarps; ++x) pre += x < w ? wtot[x] : 0;
      first[d] = pre;
#pragma unroll
      for (int x = 0; x < kSortWarps; ++x) base[x][d] += pre;
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kSortItems; ++j) {
    if (w0 + j * 32 + lane < n) {
      const int lp = base[w][(int)((k[j] >> shift) & 0xffu)] + rank[j];
      sk[lp] = k[j];
      sv[lp] = v[j];
    }
  }
  __syncthreads();
  // the tile in digit order, written by consecutive threads
  const int cnt = (int)min((int64_t)kSortTile, n - t0);
  for (int q = threadIdx.x; q < cnt; q += kSortThreads) {
    const uint64_t key = sk[q];
    const int d = (int)((key >> shift) & 0xffu);
    const int64_t pos = ALONE ? q : off[(int64_t)d * ntiles + blockIdx.x] + (q - first[d]);
    kout[pos] = key;
    vout[pos] = sv[q];
  }
}

// Entries of each fold tile that start a run of equal keys.
constexpr int kFoldThreads = 512;
constexpr int kFoldItems = 4;  // per lane, 32 consecutive at a time
constexpr int kFoldTile = kFoldThreads * kFoldItems;

__device__ __forceinline__ bool run_head(const uint64_t* key, int64_t i, uint64_t k) { return i == 0 || key[i - 1] != k; }

__global__ void __launch_bounds__(kFoldThreads) k_count_runs(const uint64_t* key, int64_t n, int64_t* runs) {
  __shared__ int cnt[kFoldThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t i0 = blockIdx.x * (int64_t)kFoldTile + w * (32 * kFoldItems) + lane;
  int c = 0;
#pragma unroll
  for (int j = 0; j < kFoldItems; ++j) {
    const int64_t i = i0 + j * 32;
    c += i < n && run_head(key, i, key[i]);
  }
  c = __reduce_add_sync(kFull, c);
  if (lane == 0) cnt[w] = c;
  __syncthreads();
  if (w == 0) {
    c = __reduce_add_sync(kFull, lane < kFoldThreads / 32 ? cnt[lane] : 0);
    if (lane == 0) runs[blockIdx.x] = c;
  }
}

// One thread per run: its column and the left fold of its values into the
// run's output entry (base[tile] = runs before the tile), and the row pointers
// its entry opens: those of the rows after the row before it, up to its own.
// The last entry also closes the rows behind it.
__global__ void __launch_bounds__(kFoldThreads) k_fold_runs(const uint64_t* key, const float* val, int64_t n,
                                                            const int64_t* base, int64_t m, int64_t rows,
                                                            int32_t* col, float* out_val, int64_t* rp) {
  __shared__ int cnt[kFoldThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t i0 = blockIdx.x * (int64_t)kFoldTile + w * (32 * kFoldItems) + lane;
  uint64_t k[kFoldItems];
  unsigned heads[kFoldItems];
  int c = 0;
#pragma unroll
  for (int j = 0; j < kFoldItems; ++j) {
    const int64_t i = i0 + j * 32;
    k[j] = i < n ? key[i] : 0;
    heads[j] = __ballot_sync(kFull, i < n && run_head(key, i, k[j]));
    c += __popc(heads[j]);
  }
  if (lane == 0) cnt[w] = c;
  __syncthreads();
  int64_t u0 = base[blockIdx.x];
  for (int x = 0; x < w; ++x) u0 += cnt[x];
#pragma unroll
  for (int j = 0; j < kFoldItems; ++j) {
    const int64_t i = i0 + j * 32;
    if ((heads[j] >> lane) & 1u) {
      const int64_t u = u0 + __popc(heads[j] & ((1u << lane) - 1u));
      float s = val[i];
      int64_t q = i + 1;
      for (; q < n && key[q] == k[j]; ++q) s = __fadd_rn(s, val[q]);
      col[u] = (int32_t)(uint32_t)(k[j] & 0xffffffffu);
      out_val[u] = s;
      const int64_t r = (int64_t)(k[j] >> 32);
      for (int64_t x = i == 0 ? 0 : (int64_t)(key[i - 1] >> 32) + 1; x <= r; ++x) rp[x] = u;
      if (q == n)
        for (int64_t x = r + 1; x <= rows; ++x) rp[x] = m;
    }
    u0 += __popc(heads[j]);
  }
}

int bits_for(int64_t n) {
  int b = 0;
  while (b < 62 && ((int64_t)1 << b) < n) ++b;
  return b;
}

}  // namespace

// COO (device arrays) -> device CSR; see the file comment.
spg_status coo_to_csr_device(spg_ctx* ctx, int64_t rows, int64_t cols, int64_t n, const int32_t* ri, const int32_t* ci,
                             const float* vi, spg_csr* out) {
  const LaunchCtx lc = launch_ctx(ctx);
  DevBuf k0, k1, v0, v1;
  SPG_TRY(k0.alloc(ctx, (size_t)std::max<int64_t>(n, 1) * 8));
  SPG_TRY(k1.alloc(ctx, (size_t)std::max<int64_t>(n, 1) * 8));
  SPG_TRY(v0.alloc(ctx, (size_t)std::max<int64_t>(n, 1) * 4));
  SPG_TRY(v1.alloc(ctx, (size_t)std::max<int64_t>(n, 1) * 4));
  // LSD passes over the column bits, then over the row bits
  const int cbits = bits_for(cols), rbits = bits_for(rows);
  const int64_t ntiles = (n + kSortTile - 1) / kSortTile;
  DevBuf hist, tmp;
  SPG_TRY(hist.alloc(ctx, (size_t)std::max<int64_t>(kDigits * ntiles + 1, 1) * 8));
  SPG_TRY(tmp.alloc(ctx, (size_t)scan_temp_elems(kDigits * ntiles + 1) * 8));
  std::vector<int> shifts;
  for (int s = 0; s < cbits; s += 8) shifts.push_back(s);
  for (int s = 0; s < rbits; s += 8) shifts.push_back(32 + s);
  // a 1 x 1 matrix or a single entry: one pass that checks the entries and makes their keys
  if (shifts.empty() || n == 1) shifts.assign(1, 0);
  CooIn in{ri, ci, rows, cols, ctx->d_flags, nullptr, vi};
  const uint64_t* kin = nullptr;  // the sorted entries
  const float* vin = nullptr;
  if (n > 0) {
    uint64_t* kout = k0.as<uint64_t>();
    float* vout = v0.as<float>();
    const bool alone = ntiles == 1;
    auto pass = [&](auto hist_kernel, auto scatter_kernel, int shift) -> spg_status {
      SPG_CUDA(ctx, cudaFuncSetAttribute(scatter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kScatterSmem));
      if (!alone) {
        hist_kernel<<<(unsigned)ntiles, kSortThreads, 0, lc.stream>>>(in, n, shift, ntiles, hist.as<int64_t>());
        launch_excl_scan(hist.as<int64_t>(), kDigits * ntiles, hist.as<int64_t>(), tmp.as<int64_t>(), lc);
      }
      scatter_kernel<<<(unsigned)ntiles, kSortThreads, kScatterSmem, lc.stream>>>(in, n, shift, ntiles,
                                                                                  hist.as<int64_t>(), kout, vout);
      in.key = kin = kout;
      in.val = vin = vout;
      kout = kin == k0.as<uint64_t>() ? k1.as<uint64_t>() : k0.as<uint64_t>();
      vout = vin == v0.as<float>() ? v1.as<float>() : v0.as<float>();
      return SPG_OK;
    };
    for (size_t i = 0; i < shifts.size(); ++i) {
      const auto first = alone ? k_radix_scatter<true, true> : k_radix_scatter<true, false>;
      const auto later = alone ? k_radix_scatter<false, true> : k_radix_scatter<false, false>;
      if (i == 0) SPG_TRY(pass(k_radix_hist<true>, first, shifts[i]));
      else SPG_TRY(pass(k_radix_hist<false>, later, shifts[i]));
    }
  }
  // runs of equal keys -> unique entries
  const int64_t nfold = (n + kFoldTile - 1) / kFoldTile;
  DevBuf runs;
  SPG_TRY(runs.alloc(ctx, (size_t)(nfold + 1) * 8));
  if (n > 0) k_count_runs<<<(unsigned)nfold, kFoldThreads, 0, lc.stream>>>(kin, n, runs.as<int64_t>());
  launch_excl_scan(runs.as<int64_t>(), nfold, runs.as<int64_t>(), tmp.as<int64_t>(), lc);
  int64_t m = 0;
  SPG_TRY(stage_reads(ctx, {{ctx->h_stage + 52, runs.as<int64_t>() + nfold, 8}, {ctx->h_stage + 53, ctx->d_flags, 4}}));
  int f = 0;
  SPG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  m = ctx->h_stage[52];
  std::memcpy(&f, &ctx->h_stage[53], sizeof f);
  if (f) {
    SPG_CUDA(ctx, cudaMemsetAsync(ctx->d_flags, 0, sizeof(int), ctx->stream));
    if (f & kFlagBadIndex) return fail(ctx, SPG_ERR_INVALID_ARG, "COO entry outside [0, rows) x [0, cols)");
  }
  DevBuf col, val, rp;
  SPG_TRY(col.alloc_result(ctx, (size_t)m * 4));
  SPG_TRY(val.alloc_result(ctx, (size_t)m * 4));
  SPG_TRY(rp.alloc_result(ctx, (size_t)(rows + 1) * 8));
  if (n > 0)
    k_fold_runs<<<(unsigned)nfold, kFoldThreads, 0, lc.stream>>>(kin, vin, n, runs.as<int64_t>(), m, rows,
                                                                 col.as<int32_t>(), val.as<float>(), rp.as<int64_t>());
  else
    SPG_CUDA(ctx, cudaMemsetAsync(rp.get(), 0, (size_t)(rows + 1) * 8, ctx->stream));
  SPG_CUDA(ctx, cudaGetLastError());
  SPG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  std::memset(out, 0, sizeof *out);
  out->rows = rows;
  out->cols = cols;
  out->nnz = m;
  out->capacity = m;
  out->index_bits = 64;
  out->location = SPG_DEVICE;
  out->row_ptr = rp.release();
  out->col_idx = static_cast<int32_t*>(col.release());
  out->val = static_cast<float*>(val.release());
  out->owner = 1;
  return SPG_OK;
}

}  // namespace spg

extern "C" spg_status spg_coo_to_csr(spg_ctx* ctx, int64_t rows, int64_t cols, int64_t n, const int32_t* row_idx,
                                     const int32_t* col_idx, const float* val, int32_t location, spg_csr* out) {
  using namespace spg;
  if (!ctx || !out) return SPG_ERR_INVALID_ARG;
  std::memset(out, 0, sizeof *out);
  if (rows < 0 || cols < 0 || n < 0) return fail(ctx, SPG_ERR_INVALID_ARG, "negative dimension");
  if (rows > INT32_MAX || cols > INT32_MAX) return fail(ctx, SPG_ERR_UNSUPPORTED, "more than 2^31-1 rows or columns");
  if (n > 0 && (!row_idx || !col_idx || !val)) return fail(ctx, SPG_ERR_INVALID_ARG, "null COO array");
  if (location != SPG_HOST && location != SPG_DEVICE) return fail(ctx, SPG_ERR_INVALID_ARG, "bad location");
  SPG_CUDA(ctx, cudaSetDevice(ctx->device));
  if (location == SPG_DEVICE) return coo_to_csr_device(ctx, rows, cols, n, row_idx, col_idx, val, out);
  DevBuf ri, ci, vi;
  SPG_TRY(ri.alloc(ctx, (size_t)n * 4));
  SPG_TRY(ci.alloc(ctx, (size_t)n * 4));
  SPG_TRY(vi.alloc(ctx, (size_t)n * 4));
  if (n > 0) {
    SPG_CUDA(ctx, cudaMemcpyAsync(ri.get(), row_idx, (size_t)n * 4, cudaMemcpyHostToDevice, ctx->stream));
    SPG_CUDA(ctx, cudaMemcpyAsync(ci.get(), col_idx, (size_t)n * 4, cudaMemcpyHostToDevice, ctx->stream));
    SPG_CUDA(ctx, cudaMemcpyAsync(vi.get(), val, (size_t)n * 4, cudaMemcpyHostToDevice, ctx->stream));
  }
  return coo_to_csr_device(ctx, rows, cols, n, ri.as<int32_t>(), ci.as<int32_t>(), vi.as<float>(), out);
}
