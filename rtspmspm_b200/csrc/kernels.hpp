// Host-side declarations of the SpGEMM kernel launchers.
#pragma once

#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>

#ifndef SPG_TILE_SHIFT
#define SPG_TILE_SHIFT 11
#endif

namespace spg {

struct DCsr;

// Bin ids.  Warp-hash bins 0..7 hold tables of 2^(5+bin) slots.
constexpr int kMinLogT = 5;
constexpr int kMaxLogT = 12;
constexpr int kNumWarpBins = kMaxLogT - kMinLogT + 1;  // 8
constexpr int kBinBlock = 8;   // symbolic: CTA hash table; numeric: CTA hash of 2^12 slots
constexpr int kBinDense = 9;   // symbolic: CTA bitmap over the column span; numeric: CTA hash of 2^14 slots
// Numeric and learned: rows expanded, sorted and folded (esc_row), by products.
constexpr int kBinEsc = 10;
constexpr int kNumEscBins = 5;
// Largest products of bin kBinEsc + i.
// (32-bit words of shared memory a warp of it takes: esc_bin_words, warp_row.cuh)
constexpr int esc_bin_products(int i) { return i == 0 ? 320 : i == 1 ? 640 : i == 2 ? 1152 : i == 3 ? 2048 : 4010; }
// Symbolic: rows with a bitmap of their column span (span.cu), by its words.
constexpr int kBinSpan = kBinEsc + 1;
constexpr int kNumSpanBins = 3;
// The largest class ends at 65,536 columns because a warp's 8 KB leave an SM 28
// warps; a class of 3,072 words would pay from about 480 products a row (80,000
// columns, symbolic stage at 288 | 480 | 1,024 products 0.51 | 0.65 | 1.16 ms hashed,
// 0.50 | 0.58 | 0.64 in it), but not in the place of this one (60,000 columns, 1,024
// products 0.47 -> 0.63).
constexpr int kSpanMinProd = 64;  // fewest products of such a row
constexpr int span_bin_words(int i) { return i == 0 ? 576 : i == 1 ? 1216 : 2048; }
// Rows of at most early_max columns that may leave the warp tables early
// (big_row): behind the other big rows of a symbolic binning, before those of a
// numeric one, so that either list goes on without a gap.
constexpr int kBinEarlySym = kBinEsc;
constexpr int kBinEarly = kBinEsc + kNumEscBins;
constexpr int kBinHeavy = kBinEarly + 1;          // numeric: column-tiled heavy rows
constexpr int kBinEmpty = kBinHeavy + 1;          // no products
constexpr int kNumBins = kBinEmpty + 1;

// Log2 of the CTA-wide numeric hash tables of kBinBlock / kBinDense.
constexpr int kBlkLogSmallT = 12;
constexpr int kBlkLogLargeT = 14;

constexpr int kBinSymbolic = 0;
constexpr int kBinNumeric = 1;
constexpr int kBinLearned = 2;

// Warps per CTA of the heavy tile kernel: up to 8 per-warp tiles (floats,
// bitmap, 32-float stage) within 227 KB of shared memory; the grid holds as
// many CTAs per SM as fit.
constexpr int kTileWarpBytes = ((1 << SPG_TILE_SHIFT) + (1 << SPG_TILE_SHIFT) / 32 + 32) * 4;
constexpr int kTileWarps = (227 * 1024) / kTileWarpBytes > 8 ? 8 : (227 * 1024) / kTileWarpBytes;
// Heavy-row units (heavy_unit.cu): threads and 32-bit words of shared memory
// a CTA, and the words a unit's rank words and entries may take (a spare word
// behind them).
#ifndef SPG_UNIT_WORDS
#define SPG_UNIT_WORDS 5600
#endif
#ifndef SPG_UNIT_THREADS
#define SPG_UNIT_THREADS 128
#endif
constexpr int kUnitThreads = SPG_UNIT_THREADS;
constexpr int kUnitWords = SPG_UNIT_WORDS;
constexpr int kUnitCost = kUnitWords - 4;
constexpr int kDenseWindowWords = 40960;   // 1,310,720 columns of bitmap per window

struct BinParams {
  int64_t warp_cap;    // largest bound (symbolic) / nnz (numeric) on a warp table
  int64_t block_cap;   // largest bound on the symbolic CTA table
  int warp_log_max;    // log2 of the largest warp table
  float max_load;      // numeric table load factor
  // numeric / learned binning: rows with more than block_min entries go to
  // the CTA-wide hash bins (kBinBlock up to blk_small_cap entries, kBinDense
  // up to blk_large_cap); block_min = INT64_MAX and the caps 0 turn them off
  int64_t block_min;
  int64_t blk_small_cap;
  int64_t blk_large_cap;
  int64_t esc_cap;     // most entries of a row in the expand-sort-fold bins
  int esc_prod;        // and most products (esc_bin_products of the last bin in use; 0: none)
  int64_t early_max;   // most entries of a row that a table of 2^kEarlyLog slots holds
  int64_t heavy_min;   // rows of more entries may be heavy below warp_cap too (big_row)
};

// Rows of more entries than this leave the warp tables for the heavy-row units
// where their bitmap allows (big_row).  A table of 2^11 or 2^12 slots leaves an
// SM 8 or 4 warps.  Call with R-MAT 16 (4 edges a vertex), 14 and 12, plain:
// from 2,048 entries 2.31, 2.53 and 1.84 ms, from 1,024 1.86, 1.79 and 1.14,
// from 512 1.52, 1.53 and 0.80, from 256 1.46, 1.52 and 0.81.
constexpr int64_t kHeavyMin = 512;
// Those that a table of 2^kEarlyLog slots holds (early_max columns) leave only
// beside others past it or when they are kEarlyRows or more: the units' launches take 40 us a call, and fewer rows
// are one wave of tables (new values of 3,000 rows, 151 of them of 513 to 560
// entries, 251 -> 203 us, of R-MAT 10, 31 of its 1,024 rows, 376 -> 335).
constexpr int kEarlyLog = 11;
constexpr int64_t kEarlyRows = 256;
// A row bounded by u entries, `likely` of them distinct if its products fell at
// random on the columns they can reach, goes the way of the heavy rows (symbolic
// bitmap, units) when it is past the warp tables, or likely past heavy_min while
// its columns' bitmap has at most 4 words an entry: clearing and counting it
// then costs no more than hashing.  Rows of many products on few columns stay
// (60,000 rows of 720 products in bands of 300 columns, counted in bitmaps and
// then hashed all the same: 1,635 us a call, hashed twice 1,260).
#ifdef __CUDACC__
__host__ __device__
#endif
inline bool big_row(int64_t u, int64_t likely, int64_t cols, int64_t warp_cap, int64_t heavy_min) {
  return u > warp_cap || (likely > heavy_min && cols <= 128 * u);
}

// Whether such a row (prod products, out entries) is folded all the same: up to
// 1,152 products, or when nearly all of them are distinct.  The fold's larger
// bins hold 8 and 4 warps an SM.  From 1,153 products to the units: R-MAT 14
// and 12 plain 2.59 -> 1.87 and 1.85 -> 1.12 ms; of Erdos-Renyi rows (100,000 x
// 40, 1,600 products with 1,587 distinct) to the units 4.36 -> 4.87 ms, folded.
#ifdef __CUDACC__
__host__ __device__
#endif
inline bool fold_big(int64_t prod, int64_t out) { return prod <= 1152 || 8 * out >= 7 * prod; }

// BinParams with the CTA-wide numeric bins turned off (paths that only
// launch the warp bins and the heavy tiles).
inline BinParams without_block_bins(BinParams bp) {
  bp.block_min = INT64_MAX;
  bp.blk_small_cap = 0;
  bp.blk_large_cap = 0;
  bp.esc_cap = bp.warp_cap;
  bp.heavy_min = INT64_MAX;
  return bp;
}

struct LaunchCtx {
  cudaStream_t stream;
  int sms;
  int device;
  unsigned long long driver_ctx;  // driver_ctx_id() of the device's context
};

// A number of the current driver context that no other context of the process
// has or had, or 0.  A device reset ends a context and with it what was set or
// made there: kernels' shared-memory limits, memory pools.
unsigned long long driver_ctx_id();

void launch_widen_rp(const int32_t* in, int64_t n, int64_t* out, const LaunchCtx& lc);
void launch_narrow_rp(const int64_t* in, int64_t n, int32_t* out, const LaunchCtx& lc);
void launch_validate(const DCsr& M, int64_t nnz, int* flags, const LaunchCtx& lc);
// Products of every row and, when `span` is given, the words of its column
// span's bitmap: 0 unknown, below 0 (for rows past heavy_min) when the row takes
// no span bin.  Rows of more than `most` possible columns have none.
void launch_row_products(const DCsr& A, const DCsr& B, int64_t* prod, const LaunchCtx& lc, int32_t* span = nullptr,
                         int64_t most = 0, int64_t heavy_min = INT64_MAX);
// The same words for the `count` (on the device) listed rows, 0 for all others.
void launch_listed_spans(const DCsr& A, const DCsr& B, const int32_t* rows, const unsigned long long* count,
                         const int64_t* prod, int32_t* span, int64_t most, int64_t heavy_min, const LaunchCtx& lc);

// Small products (at most kSmallMaxRows rows of A, every row of at most
// 2^kSmallLogT products): products and exact counts per row in one launch
// (nnz[row] = -1 for a row of more products), then one CTA scans the counts
// into C's row pointers (int64 in place, int32 into rp32 when given and the
// total fits) and puts the total, the products, the largest count and the
// too-large rows into out[0..3] (mapped host words).
constexpr int kSmallLogT = 11;
constexpr int kSmallCountWarps = 4;
constexpr int kSmallScanThreads = 1024;
constexpr int64_t kSmallMaxRows = 65536;
constexpr int kSmallDefaultRows = 8192;
// `stop` (one device word, zero between calls): set by the counting launch
// at its first too-large row so that the remaining rows skip their counts;
// the scan clears it.
void launch_small_count(const DCsr& A, const DCsr& B, int64_t* prod, int64_t* nnz, unsigned long long* stop,
                        int* flags, const LaunchCtx& lc);
void launch_small_scan(int64_t* nnz, const int64_t* prod, int64_t rows, int32_t* rp32, unsigned long long* stop,
                       int64_t* out, const LaunchCtx& lc);
// Default smallest product count of an expand-sort-fold row.  Numeric stage
// of 200,000-row Erdos-Renyi products with 36 | 64 | 100 | 144 products a row:
// from 128 products 0.32 | 0.44 | 0.52 | 0.53 ms, from 64 0.30 | 0.33 | 0.37 |
// 0.44, from 32 0.24 | 0.29 | 0.35 | 0.43; 20 uneven products 3.40, 3.15 and
// 3.08 ms a call.
constexpr int kEscMinProd = 32;
// Expand-sort-fold rows in the warp numeric kernels: the row products
// (nullptr: off) and the smallest product count that takes the path
// (0: off).
struct EscArgs {
  const int64_t* prod = nullptr;
  int min_prod = 0;
  float per_margin = 0.f;  // learned: 1 / margin and slack of a capacity (esc_guess)
  int slack = 0;
};
void launch_sum(const int64_t* v, int64_t n, unsigned long long* out, const LaunchCtx& lc);
// Rows into bins by their key; with `esc`, numeric and learned binnings send
// the rows it wants to the expand-sort-fold bins, with `span`, symbolic ones
// the rows of few span words to the span bins.
void launch_binning(const int64_t* key, int64_t rows, int64_t cols, int mode, const BinParams& bp,
                    uint8_t* bin_of_row, int64_t* counts, int64_t* offsets, int64_t* cursors, int32_t* lists,
                    const LaunchCtx& lc, const EscArgs& esc = EscArgs{}, const int32_t* span = nullptr);
int64_t scan_temp_elems(int64_t n);
void launch_excl_scan(const int64_t* in, int64_t n, int64_t* out, int64_t* tmp, const LaunchCtx& lc);

void launch_sym_warp(int log_t, const DCsr& A, const DCsr& B, const int32_t* rows, int64_t nrows, int64_t* nnz,
                     int* flags, const LaunchCtx& lc, int wpb);
void launch_sym_block(const DCsr& A, const DCsr& B, const int32_t* rows, int64_t nrows, int log_table,
                      int64_t slot_base, int64_t* nnz, int32_t* big_slot, int32_t* tile_cnt, int ntiles, int* flags,
                      const LaunchCtx& lc);
void launch_sym_dense(const DCsr& A, const DCsr& B, const int32_t* rows, int64_t nrows, int64_t slot_base,
                      int64_t* nnz, int32_t* big_slot, int32_t* tile_cnt, int ntiles, uint32_t* bitmap, int* flags,
                      const LaunchCtx& lc);
void launch_num_warp(int log_t, const DCsr& A, const DCsr& B, const int32_t* rows, int64_t nrows,
                     const int64_t* c_rp, int32_t* c_col, float* c_val, int* flags, const LaunchCtx& lc, int wpb,
                     const EscArgs& esc = EscArgs{});
void launch_num_warp_learned(int log_t, const DCsr& A, const DCsr& B, const int32_t* rows, int64_t nrows,
                             const int64_t* cap, const int64_t* slab_off, int32_t* slab_col, float* slab_val,
                             int64_t* nnz_out, int32_t* retry_rows, unsigned long long* retry_count, int* flags,
                             const LaunchCtx& lc, int wpb, const EscArgs& esc = EscArgs{});
// Span bitmaps: exact counts of the rows of a symbolic bin.
void launch_sym_span(int bin, const DCsr& A, const DCsr& B, const int32_t* rows, int64_t nrows, int64_t* nnz,
                     int* flags, const LaunchCtx& lc);
// Expand-sort-fold pass over the rows of the bins kBinEsc .. (bin_off: the
// binning's offsets into `lists`, on the host): into C (off = its row pointers,
// cap = null; the counts are checked) or into the slab (off = its offsets; rows of
// more than cap[row] entries to `retry`, nnz -1).  Returns its launches.
int launch_num_esc(const int64_t* bin_off, const DCsr& A, const DCsr& B, const int32_t* lists, const int64_t* prod,
                   const int64_t* off, int32_t* out_col, float* out_val, const int64_t* cap, int64_t* nnz,
                   int32_t* retry, unsigned long long* retry_count, int* flags, const LaunchCtx& lc, int wpb);
// CTA-wide hash numeric pass over the rows of bin kBinBlock (2^12-slot
// tables) or kBinDense (2^14) of a numeric / learned binning.
void launch_num_block(int bin, const DCsr& A, const DCsr& B, const int32_t* rows, int64_t nrows, const int64_t* c_rp,
                      int32_t* c_col, float* c_val, int* flags, const LaunchCtx& lc);
void launch_num_block_learned(int bin, const DCsr& A, const DCsr& B, const int32_t* rows, int64_t nrows,
                              const int64_t* cap, const int64_t* slab_off, int32_t* slab_col, float* slab_val,
                              int64_t* nnz_out, int32_t* retry_rows, unsigned long long* retry_count, int* flags,
                              const LaunchCtx& lc);
// Copies a few runs of 32-bit words with one small kernel (dst may be mapped
// pinned host memory: the read-back then needs no copy engine).
struct StageCopies {
  static constexpr int kMax = 4;
  const uint32_t* src[kMax];
  uint32_t* dst[kMax];
  int words[kMax];
  int n;
};
void launch_copy_words(const StageCopies& c, const LaunchCtx& lc);
// Row pointers shifted by `off` into an int32 (out_bits 32) or int64 array.
void launch_shift_rp(const int64_t* in, int64_t n, int64_t off, void* out, int out_bits, const LaunchCtx& lc);
// Value-only recompute: row lengths of C, and heavy-row slots and per-tile
// counts from C's sorted columns (tile_cnt zeroed by the caller).
void launch_row_lengths(const int64_t* rp, int64_t rows, int64_t* len, const LaunchCtx& lc);
void launch_tile_counts_from_cols(const int32_t* heavy_rows, int64_t nheavy, const int64_t* c_rp,
                                  const int32_t* c_col, int ntiles, int32_t* big_slot, int32_t* tile_cnt, int* flags,
                                  const LaunchCtx& lc);
// Per heavy row: tile offsets (scan of the tile counts) and, when nz_cnt is
// given, its number of non-empty tiles.
void launch_tile_offsets(const int32_t* heavy_rows, int64_t nheavy, const int32_t* big_slot, const int32_t* tile_cnt,
                         int ntiles, int32_t* tile_off, int64_t* nz_cnt, const LaunchCtx& lc);
// The non-empty (heavy row, tile) units, h * ntiles + tile, at nz_off[h].
void launch_tile_worklist(const int32_t* heavy_rows, int64_t nheavy, const int32_t* big_slot, const int32_t* tile_cnt,
                          int ntiles, const int64_t* nz_off, int64_t* work, const LaunchCtx& lc);
void launch_build_blocked_index(const DCsr& B, int ntiles, int32_t* bidx, const LaunchCtx& lc);
// Tile occupancy bits of B from its blocked index (ceil(ntiles / 32) words per row).
void launch_build_tile_occupancy(int64_t rows, const int32_t* bidx, int ntiles, uint32_t* tocc, const LaunchCtx& lc);
// B's arrays take bulk copies (16-byte aligned).
bool bulk_aligned(const DCsr& B);
// Tiles by themselves, segments of 64+ entries staged into shared memory by
// bulk copies (bulk_aligned(B) only).  bidx: blocked index of B
// (launch_build_blocked_index) or null (binary searches); tocc: its occupancy
// bits or null; work/nwork: the list of non-empty tiles (launch_tile_worklist)
// and its length on the device, or null (every tile is visited)
void launch_num_tile(const DCsr& A, const DCsr& B, const int32_t* heavy_rows, int64_t nheavy, const int32_t* big_slot,
                     const int32_t* tile_cnt, const int32_t* tile_off, int ntiles, const int64_t* c_rp,
                     int32_t* c_col, float* c_val, const int32_t* bidx, const uint32_t* tocc, const int64_t* work,
                     const int64_t* nwork, unsigned long long* tile_counter, int* flags, const LaunchCtx& lc);
// Heavy rows as units of consecutive column tiles (heavy_unit.cu).  `units`
// holds room = heavy_unit_bound(nheavy, ntiles, entries of those rows);
// bidx as above; bitmap: the rows' column bitmaps at big_slot * stride words
// (from launch_sym_dense), or null: with c_known the columns are those in c_col,
// which stays as it is (a product on another column or an entry without a product
// raises a flag), else each unit finds its columns itself and compares them with
// tile_cnt.  Either way rows of at most whole_max entries see every product, also
// those outside the tiles with entries.  counters: two device words.
int64_t heavy_unit_bound(int64_t nheavy, int ntiles, int64_t entries);
void launch_num_units(const DCsr& A, const DCsr& B, const int32_t* heavy_rows, int64_t nheavy, const int32_t* big_slot,
                      const int32_t* tile_cnt, int ntiles, const int64_t* c_rp, int32_t* c_col, float* c_val,
                      const int32_t* bidx, const uint32_t* bitmap, int64_t stride, bool c_known, int64_t whole_max,
                      int4* units, int64_t room, unsigned long long* counters, int* flags, const LaunchCtx& lc);
void launch_compact_rows(const int32_t* rows, int64_t nrows, const uint8_t* need_exact, const int64_t* slab_off,
                         const int32_t* slab_col, const float* slab_val, const int64_t* c_rp, int32_t* c_col,
                         float* c_val, const LaunchCtx& lc);
void launch_mark_rows(const int32_t* retry, const unsigned long long* count, uint8_t* need_exact, const LaunchCtx& lc);
// out[r] = scan[r + 1] - scan[r] (undoes an exclusive scan of rows counts).
void launch_adjacent_diff(const int64_t* scan, int64_t rows, int64_t* out, const LaunchCtx& lc);
void launch_mask_key(const int64_t* src, const uint8_t* mask, int64_t rows, int64_t* dst, const LaunchCtx& lc);

}  // namespace spg
